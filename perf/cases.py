"""The work this package is used for, as performance cases.

A case is a dict of plain values; `prepare` makes its inputs on the GPU, `run` takes one pass through the package's public
entry points and returns what the path computes.  All values are drawn from N(0,1) and quantised the way the package's own
drivers do it (bench.py); head weights are N(0,1)/8 with the query scale and head_dim**-0.5 folded in.

The indexer's selected positions come in no particular order (the contract of ops.topk_select), so the cases return what is
computed from them: attention outputs.

Kinds
  prefill       a whole sequence through layer.PrefillPipeline: indexer -> top-k -> sparse MLA, causal
  chunk         layer.dsa_prefill on `rows` new tokens at the end of a `keys`-token context (chunked prefill, prefix-cache
                hits; `heads` < 128 is a tensor-parallel rank's share of the attention heads)
  decode        layer.dsa_decode_step over paged FP8 caches, one new token per sequence
  layer         layer.DSALayer from hidden states, projections included
  block_sparse  the block-sparse attention that DSA.register_sparse_fa returns
  cache_write   the write side of both decode caches: latent records and indexer keys of `tokens` new tokens
"""
import math

import torch

from llmdivedeep_b200 import DSA, layer, ops

IDX_HEADS, IDX_DIM, TOPK = 64, 128, 2048
SCALE = 192 ** -0.5
DEV = "cuda"

# hidden, q_lora, indexer heads, indexer dim, rope dim, top-k, attention heads, interleaved rope
LAYERS = {
    "small": (1024, 256, 4, 64, 64, 256, 16, False),       # DSALayer's defaults: the small configuration
    "dsv32": (7168, 1536, 64, 128, 64, 2048, 128, False),  # DSA.SPECS["dsv32"]
    "glm": (6144, 2048, 64, 128, 64, 2048, 64, True),      # DSA.SPECS["glm"]
}


def listed():
    return [
        # decode: a single short conversation, a few long ones, the 128K batch of the headline, a large batch of ordinary ones
        {"name": "decode_1x2k", "kind": "decode", "batch": 1, "ctx": 2000, "ragged": False, "heads": 128, "w": "f32"},
        {"name": "decode_7x33k", "kind": "decode", "batch": 7, "ctx": 33000, "ragged": True, "heads": 128, "w": "f32"},
        {"name": "decode_64x128k", "kind": "decode", "batch": 64, "ctx": 131072, "ragged": False, "heads": 128, "w": "f32"},
        {"name": "decode_160x9k", "kind": "decode", "batch": 160, "ctx": 9000, "ragged": True, "heads": 128, "w": "bf16"},
        # one attention layer from hidden states: the small configuration, and the full-size one on an ordinary prompt
        {"name": "layer_small_2k", "kind": "layer", "spec": "small", "rows": 2048},
        {"name": "layer_dsv32_3k", "kind": "layer", "spec": "dsv32", "rows": 3000},
        # prefill: a whole 32K sequence; a chunk of a 128K one; a follow-up question on a cached 20K prompt (odd sizes);
        # one rank of eight splitting the attention heads
        {"name": "prefill_32k", "kind": "prefill", "rows": 32768, "heads": 128},
        {"name": "chunk_4k_of_128k", "kind": "chunk", "rows": 4096, "keys": 131072, "heads": 128, "w": "bf16"},
        {"name": "chunk_257_of_20k", "kind": "chunk", "rows": 257, "keys": 20011, "heads": 128, "w": "f32"},
        {"name": "chunk_2k_of_16k_tp8", "kind": "chunk", "rows": 2048, "keys": 16384, "heads": 16, "w": "bf16"},
        # the block-sparse shape of the published table (24 heads, 5 % of the key blocks)
        {"name": "block_sparse_16k", "kind": "block_sparse", "batch": 1, "seq": 16384, "heads": 24, "share": 0.05},
        # cache write of one prefill chunk
        {"name": "cache_write_8k", "kind": "cache_write", "tokens": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "chunk", "chunk", "prefill", "layer", "layer", "block_sparse", "cache_write"])
    if kind == "decode":
        batch = _log(rng, 1, 256)
        ctx = _log(rng, 500, min(131072, 64 * 131072 // batch))
        return {"kind": kind, "batch": batch, "ctx": ctx, "ragged": rng.random() < 0.7, "heads": rng.choice([128, 128, 64]),
                "w": rng.choice(["f32", "bf16"])}
    if kind == "chunk":
        keys = _log(rng, 2048, 131072)
        return {"kind": kind, "rows": _log(rng, 64, min(4096, keys)), "keys": keys, "heads": rng.choice([128, 128, 64, 16]),
                "w": rng.choice(["f32", "bf16"])}
    if kind == "prefill":
        return {"kind": kind, "rows": _log(rng, 2048, 32767), "heads": rng.choice([128, 128, 64])}
    if kind == "layer":
        spec = rng.choice(sorted(LAYERS))
        return {"kind": kind, "spec": spec, "rows": _log(rng, 256, 6000)}
    if kind == "block_sparse":
        return {"kind": kind, "batch": rng.choice([1, 1, 2]), "seq": 64 * _log(rng, 32, 256), "heads": rng.choice([8, 16, 24]),
                "share": rng.choice([0.05, 0.05, 0.1])}
    return {"kind": kind, "tokens": _log(rng, 64, 131072)}


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, device=DEV, generator=g, dtype=dtype)


def _q_side(g, rows, w):
    q8, qs = ops.fp8_quant_per_block(_randn(g, rows, IDX_HEADS, IDX_DIM), IDX_DIM)
    wt = (_randn(g, rows, IDX_HEADS) / 8 * qs * IDX_DIM ** -0.5).to(torch.float32 if w == "f32" else torch.bfloat16)
    return q8, wt


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    st = {"kind": kind}
    if kind in ("prefill", "chunk"):
        rows, keys, heads = case["rows"], case.get("keys", case["rows"]), case["heads"]
        st["q8"], st["w"] = _q_side(g, rows, case.get("w", "bf16"))
        st["k8"], st["ksc"] = ops.fp8_quant_per_block(_randn(g, keys, IDX_DIM), IDX_DIM)
        st["q"] = _randn(g, rows, heads, 576, dtype=torch.bfloat16)
        st["kv"] = _randn(g, keys, 576, dtype=torch.bfloat16)
        if kind == "prefill":
            st["pipe"] = layer.PrefillPipeline(rows, DEV, n_heads=heads, topk=TOPK, chunk_rows=4096, softmax_scale=SCALE)
            st["out"] = st["pipe"].output_buffer()
        else:
            st["ks"] = torch.zeros(rows, dtype=torch.int32, device=DEV)
            st["ke"] = torch.arange(keys - rows + 1, keys + 1, dtype=torch.int32, device=DEV)
    elif kind == "decode":
        batch, ctx, heads = case["batch"], case["ctx"], case["heads"]
        pages = -(-ctx // 64)
        n = batch * pages * 64
        st["kcache"] = torch.empty(n, IDX_DIM, dtype=torch.float8_e4m3fn, device=DEV)
        st["kscale"] = torch.empty(n, dtype=torch.float32, device=DEV)
        st["latent"] = torch.empty(n, layer.LATENT_TOKEN_BYTES, dtype=torch.uint8, device=DEV)
        step = 1 << 20
        for a in range(0, n, step):
            b = min(n, a + step)
            st["kcache"][a:b], st["kscale"][a:b] = ops.fp8_quant_per_block(_randn(g, b - a, IDX_DIM), IDX_DIM)
            layer.pack_latent_cache(_randn(g, b - a, 576, dtype=torch.bfloat16), out=st["latent"][a:b])
        st["table"] = torch.randperm(batch * pages, device=DEV, generator=g).int().view(batch, pages)
        st["ctx"] = (torch.randint(ctx // 2, ctx + 1, (batch,), device=DEV, generator=g).int() if case["ragged"]
                     else torch.full((batch,), ctx, dtype=torch.int32, device=DEV))
        st["q8"], st["w"] = _q_side(g, batch, case["w"])
        st["q"] = _randn(g, batch, heads, 576, dtype=torch.bfloat16)
        st["ws"] = layer.DecodeWorkspace(batch, heads, pages * 64, TOPK, DEV)
    elif kind == "layer":
        hidden, q_lora, ih, idim, rope, topk, heads, interleave = LAYERS[case["spec"]]
        torch.manual_seed(seed)
        with torch.device(DEV):
            st["layer"] = layer.DSALayer(hidden, q_lora, ih, idim, rope, topk, heads, SCALE, interleave)
        st["x"] = _randn(g, case["rows"], hidden, dtype=torch.bfloat16)
    elif kind == "block_sparse":
        torch.manual_seed(seed)
        shape = (case["batch"], case["seq"], case["heads"], 128)
        st["q"], st["k"], st["v"] = (_randn(g, *shape, dtype=torch.bfloat16) for _ in range(3))
        build_lut, st["attend"] = DSA.register_sparse_fa()
        st["idx"], st["num"], _ = build_lut(st["q"], case["seq"], case["share"])
    else:
        st["kv"] = _randn(g, case["tokens"], 576, dtype=torch.bfloat16)
        st["k"] = _randn(g, case["tokens"], IDX_DIM, dtype=torch.bfloat16)
    return st


def run(st):
    kind = st["kind"]
    if kind == "prefill":
        return st["pipe"].run(st["q8"], st["k8"], st["ksc"], st["w"], st["q"], st["kv"], st["out"])
    if kind == "chunk":
        return layer.dsa_prefill(st["q8"], st["k8"], st["ksc"], st["w"], st["ks"], st["ke"], TOPK, st["q"], st["kv"], SCALE)[1]
    if kind == "decode":
        return layer.dsa_decode_step(st["q8"], st["w"], st["kcache"], st["kscale"], st["table"], st["ctx"], st["q"], st["latent"],
                                     SCALE, st["ws"])[1]
    if kind == "layer":
        return st["layer"](st["x"])
    if kind == "block_sparse":
        return st["attend"](st["q"], st["k"], st["v"], st["idx"], st["num"], 128 ** -0.5)
    latent = layer.pack_latent_cache(st["kv"])
    k8, ksc = DSA.fp8_quant_per_block(st["k"])
    return {"latent": latent, "k8": k8.view(torch.uint8), "k_scale": ksc}


def _causal(rows, keys):
    """(query, key) pairs inside the causal windows of the last `rows` of `keys` positions."""
    return rows * (keys - rows) + rows * (rows + 1) // 2


def _selected(rows, keys, k):
    """Selected pairs of the same rows: min(window, k) each."""
    short = min(rows, max(0, k - (keys - rows)))           # rows whose window is at most k
    first = keys - rows + 1
    return short * first + short * (short - 1) // 2 + (rows - short) * k


def work(case):
    kind = case["kind"]
    if kind in ("prefill", "chunk"):
        rows, keys, heads = case["rows"], case.get("keys", case["rows"]), case["heads"]
        w = 4 if case.get("w") == "f32" else 2
        return {"bytes": rows * IDX_HEADS * (IDX_DIM + w) + keys * (IDX_DIM + 4) + rows * heads * (1152 + 1024) + keys * 1152,
                "flops": 2 * IDX_HEADS * IDX_DIM * _causal(rows, keys) + 2 * heads * 1088 * _selected(rows, keys, TOPK)}
    if kind == "decode":
        batch, heads = case["batch"], case["heads"]
        ctx = case["ctx"] * (0.75 if case["ragged"] else 1.0)
        sel = min(ctx, TOPK)
        return {"bytes": batch * (ctx * (IDX_DIM + 4 + 4 / 64) + sel * 656 + IDX_HEADS * (IDX_DIM + 4) + heads * (1152 + 1024)),
                "flops": batch * (2 * IDX_HEADS * IDX_DIM * ctx + 2 * heads * 1088 * sel)}
    if kind == "layer":
        hidden, q_lora, ih, idim, _, topk, heads, _ = LAYERS[case["spec"]]
        rows = case["rows"]
        weights = hidden * (q_lora + idim + ih + 576) + q_lora * (ih * idim + heads * 576)
        return {"bytes": 2 * (weights + rows * hidden + rows * heads * 512),
                "flops": 2 * rows * weights + 2 * ih * idim * _causal(rows, rows) + 2 * heads * 1088 * _selected(rows, rows, min(topk, rows))}
    if kind == "block_sparse":
        blocks = case["seq"] // 64
        picked = max(1, int(round(case["share"] * blocks)))
        n = case["batch"] * case["heads"] * case["seq"]
        return {"bytes": n * 128 * 2 * 4 + n // 64 * (picked + 1) * 4, "flops": 4 * 128 * 64 * picked * n}
    return {"bytes": case["tokens"] * (1152 + 656 + 256 + 132), "flops": 0}


def tolerance(case):
    if case["kind"] == "cache_write":
        return "exact"                                      # whole bytes, and scales that are one IEEE division
    # against the same attention in float64 the outputs differ by rel 1.2e-3 .. 3.5e-3 (bf16 operands, probabilities and
    # outputs; decode also rounds the dequantised cache to bf16) and by at most 0.025 of a value: four times that
    return {"rel": 0.012, "max": 0.1}


# ---- the same results in plain torch, in 64 bits ------------------------------------------------------------------
def _quant(x, block):
    """bf16 / fp32 values -> (e4m3 values, fp32 scale per block), both widened to float64."""
    xb = x.float().reshape(*x.shape[:-1], -1, block)
    scale = xb.abs().amax(-1).clamp_min(1e-6) / 448
    q8 = (xb / scale.unsqueeze(-1)).to(torch.float8_e4m3fn).reshape(x.shape)
    return q8.double(), scale.double()


def _rope(x, rope, interleave):
    """x [T, ..., dim]: rotation of the first `rope` values at position = row."""
    half = rope // 2
    inv = 1.0 / (10000.0 ** (torch.arange(0, half, device=DEV, dtype=torch.float32) / half))
    ang = torch.outer(torch.arange(x.shape[0], device=DEV, dtype=torch.float32), inv).view(x.shape[0], *([1] * (x.dim() - 2)), half)
    cos, sin = ang.cos(), ang.sin()
    a, b = (x[..., 0:rope:2], x[..., 1:rope:2]) if interleave else (x[..., :half], x[..., half:rope])
    y = (a * cos - b * sin, a * sin + b * cos)
    y = torch.stack(y, -1).flatten(-2).to(x.dtype) if interleave else torch.cat(y, -1)
    return torch.cat((y, x[..., rope:].to(y.dtype)), -1)


def _attend(q8, w, k8, ksc, first, q, kv, topk, out):
    """Rows of one sequence, row i seeing the first `first + i` keys: scores, selection, attention; all in float64."""
    rows, heads, keys = q8.shape[0], q8.shape[1], k8.shape[0]
    k8t, pos = k8.double().t(), torch.arange(keys, device=DEV)
    step = max(1, min(64, (1 << 27) // (heads * keys)))
    for a in range(0, rows, step):
        b = min(rows, a + step)
        s = (q8[a:b].double().reshape(-1, q8.shape[2]) @ k8t).relu_().view(b - a, heads, keys)
        s = torch.einsum("ths,th->ts", s, w[a:b].double()) * ksc.double()
        window = torch.arange(first + a, first + b, device=DEV).unsqueeze(1)
        top = s.masked_fill(pos >= window, -math.inf).topk(min(topk, keys), dim=-1)
        for c in range(a, b, 32):
            d = min(b, c + 32)
            g = kv[top.indices[c - a:d - a]].double()
            p = torch.bmm(q[c:d].double(), g.transpose(1, 2)) * SCALE
            p = p.masked_fill((top.values[c - a:d - a] == -math.inf).unsqueeze(1), -math.inf).softmax(-1)
            out[c:d] = torch.bmm(p, g[..., :512])
    return out


def exact(case, seed):
    """What `run` returns for the inputs `prepare` makes, in float64 from the same quantised and bf16 operands.  A layer's
    projections stay the bf16 Linears that its module consists of: their outputs are the operands."""
    kind, st = case["kind"], prepare(case, seed)
    if kind in ("prefill", "chunk"):
        out = torch.empty(case["rows"], case["heads"], 512, dtype=torch.float64, device=DEV)
        return _attend(st["q8"], st["w"], st["k8"], st["ksc"], case.get("keys", case["rows"]) - case["rows"] + 1, st["q"], st["kv"],
                       TOPK, out)
    if kind == "decode":
        out = torch.empty(case["batch"], case["heads"], 512, dtype=torch.float64, device=DEV)
        for b, n in enumerate(st["ctx"].tolist()):
            row = torch.arange(n, device=DEV)
            row = st["table"][b, row // 64].long() * 64 + row % 64
            rec = st["latent"][row]
            lat = rec[:, :512].contiguous().view(torch.float8_e4m3fn).double().view(n, 4, 128)
            lat = lat * rec[:, 512:528].contiguous().view(torch.float32).double().unsqueeze(-1)
            kv = torch.cat((lat.view(n, 512), rec[:, 528:].contiguous().view(torch.bfloat16).double()), -1)
            k8 = st["kcache"].view(torch.uint8)[row].view(torch.float8_e4m3fn)
            _attend(st["q8"][b:b + 1], st["w"][b:b + 1], k8, st["kscale"][row], n, st["q"][b:b + 1], kv, TOPK, out[b:b + 1])
        return out
    if kind == "layer":
        _, _, ih, idim, rope, topk, heads, interleave = LAYERS[case["spec"]]
        m, x, rows = st["layer"], st["x"], case["rows"]
        linear = torch.nn.functional.linear
        with torch.no_grad():
            ql, ind = linear(x, m.q_a.weight), m.indexer
            k = torch.nn.functional.layer_norm(linear(x, ind.wk.weight), (idim,), ind.k_norm.weight, ind.k_norm.bias, ind.k_norm.eps)
            q8, qs = _quant(_rope(linear(ql, ind.wq_b.weight).view(rows, ih, idim), rope, interleave), idim)
            k8, ksc = _quant(_rope(k, rope, interleave), idim)
            w = (linear(x, ind.weights_proj.weight).float() * ih ** -0.5).double() * qs.squeeze(-1) * idim ** -0.5
            q, kv = linear(ql, m.wq.weight).view(rows, heads, 576), linear(x, m.wkv.weight)
            return _attend(q8, w, k8, ksc.squeeze(-1), 1, q, kv, topk,
                           torch.empty(rows, heads, 512, dtype=torch.float64, device=DEV))
    if kind == "block_sparse":
        batch, seq, heads = case["batch"], case["seq"], case["heads"]
        out = torch.empty(batch, seq, heads, 128, dtype=torch.float64, device=DEV)
        for b in range(batch):
            for h in range(heads):
                k, v = (st[n][b, :, h].double().view(seq // 64, 64, 128) for n in ("k", "v"))
                q = st["q"][b, :, h].double().view(seq // 64, 64, 128)
                for i in range(0, seq // 64, 32):
                    lut = st["idx"][b, h, i:i + 32].long()
                    kk, vv = (t[lut].flatten(1, 2) for t in (k, v))
                    p = (torch.bmm(q[i:i + 32], kk.transpose(1, 2)) * 128 ** -0.5).softmax(-1)
                    out[b, i * 64:(i + 32) * 64, h] = torch.bmm(p, vv).flatten(0, 1)
        return out
    return None                                             # whole bytes, and scales that are compared bit for bit
