"""Decode path through the C ABI: paged FP8 indexer scan, top-k over each sequence's context,
sparse MLA over the paged FP8 latent cache -- each stage and the composed step against the oracle."""
import pytest
import torch

from llmdivedeep_b200 import layer, ops
from oracle import dsa_oracle as O

pytestmark = pytest.mark.gpu
REL_TOL = 4e-6
ULP_TOL = 4.0


def make_cache(B, P, H, seed, ragged=True):
    g = torch.Generator().manual_seed(seed)
    n_pages = B * P + 3                                           # a few pages no sequence uses
    k = torch.randn(n_pages * 64, 128, generator=g)
    k8, ksc = O.fp8_quant_per_block(k, 128)
    table = torch.randperm(n_pages, generator=g)[: B * P].int().view(B, P)
    ctx = torch.randint(P * 64 // 2, P * 64 + 1, (B,), generator=g).int() if ragged else torch.full((B,), P * 64).int()
    q = torch.randn(B, H, 128, generator=g)
    q8, qs = O.fp8_quant_per_block(q, 128)
    w = O.fold_weights(torch.randn(B, H, generator=g) / 8, qs, 128)
    return q8, w, k8, ksc, table, ctx


@pytest.mark.parametrize("B,P,H", [(4, 6, 64), (3, 33, 64), (2, 5, 32), (5, 1, 64)])
def test_paged_logits_match_oracle(B, P, H):
    q8, w, k8, ksc, table, ctx = make_cache(B, P, H, seed=B * 7 + P)
    out = ops.fp8_paged_mqa_logits(q8.cuda(), w.cuda(), k8.cuda(), ksc.cuda(), table.cuda(), ctx.cuda(), P * 64)
    ops.check_status("cuda")
    o = out.cpu().double()
    for b in range(B):
        n = int(ctx[b])
        rows = O.physical_rows(table[b], torch.arange(n))
        ref = O.indexer_logits_fp64(q8[b:b + 1], k8[rows], ksc[rows], w[b:b + 1], torch.zeros(1, dtype=torch.int32),
                                    torch.tensor([n], dtype=torch.int32))[0]
        err = (o[b, :n] - ref).abs().max()
        assert float(err) <= REL_TOL * float(ref.abs().max()), (b, float(err))
        tile_end = min(P * 64, (n + 127) // 128 * 128)
        assert bool(torch.isinf(out[b, n:tile_end]).all())       # masked tail of the last tile


def test_paged_equals_contiguous_kernel_bitwise():
    """Same keys through the paged and the contiguous entry point give identical logits."""
    B, P, H = 2, 16, 64
    q8, w, k8, ksc, table, ctx = make_cache(B, P, H, seed=3, ragged=False)
    paged = ops.fp8_paged_mqa_logits(q8.cuda(), w.cuda(), k8.cuda(), ksc.cuda(), table.cuda(), ctx.cuda(), P * 64)
    for b in range(B):
        rows = O.physical_rows(table[b], torch.arange(P * 64))
        ke = torch.tensor([P * 64], dtype=torch.int32).cuda()
        flat = ops.fp8_mqa_logits(q8[b:b + 1].cuda(), (k8[rows].cuda(), ksc[rows].cuda()), w[b:b + 1].cuda(), None, ke)
        assert torch.equal(flat[0], paged[b])


def test_bad_page_id_is_flagged_not_read():
    q8, w, k8, ksc, table, ctx = make_cache(2, 4, 64, seed=5, ragged=False)
    table[1, 2] = 10_000
    out = ops.fp8_paged_mqa_logits(q8.cuda(), w.cuda(), k8.cuda(), ksc.cuda(), table.cuda(), ctx.cuda(), 256)
    with pytest.raises(ops.DsaError, match="out of range"):
        ops.check_status("cuda")
    assert bool(torch.isfinite(out[0]).all())


def test_decode_step_composition():
    B, P, H, K = 6, 20, 128, 256
    g = torch.Generator().manual_seed(12)
    q8, w, k8, ksc, table, ctx = make_cache(B, P, 64, seed=12)
    n_rows = k8.shape[0]
    kv = torch.randn(n_rows, 576, generator=g).to(torch.bfloat16)
    cache = O.pack_latent_cache(kv)
    q = torch.randn(B, H, 576, generator=g).to(torch.bfloat16)
    ws = layer.DecodeWorkspace(B, H, P * 64, K, "cuda")
    idx, out = layer.dsa_decode_step(q8.cuda(), w.cuda(), k8.cuda(), ksc.cuda(), table.cuda(), ctx.cuda(), q.cuda(),
                                     cache.cuda(), 0.05, ws)
    ops.check_status("cuda")
    # selection against float64 scores
    ref = O.indexer_logits_paged(q8, w, k8, ksc, table, ctx).double()
    for b in range(B):
        n = int(ctx[b])
        rows = O.physical_rows(table[b], torch.arange(n))
        ref[b, :n] = O.indexer_logits_fp64(q8[b:b + 1], k8[rows], ksc[rows], w[b:b + 1], torch.zeros(1, dtype=torch.int32),
                                           torch.tensor([n], dtype=torch.int32))[0]
    r = O.check_topk_sets(idx.cpu().numpy(), ref.numpy(), [0] * B, ctx.tolist(), K, ulp_tol=ULP_TOL)
    assert not r["bad_rows"], r
    # attention over the kernel's own selection
    want = O.sparse_mla_decode_paged(q.float(), cache, table, idx.cpu(), 0.05, round_bf16=True)
    d = (out.float().cpu() - want).abs()
    assert float(d.max()) <= 2e-2 and float(d.mean()) <= 2e-3


def test_prefill_composition_small_config():
    """The small CPU-reference configuration end to end: 2048 tokens, 4 indexer heads of 64,
    top-k 256, 16 attention heads over one shared latent KV."""
    from tests.helpers import indexer_inputs
    T, K = 2048, 256
    q8, k8, ksc, w, ks, ke = indexer_inputs(T, T, 4, 64, seed=0, window="causal")
    g = torch.Generator().manual_seed(1)
    q = torch.randn(T, 16, 576, generator=g).to(torch.bfloat16)
    kv = torch.randn(T, 576, generator=g).to(torch.bfloat16)
    idx, out = layer.dsa_prefill(q8.cuda(), k8.cuda(), ksc.cuda(), w.cuda(), ks.cuda(), ke.cuda(), K, q.cuda(), kv.cuda(),
                                 192 ** -0.5)
    ops.check_status("cuda")
    ref = O.indexer_logits_fp64(q8, k8, ksc, w, ks, ke).numpy()
    r = O.check_topk_sets(idx.cpu().numpy(), ref, ks.numpy(), ke.numpy(), K, ulp_tol=ULP_TOL)
    assert not r["bad_rows"], r
    rows = torch.arange(0, T, 37)                                   # oracle attention on a sample of rows
    want = O.sparse_mla(q[rows].float(), kv.float(), idx.cpu()[rows], 192 ** -0.5)
    d = (out.float().cpu()[rows] - want).abs()
    assert float(d.max()) <= 2e-2 and float(d.mean()) <= 2e-3


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2000])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_pack_latent_cache_records(n, dtype):
    """Every form of input and record tensor gives the oracle's bytes: dense rows and rows cut out of wider ones (the
    one-kernel path), strided columns, unaligned rows and strided records (the quantiser and copies)."""
    from llmdivedeep_b200 import layer
    g = torch.Generator().manual_seed(n)
    kv = torch.randn(n, 576, generator=g).to(dtype)
    kv[0, :128] = 0
    kv[n - 1, 100:140] *= 1e4
    want = O.pack_latent_cache(kv)
    wide = torch.zeros(n, 640, dtype=dtype)
    wide[:, 32:608] = kv
    odd = torch.zeros(n, 577, dtype=dtype)
    odd[:, 1:] = kv
    forms = [kv.cuda(), wide.cuda()[:, 32:608], kv.t().contiguous().cuda().t()]
    if n > 1:                                          # (one unaligned row counts as contiguous, and the quantiser refuses it)
        forms.append(odd.cuda()[:, 1:])
    for x in forms:
        assert torch.equal(layer.pack_latent_cache(x).cpu(), want)
        out = torch.zeros(n, 700, dtype=torch.uint8, device="cuda")
        assert torch.equal(layer.pack_latent_cache(x, out=out[:, 3:659]).cpu(), want)
        assert int(out[:, :3].sum()) == 0 and int(out[:, 659:].sum()) == 0


@pytest.mark.parametrize("block", [64, 128])
@pytest.mark.parametrize("n_blocks", [1, 3, 8, 33, 70001])
def test_quantiser_ragged_block_counts_and_unaligned_output(n_blocks, block):
    from llmdivedeep_b200 import _lib
    x = torch.randn(n_blocks, block, generator=torch.Generator().manual_seed(n_blocks)).to(torch.bfloat16)
    want_q, want_s = O.fp8_quant_per_block(x, block)
    xd = x.cuda()
    for off in (0, 4):
        q = torch.zeros(n_blocks * block + 8, dtype=torch.uint8, device="cuda")
        s = torch.zeros(n_blocks + 1, device="cuda")
        _lib.check(_lib.load().dsa_fp8_quant_per_block(xd.data_ptr(), 1, n_blocks, block, q.data_ptr() + off, s.data_ptr(),
                                                       torch.cuda.current_stream().cuda_stream))
        assert torch.equal(q[off:off + n_blocks * block].cpu(), want_q.view(torch.uint8).reshape(-1)) and not q[off + n_blocks * block:].any()
        assert torch.equal(s[:n_blocks].cpu(), want_s.reshape(-1)) and float(s[n_blocks]) == 0


@pytest.mark.parametrize("B,P,H", [(1, 1, 64), (1, 8, 64), (1, 9, 64), (1, 33, 16), (7, 66, 64), (150, 9, 64)])
def test_paged_logits_of_calls_with_few_tiles(B, P, H):
    """Calls too small to give every SM a unit of eight tiles: units of four, two and one tile."""
    test_paged_logits_match_oracle(B, P, H)


def test_calls_without_a_workspace_on_two_streams():
    """Split decode batches and an indexer_topk on streams of their own, none given a workspace: the results of the same calls
    one after the other."""
    from tests.helpers import indexer_inputs, to_dev
    g = torch.Generator().manual_seed(5)
    B, H, P, K = 75, 128, 10, 600                      # one query beyond a round of CTA pairs: cut into parts
    caches = [O.pack_latent_cache(torch.randn(B * P * 64, 576, generator=g).to(torch.bfloat16)).cuda() for _ in range(2)]
    table = torch.randperm(B * P, generator=g).int().view(B, P).cuda()
    idx = torch.rand(B, P * 64, generator=g).topk(K, dim=-1).indices.int().cuda()
    q = torch.randn(B, H, 576, generator=g).to(torch.bfloat16).cuda()
    ind = to_dev(*indexer_inputs(512, 2048, 64, 128, seed=6))
    calls = [lambda: ops.sparse_mla_decode_paged(q[:9], caches[0], table[:9], idx[:9], 0.06),
             lambda: ops.sparse_mla_decode_paged(q, caches[1], table, idx, 0.06),
             lambda: ops.indexer_topk(*ind, 256)]
    want = [c() for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    got = [[] for _ in calls]
    for _ in range(20):
        for c, s, o in zip(calls, streams, got):
            with torch.cuda.stream(s):
                o.append(c())
    torch.cuda.synchronize()
    ops.check_status("cuda")
    for w, o in zip(want, got):
        assert all(torch.equal(x, w) for x in o)


def test_smaller_batches_in_the_workspace_of_a_larger_one():
    """The parts of every batch fit the buffer made for the largest: the bits of the call with scratch of its own.  Buffers of
    fewer parts give fewer parts, and the same result within the merge's rounding."""
    B, H, P, K = 64, 128, 34, 2048
    g = torch.Generator().manual_seed(64)
    cache = O.pack_latent_cache(torch.randn(B * P * 64, 576, generator=g).to(torch.bfloat16)).cuda()
    table = torch.randperm(B * P, generator=g).int().view(B, P).cuda()
    idx = torch.rand(B, P * 64, generator=g).topk(K, dim=-1).indices.int().cuda()
    q = torch.randn(B, H, 576, generator=g).to(torch.bfloat16).cuda()
    ws = layer.DecodeWorkspace(B, H, P * 64, K, "cuda").mla_ws
    for b in (1, 7, 12, 23, 37, 38, 64):
        args = (q[:b], cache, table[:b], idx[:b], 0.06)
        own = ops.sparse_mla_decode_paged(*args)
        assert torch.equal(ops.sparse_mla_decode_paged(*args, workspace=ws), own)
        assert torch.equal(ops.sparse_mla_decode_paged(*args, workspace=ws), own)
        whole = ops.sparse_mla_decode_paged(*args, workspace=ws[:16])
        for parts in (1, 2, 3, 5):                     # per query; poison behind what such a buffer may use
            small = torch.full((b * parts * H * 514 * 4 + 4096,), 7, dtype=torch.uint8, device="cuda")
            out = ops.sparse_mla_decode_paged(*args, workspace=small[: b * parts * H * 514 * 4 + 100])
            assert bool((small[b * parts * H * 514 * 4:] == 7).all())
            assert float((out.float() - whole.float()).abs().max()) <= 2e-2
            assert not torch.isnan(out).any()
    ops.check_status("cuda")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("block", [64, 128])
def test_quantiser_around_the_change_of_values_per_thread(block, dtype):
    """Few blocks take four values a thread, many sixteen: the oracle's bytes and scales on both sides of the line, with zero
    blocks among them."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = sms * (256 if dtype == torch.bfloat16 else 512) // (block // 16)
    x = torch.randn(line + 1, block, generator=torch.Generator().manual_seed(block)).to(dtype)
    x[::37] = 0
    want_q, want_s = O.fp8_quant_per_block(x, block)
    for n in (line - 1, line, line + 1):
        q, s = ops.fp8_quant_per_block(x[:n].cuda(), block)
        assert torch.equal(q.view(torch.uint8).cpu(), want_q[:n].view(torch.uint8)) and torch.equal(s.cpu().reshape(-1), want_s[:n].reshape(-1))


@pytest.mark.parametrize("B,P,lens", [(1, 3, "full"), (3, 130, "ragged"), (40, 141, "ragged"), (64, 300, "ragged"), (160, 60, "full"), (300, 20, "short")])
def test_paged_scan_units_cover_every_context(B, P, lens):
    """The cut of the paged scan into units (four tiles, or what leaves the longest CTA least to do): every position of every
    context scored, against the contiguous kernel on the same keys."""
    g = torch.Generator(device="cuda").manual_seed(B + P)
    k8, ksc = ops.fp8_quant_per_block(torch.randn(B * P * 64, 128, device="cuda", generator=g), 128)
    table = torch.randperm(B * P, device="cuda", generator=g).int().view(B, P)
    lo = {"full": P * 64, "ragged": P * 32, "short": 1}[lens]
    ctx = torch.randint(lo, P * 64 + 1, (B,), device="cuda", generator=g).int()
    q8, _ = ops.fp8_quant_per_block(torch.randn(B, 64, 128, device="cuda", generator=g), 128)
    w = torch.randn(B, 64, device="cuda", generator=g)
    got = ops.fp8_paged_mqa_logits(q8, w, k8, ksc, table, ctx, P * 64)
    ops.check_status("cuda")
    for b in sorted({0, B // 2, B - 1}):
        rows = (table[b].long().unsqueeze(1) * 64 + torch.arange(64, device="cuda")).flatten()
        n = int(ctx[b])
        one = ops.fp8_mqa_logits(q8[b:b + 1], (k8.view(torch.uint8)[rows].view(ops.FP8), ksc[rows]), w[b:b + 1], None, ctx[b:b + 1].clone())
        assert torch.allclose(got[b, :n], one[0, :n], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("B,heads,w_dtype", [(1, 128, torch.float32), (5, 64, torch.bfloat16), (80, 16, torch.float32)])
def test_one_call_decode_step_equals_the_three_calls(B, heads, w_dtype):
    """layer.dsa_decode_step makes one library call for tensors of the plain form and three wrapper calls for others (here: a
    strided block table): the same selection and the same bits, in a workspace made for more sequences too."""
    g = torch.Generator(device="cuda").manual_seed(B)
    P, k = 40, 512
    n = B * P * 64
    kc, ksc = ops.fp8_quant_per_block(torch.randn(n, 128, device="cuda", generator=g), 128)
    lat = layer.pack_latent_cache(torch.randn(n, 576, device="cuda", generator=g).bfloat16())
    table = torch.randperm(B * P, device="cuda", generator=g).int().view(B, P)
    ctx = torch.randint(300, P * 64 + 1, (B,), device="cuda", generator=g).int()
    q8, qs = ops.fp8_quant_per_block(torch.randn(B, 64, 128, device="cuda", generator=g), 128)
    w = (torch.randn(B, 64, device="cuda", generator=g) * qs).to(w_dtype)
    q = torch.randn(B, heads, 576, device="cuda", generator=g).bfloat16()
    strided = torch.zeros(B, P + 3, dtype=torch.int32, device="cuda")[:, :P]
    strided.copy_(table)
    got = []
    for tab, room in ((table, B), (strided, B), (table, B + 3)):
        ws = layer.DecodeWorkspace(room, heads, P * 64, k, "cuda")
        idx, out = layer.dsa_decode_step(q8, w, kc, ksc, tab, ctx, q, lat, 0.07, ws)
        got.append((idx.clone(), out.clone()))
    ops.check_status("cuda")
    for idx, out in got[1:]:
        assert torch.equal(idx, got[0][0])
    assert torch.equal(got[1][1], got[0][1]) and torch.equal(got[2][1], got[0][1])
    with pytest.raises(ops.DsaError):
        layer.dsa_decode_step(q8, w, kc, ksc, table, ctx.long(), q, lat, 0.07, layer.DecodeWorkspace(B, heads, P * 64, k, "cuda"))


@pytest.mark.parametrize("B,heads", [(1, 128), (6, 64), (24, 128), (25, 128)])
def test_overlapping_kernels_of_steps_in_a_row(B, heads):
    """Up to 24 sequences each kernel of a step may start under the one before: many steps back to back on two sets of inputs in one
    workspace, eager and from a graph, equal those of the three separate calls."""
    g = torch.Generator(device="cuda").manual_seed(B)
    P, k = 60, 1024
    n = B * P * 64
    sets = []
    for _ in range(2):
        kc, ksc = ops.fp8_quant_per_block(torch.randn(n, 128, device="cuda", generator=g), 128)
        lat = layer.pack_latent_cache(torch.randn(n, 576, device="cuda", generator=g).bfloat16())
        table = torch.randperm(B * P, device="cuda", generator=g).int().view(B, P)
        ctx = torch.randint(1200, P * 64 + 1, (B,), device="cuda", generator=g).int()
        q8, qs = ops.fp8_quant_per_block(torch.randn(B, 64, 128, device="cuda", generator=g), 128)
        w = torch.randn(B, 64, device="cuda", generator=g) * qs
        q = torch.randn(B, heads, 576, device="cuda", generator=g).bfloat16()
        lg = ops.fp8_paged_mqa_logits(q8, w, kc, ksc, table, ctx, P * 64)
        idx = ops.topk_select(lg, k, None, ctx)
        sets.append(((q8, w, kc, ksc, table, ctx, q, lat), idx, ops.sparse_mla_decode_paged(q, lat, table, idx, 0.07, P * 64)))
    ws = layer.DecodeWorkspace(B, heads, P * 64, k, "cuda")
    got = []
    for i in range(60):
        idx, out = layer.dsa_decode_step(*sets[i % 2][0], 0.07, ws)
        got.append((idx.clone(), out.clone()))
    ops.check_status("cuda")
    for i, (idx, out) in enumerate(got):
        assert torch.equal(idx, sets[i % 2][1]) and torch.equal(out, sets[i % 2][2]), i
    outs = [torch.empty_like(ws.out) for _ in range(20)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for i, o in enumerate(outs):
            o.copy_(layer.dsa_decode_step(*sets[i % 2][0], 0.07, ws)[1])
    for _ in range(3):
        for o in outs:
            o.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, sets[i % 2][2]) for i, o in enumerate(outs))
