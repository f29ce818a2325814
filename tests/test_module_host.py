"""Host-only checks of the module mirror (llmdivedeep_b200/DSA.py) and of the oracle's stage
outputs against the reference's recorded ones: nothing here launches a kernel."""
import contextlib
import os
import weakref

import numpy as np
import pytest
import torch

from llmdivedeep_b200 import DSA, ops
from oracle import dsa_oracle as O

G = np.load(os.path.join(os.path.dirname(__file__), "golden", "reference_golden.npz"))


def bf16(a):
    return torch.from_numpy(a.view(np.int16).copy()).view(torch.bfloat16)


def _params(tag):
    return {k: bf16(G[f"mod_{tag}_{k}"]) for k in ("wq_b", "wk", "weights_proj", "k_norm_w", "k_norm_b")}


@pytest.mark.parametrize("tag,interleave", [("neox", False), ("glm", True)])
def test_oracle_stage_outputs_equal_the_reference_bytes(tag, interleave):
    """Projections -> k_norm -> RoPE -> FP8 quantiser of the oracle give the bytes, scales and
    head gates the unmodified reference hands to its scorer (sparse_attn/DSA.py:530-543)."""
    x, ql = bf16(G[f"mod_{tag}_x"]), bf16(G[f"mod_{tag}_qlora"])
    q8, k8, ksc, w_eff, ks, ke = O.dsa_indexer_inputs(_params(tag), x, ql, 4, 128, 64, interleave=interleave)
    assert np.array_equal(q8.view(torch.uint8).numpy(), G[f"mod_{tag}_q_fp8"])
    assert np.array_equal(k8.view(torch.uint8).numpy(), G[f"mod_{tag}_k_fp8"])
    assert np.array_equal(ksc.numpy(), G[f"mod_{tag}_k_scale"])
    ref_w = O.fold_weights(torch.from_numpy(G[f"mod_{tag}_w"]), torch.from_numpy(G[f"mod_{tag}_q_scale"]), 128)
    assert torch.equal(w_eff, ref_w)


@pytest.mark.parametrize("tag,interleave", [("neox", False), ("glm", True)])
def test_mirror_rope_feeds_the_quantiser_the_reference_values(tag, interleave):
    """DSA._rope_head on the module's bf16 projections, quantised, must give the reference's FP8
    bytes and scales: the NeoX form hands the quantiser unrounded fp32 products, the interleaved
    form values rounded to bf16 (sparse_attn/DSA.py:444-469, 513-524)."""
    p = _params(tag)
    x, ql = bf16(G[f"mod_{tag}_x"]), bf16(G[f"mod_{tag}_qlora"])
    T = x.shape[0]
    q = torch.nn.functional.linear(ql, p["wq_b"]).view(T, 4, 128)
    k = torch.nn.functional.layer_norm(torch.nn.functional.linear(x, p["wk"]), (128,), p["k_norm_w"], p["k_norm_b"])
    q, k = DSA._rope_head(q, 64, T, interleave), DSA._rope_head(k, 64, T, interleave)
    assert q.dtype == (torch.bfloat16 if interleave else torch.float32)
    q8, qs = O.fp8_quant_per_block(q)
    k8, ksc = O.fp8_quant_per_block(k)
    assert np.array_equal(q8.view(torch.uint8).numpy(), G[f"mod_{tag}_q_fp8"])
    assert np.array_equal(qs.numpy(), G[f"mod_{tag}_q_scale"])
    assert np.array_equal(k8.view(torch.uint8).numpy(), G[f"mod_{tag}_k_fp8"])
    assert np.array_equal(ksc.numpy(), G[f"mod_{tag}_k_scale"])


def test_rope_forms_equal_the_oracle_on_fp32_and_bf16():
    cos, sin = O.rope_cossin(10, 64)
    for dt in (torch.float32, torch.bfloat16):
        x = torch.randn(10, 3, 64).to(dt)
        assert torch.equal(DSA._rotate(x, cos, sin, False), O.apply_rope_neox(x, cos, sin))
        assert torch.equal(DSA._rotate(x, cos, sin, True), O.apply_rope_interleave(x, cos, sin))


def test_ops_refuse_cpu_tensors():
    q8 = torch.zeros(4, 64, 128).to(torch.float8_e4m3fn)
    with pytest.raises(ops.DsaError):
        ops.fp8_mqa_logits(q8, (q8[0], torch.ones(64)), torch.ones(4, 64), None, torch.ones(4, dtype=torch.int32))


class _FakeCudaTensor:
    """Stands in for a CUDA tensor in the argument checks (which only look at is_cuda / device)."""
    is_cuda = True

    def __init__(self, index):
        self.device = torch.device("cuda", index)


def test_ops_refuse_tensors_of_different_devices():
    assert ops._need_cuda(_FakeCudaTensor(1), None, _FakeCudaTensor(1)) == torch.device("cuda", 1)
    with pytest.raises(ops.DsaError, match="one device"):
        ops._need_cuda(_FakeCudaTensor(0), _FakeCudaTensor(1))
    with pytest.raises(ops.DsaError):
        ops._need_cuda(_FakeCudaTensor(0), torch.zeros(1))
    with pytest.raises(ops.DsaError):
        ops._dev_index("cpu")
    assert ops._dev_index("cuda:3") == 3


def test_index_output_must_have_the_kernel_stride():
    ok = torch.empty(6, 8, dtype=torch.int32)
    assert ops._check_idx_out(ok, 6, 8, "cpu") is ok
    for bad in (torch.empty(6, 16, dtype=torch.int32)[:, :8], torch.empty(6, 8, dtype=torch.int64),
                torch.empty(6, 16, dtype=torch.int32)):
        with pytest.raises(ops.DsaError):
            ops._check_idx_out(bad, 6, 8, "cpu")


def test_index_share_runs_the_indexer_every_freq_layers():
    from llmdivedeep_b200 import layer
    calls = []

    def indexer(x):
        calls.append(x)
        return len(calls)

    share = layer.IndexShare(freq=4)
    got = [share.select(i, indexer, i) for i in range(10)]
    assert calls == [0, 4, 8] and got == [1, 1, 1, 1, 2, 2, 2, 2, 3, 3] and share.runs == 3
    assert [layer.IndexShare(1).select(i, indexer, i) for i in range(3)] == [4, 5, 6]
    with pytest.raises(ValueError):
        layer.IndexShare(0)


@pytest.mark.parametrize("call", ["decode", "indexer_topk"])
def test_overlapping_calls_without_a_workspace_share_no_scratch(monkeypatch, call):
    """A second call that starts while the first one's kernels are in flight -- here from inside the library call, as another
    thread or stream would -- must get scratch of its own, and none may be kept once the calls are over."""
    real_empty, spans, kept = torch.empty, [], []

    class Lib:
        def dsa_sparse_mla_decode_workspace_bytes(self, *a):
            return 4096

        def dsa_indexer_topk_workspace_bytes(self, T, S):
            return T * S * 4

        def _enter(self, ptr, nbytes):
            spans.append((ptr, ptr + nbytes))
            if len(spans) == 1:
                run()
            return 0

        def dsa_sparse_mla_decode_paged(self, *a):
            return self._enter(a[12], a[13])

        def dsa_indexer_topk(self, *a):
            return self._enter(a[13], a[14])

    def empty(*a, device=None, **kw):                  # "cuda:0" lives on the CPU here
        t = real_empty(*a, **kw)
        if t.dtype == torch.uint8:
            kept.append(weakref.ref(t))
        return t

    monkeypatch.setattr(torch, "empty", empty)
    monkeypatch.setattr(ops._lib, "load", Lib)
    monkeypatch.setattr(ops, "_need_cuda", lambda *ts: torch.device("cpu"))
    monkeypatch.setattr(ops, "_dev_index", lambda d: 0)
    monkeypatch.setattr(ops, "_on", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(ops, "_stream", lambda d: 0)
    monkeypatch.setattr(ops, "status_word", lambda d: torch.zeros(1, dtype=torch.int32))
    if call == "decode":
        q = torch.zeros(2, 16, 576, dtype=torch.bfloat16)
        cache, table = torch.zeros(64, 656, dtype=torch.uint8), torch.zeros(2, 1, dtype=torch.int32)
        run = lambda: ops.sparse_mla_decode_paged(q, cache, table, torch.zeros(2, 8, dtype=torch.int32), 0.1)
    else:
        q8 = torch.zeros(4, 64, 128).to(torch.float8_e4m3fn)
        ke = torch.ones(4, dtype=torch.int32)
        run = lambda: ops.indexer_topk(q8, q8[0], torch.ones(64), torch.ones(4, 64), None, ke, 8)
    run()
    (a0, a1), (b0, b1) = spans
    assert a1 > a0 and b1 > b0 and (a1 <= b0 or b1 <= a0)
    assert kept and all(r() is None for r in kept)

class _OnGpu(torch.Tensor):
    """A host tensor that says it lives on cuda:0: enough for the checks that a wrapper makes before it calls the library."""
    device = property(lambda self: torch.device("cuda", 0))
    is_cuda = property(lambda self: True)

    def get_device(self):
        return 0


def _decode_step_call(monkeypatch, B=4, max_ctx=1024, k=256, heads=2):
    """Arguments of ops.decode_step in its plain form (tiny caches), and the list that a stand-in for the library fills."""
    calls = []

    class Lib:
        def dsa_decode_step(self, *args):
            calls.append(args)
            return 0

    monkeypatch.setattr(ops._lib, "load", Lib)
    monkeypatch.setattr(ops, "_on", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(ops, "_stream", lambda dev: 0)
    monkeypatch.setattr(ops, "status_word", lambda dev: torch.zeros(1, dtype=torch.int32))
    pages = max_ctx // 64
    args = dict(q_fp8=torch.zeros(B, 64, 128).to(ops.FP8), weights=torch.zeros(B, 64), kcache=torch.zeros(64, 128).to(ops.FP8),
                kscale=torch.zeros(64), block_table=torch.zeros(B, pages, dtype=torch.int32),
                ctx_len=torch.full((B,), max_ctx, dtype=torch.int32), q=torch.zeros(B, heads, 576, dtype=torch.bfloat16),
                cache=torch.zeros(64, 656, dtype=torch.uint8), logits=torch.zeros(B + 1, max_ctx), idx=torch.zeros(B, k, dtype=torch.int32),
                out=torch.zeros(B, heads, 512, dtype=torch.bfloat16), workspace=torch.zeros(16, dtype=torch.uint8))
    return {n: t.as_subclass(_OnGpu) for n, t in args.items()}, dict(scale=0.07, max_ctx=max_ctx), calls


@pytest.mark.parametrize("B", [1, 4])
def test_decode_step_passes_on_the_row_pitch_that_its_logits_have(monkeypatch, B):
    """Rows further apart than max_ctx are passed on with their pitch; rows closer together than that (an expanded or overlapping
    buffer) would be written past their storage and go to the wrappers, which refuse them."""
    args, rest, calls = _decode_step_call(monkeypatch, B)
    assert ops.decode_step(**args, **rest) and len(calls) == 1
    pitch = 10                                                  # position of ld_logits in the C signature
    assert calls[0][pitch - 1] == args["logits"].data_ptr() and calls[0][pitch] == 1024
    wide = torch.zeros(B, 1500).as_subclass(_OnGpu)
    assert ops.decode_step(**{**args, "logits": wide}, **rest) and calls[1][pitch] == 1500
    for stride in (0, 256, 1023):
        bad = torch.zeros(1024 + stride * B).as_strided((B, 1024), (stride, 1))
        assert not ops.decode_step(**{**args, "logits": bad.as_subclass(_OnGpu)}, **rest)
    assert len(calls) == 2


@pytest.mark.parametrize("missing", ["logits", "workspace"])
def test_decode_step_leaves_absent_scratch_to_the_wrappers(monkeypatch, missing):
    """The wrappers allocate a logits buffer or a split workspace that is None; the one library call needs both."""
    args, rest, calls = _decode_step_call(monkeypatch)
    assert ops.decode_step(**{**args, missing: None}, **rest) is False and not calls


def _host_layer(monkeypatch, T=5):
    """A DSALayer whose selection and attention are stand-ins on the host, and the dtypes that the two were asked for / given."""
    from llmdivedeep_b200 import layer
    seen = {}

    def select(self, q, k, gate, ke, topk, dtype, w=None):
        seen["selected"], seen["w"] = dtype, w
        return torch.zeros(T, topk, dtype=dtype)

    monkeypatch.setattr(DSA.DsaIndexer, "_select", select)
    m = layer.DSALayer(hidden_size=32, q_lora_rank=16, index_n_heads=2, n_heads=1, index_topk=3, seed=0)
    m.attn.forward = lambda q, kv, idx: seen.setdefault("attended", idx)
    return m, torch.zeros(T, 32), seen


def test_layer_takes_its_own_indexers_positions_without_a_detour(monkeypatch):
    m, x, seen = _host_layer(monkeypatch)
    assert m.stages(x)["idx"].dtype == torch.int32 and seen["selected"] == torch.int32


@pytest.mark.parametrize("where", ["instance", "class"])
def test_layer_calls_a_replaced_indexer_forward_with_two_arguments(monkeypatch, where):
    m, x, seen = _host_layer(monkeypatch)
    if where == "instance":
        m.indexer.forward = lambda x, q_lora: torch.full((5, 3), 7)
    else:
        monkeypatch.setattr(DSA.DsaIndexer, "forward", lambda self, x, q_lora: torch.full((5, 3), 7))
    assert torch.equal(m.stages(x)["idx"], torch.full((5, 3), 7, dtype=torch.int32)) and seen["attended"].dtype == torch.int32


@pytest.mark.parametrize("scope", ["module", "global", "pre"])
def test_hooks_on_the_layers_indexer_see_its_int64_positions(monkeypatch, scope):
    m, x, seen = _host_layer(monkeypatch)
    outs, ins = [], []
    if scope == "module":
        h = m.indexer.register_forward_hook(lambda mod, args, out: outs.append(out.dtype))
    elif scope == "global":
        h = torch.nn.modules.module.register_module_forward_hook(lambda mod, args, out: outs.append(out.dtype) if mod is m.indexer else None)
    else:
        h = m.indexer.register_forward_pre_hook(lambda mod, args, kwargs: ins.append(kwargs), with_kwargs=True)
    try:
        assert m.stages(x)["idx"].dtype == torch.int32
    finally:
        h.remove()
    assert outs == ([] if scope == "pre" else [torch.int64]) and ins == ([{}] if scope == "pre" else [])


def test_projections_replaced_on_the_class_are_called(monkeypatch):
    """As those of a subclass or an instance are."""
    m, x, seen = _host_layer(monkeypatch)
    w = torch.full((5, 2), 0.25)
    monkeypatch.setattr(DSA.DsaIndexer, "projections", lambda self, x, q_lora: (torch.zeros(5, 2, 64), torch.zeros(5, 64), w))
    m.stages(x)
    assert seen["w"] is w


def test_pack_latent_records_answers_yes_or_no(monkeypatch):
    """Into the caller's records: True once the kernel has the call, False, with nothing done, for rows that it does not take."""
    calls = []

    class Lib:
        def dsa_pack_latent_cache(self, *args):
            calls.append(args)
            return 0

    monkeypatch.setattr(ops._lib, "load", Lib)
    monkeypatch.setattr(ops, "_on", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(ops, "_stream", lambda dev: 0)
    kv = torch.zeros(2, 576, dtype=torch.bfloat16).as_subclass(_OnGpu)
    out = torch.zeros(2, 656, dtype=torch.uint8).as_subclass(_OnGpu)
    assert ops.pack_latent_records(kv, out) is True and len(calls) == 1
    assert ops.pack_latent_records(kv.half(), out) is False and ops.pack_latent_records(kv, out[:1]) is False and len(calls) == 1


@pytest.mark.parametrize("gates", [(5, 1), (1, 2), (5, 2)])
def test_gates_shared_by_heads_or_rows_broadcast(monkeypatch, gates):
    """A replaced weights_proj may give one gate for all heads (or rows): folded by torch, as every gate once was; the kernel
    takes one for each."""
    taken = []

    def kernel(x, cos, sin, rd, il, rows, gate=None, mul=None):
        taken.append(gate is not None)
        out = x.to(ops.FP8), torch.full(x.shape[:-1], 2.0)
        return out if gate is None else (*out, torch.zeros(x.shape[:-1]))

    monkeypatch.setattr(ops, "rope_fp8_quant", kernel)
    ix = DSA.DsaIndexer(DSA.IndexerSpec("t", 32, 16, 2, 64, 32, 3), dtype=torch.bfloat16)
    x, gate = torch.randn(5, 2, 64).bfloat16(), torch.randn(gates).bfloat16()
    w = ix._rope_quant(x, 5, 2, gate)[2]
    assert taken == [gates == (5, 2)]
    if gates != (5, 2):
        assert torch.equal(w, gate.float() * 2 ** -0.5 * torch.full((5, 2), 2.0) * 64 ** -0.5)
