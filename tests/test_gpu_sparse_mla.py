"""dsa_sparse_mla_prefill / dsa_sparse_mla_decode_paged (through the C ABI) against the CPU oracle.

Floating point: bf16 inputs, bf16 tensor-core products with fp32 accumulation, the other CTA's
half of every score rounded to fp16 on its way between the pair, P rounded to bf16, bf16 output.  Tolerance (the one stated for this path): max-abs 2e-2 and mean-abs 2e-3
against the oracle's fp32 computation on the same bf16 inputs.
"""
import math
import os
import re

import pytest
import torch

from llmdivedeep_b200 import ops
from oracle import dsa_oracle as O

pytestmark = pytest.mark.gpu
MAX_ABS, MEAN_ABS = 2e-2, 2e-3


def make(T, H, S, K, seed, causal=True):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(T, H, 576, generator=g).to(torch.bfloat16)
    kv = torch.randn(S, 576, generator=g).to(torch.bfloat16)
    idx = torch.full((T, K), -1, dtype=torch.int32)
    for t in range(T):
        hi = (S - T + t + 1) if causal else S
        n = min(K, hi)
        idx[t, :n] = torch.randperm(hi, generator=g)[:n].int()
    return q, kv, idx


def check(out, ref):
    d = (out.float().cpu() - ref).abs()
    assert float(d.max()) <= MAX_ABS and float(d.mean()) <= MEAN_ABS, (float(d.max()), float(d.mean()))


@pytest.mark.parametrize("T,H,S,K", [(4, 128, 256, 64), (8, 128, 1000, 192), (6, 128, 3000, 2048), (5, 16, 500, 256),
                                     (3, 200, 400, 100), (2, 1, 130, 65), (70, 128, 200, 64), (3, 64, 5000, 1)])
def test_prefill_matches_oracle(T, H, S, K):
    q, kv, idx = make(T, H, S, K, seed=T * 3 + K)
    scale = 576 ** -0.5 * 2
    out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), scale)
    ops.check_status("cuda")
    check(out, O.sparse_mla(q.float(), kv.float(), idx, scale))


def test_short_rows_holes_and_empty_rows():
    """Causal rows shorter than K (the first tokens of a sequence), holes in the middle of the
    slot list, and a row with no valid slot at all (zeros)."""
    q, kv, idx = make(40, 128, 40, 128, seed=9)      # row t has t+1 valid slots
    idx[7, ::3] = -1
    idx[11] = -1
    out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), 0.05)
    ops.check_status("cuda")
    check(out, O.sparse_mla(q.float(), kv.float(), idx, 0.05))
    assert float(out[11].float().abs().max()) == 0.0


def test_large_scores_trigger_rescaling():
    """Scores that keep growing along the slot list force the running-maximum rescale path."""
    g = torch.Generator().manual_seed(3)
    T, H, S, K = 4, 128, 1024, 1024
    q = torch.randn(T, H, 576, generator=g).to(torch.bfloat16)
    kv = torch.randn(S, 576, generator=g)
    kv *= torch.linspace(0.1, 1.0, S).unsqueeze(1)          # later rows have larger norms
    kv = kv.to(torch.bfloat16)
    idx = torch.arange(K, dtype=torch.int32).repeat(T, 1)
    # scale 0.2: logits reach +-20 and the block maximum climbs by ~25 log2 units along the list (several rescales).
    # The other CTA's half of a score arrives as fp16 (11 significant bits), so the error of a logit grows with
    # scale * |score|; DSA's own scale is 576^-0.5 or 192^-0.5, five to three times smaller than this one.
    out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), 0.2)
    check(out, O.sparse_mla(q.float(), kv.float(), idx, 0.2))


def test_caller_supplied_out_must_be_dense_bf16_of_the_right_shape():
    q, kv, idx = make(4, 128, 256, 64, seed=2)
    q, kv, idx = q.cuda(), kv.cuda(), idx.cuda()
    good = torch.empty(4, 128, 512, dtype=torch.bfloat16, device="cuda")
    assert ops.sparse_mla_prefill(q, kv, idx, 0.05, out=good) is good
    for bad in (torch.empty(4, 128, 512, dtype=torch.float16, device="cuda"),
                torch.empty(4, 128, 256, dtype=torch.bfloat16, device="cuda"),
                torch.empty(4, 128, 1024, dtype=torch.bfloat16, device="cuda")[:, :, ::2]):
        with pytest.raises(ops.DsaError, match="out must be"):
            ops.sparse_mla_prefill(q, kv, idx, 0.05, out=bad)


def test_out_of_range_index_is_skipped_and_flagged():
    q, kv, idx = make(2, 128, 100, 64, seed=1, causal=False)
    bad = idx.clone()
    bad[0, 5] = 100                                          # == S_kv
    out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), bad.cuda(), 0.05)
    with pytest.raises(ops.DsaError, match="out of range"):
        ops.check_status("cuda")
    ref_idx = idx.clone()
    ref_idx[0, 5] = -1
    check(out, O.sparse_mla(q.float(), kv.float(), ref_idx, 0.05))


def test_deterministic_and_permutation_invariant():
    q, kv, idx = make(3, 128, 2000, 512, seed=5, causal=False)
    a = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), 0.04)
    b = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), 0.04)
    assert torch.equal(a, b)
    perm = torch.randperm(512)
    c = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx[:, perm].contiguous().cuda(), 0.04)
    assert float((a.float() - c.float()).abs().max()) <= 1e-2    # softmax does not depend on slot order


def test_full_size_row_equals_dense_attention():
    """Bench-size shape property: with every key of a 2048-key context selected, sparse MLA is
    dense softmax attention (checked against torch on the GPU in fp32)."""
    g = torch.Generator().manual_seed(8)
    T, H, S = 16, 128, 2048
    q = torch.randn(T, H, 576, generator=g).to(torch.bfloat16).cuda()
    kv = torch.randn(S, 576, generator=g).to(torch.bfloat16).cuda()
    idx = torch.stack([torch.randperm(S, generator=g) for _ in range(T)]).int().cuda()
    scale = 192 ** -0.5
    out = ops.sparse_mla_prefill(q, kv, idx, scale)
    p = torch.softmax(torch.einsum("thd,sd->ths", q.float(), kv.float()) * scale, dim=-1)
    ref = torch.einsum("ths,sd->thd", p, kv.float()[:, :512])
    d = (out.float() - ref).abs()
    assert float(d.max()) <= MAX_ABS and float(d.mean()) <= MEAN_ABS


@pytest.mark.parametrize("B,H,P,K", [(4, 128, 8, 200), (3, 128, 40, 2048), (2, 32, 4, 64)])
def test_decode_paged_matches_oracle(B, H, P, K):
    g = torch.Generator().manual_seed(B * 11 + K)
    kv = torch.randn(B * P * 64, 576, generator=g).to(torch.bfloat16)
    cache = O.pack_latent_cache(kv)
    table = torch.randperm(B * P, generator=g).int().view(B, P)
    idx = torch.stack([torch.randperm(P * 64, generator=g)[:K] for _ in range(B)]).int()
    idx[B - 1, K // 2:] = -1
    q = torch.randn(B, H, 576, generator=g).to(torch.bfloat16)
    out = ops.sparse_mla_decode_paged(q.cuda(), cache.cuda(), table.cuda(), idx.cuda(), 0.06)
    ops.check_status("cuda")
    check(out, O.sparse_mla_decode_paged(q.float(), cache, table, idx, 0.06, round_bf16=True))


def test_decode_holes_and_odd_block_counts():
    """Holes inside the slot list (empty slots are zero-filled rows with a cleared validity bit) and slot lists of one,
    three and five 64-key blocks: a gather warp alternates between two raw stages of its own."""
    for K in (40, 130, 300):
        g = torch.Generator().manual_seed(K)
        B, H, P = 3, 128, 6
        kv = torch.randn(B * P * 64, 576, generator=g).to(torch.bfloat16)
        cache = O.pack_latent_cache(kv)
        table = torch.randperm(B * P, generator=g).int().view(B, P)
        idx = torch.stack([torch.randperm(P * 64, generator=g)[:K] for _ in range(B)]).int()
        idx[0, ::3] = -1
        idx[1, 1::2] = -1
        idx[2, : K // 2] = -1                                  # leading blocks empty, trailing ones used
        q = torch.randn(B, H, 576, generator=g).to(torch.bfloat16)
        out = ops.sparse_mla_decode_paged(q.cuda(), cache.cuda(), table.cuda(), idx.cuda(), 0.06)
        ops.check_status("cuda")
        check(out, O.sparse_mla_decode_paged(q.float(), cache, table, idx, 0.06, round_bf16=True))


def test_decode_bad_page_is_flagged():
    g = torch.Generator().manual_seed(2)
    kv = torch.randn(4 * 64, 576, generator=g).to(torch.bfloat16)
    cache = O.pack_latent_cache(kv)
    table = torch.tensor([[0, 1, 2, 9]], dtype=torch.int32)      # page 9 does not exist
    idx = torch.arange(256, dtype=torch.int32).view(1, 256)
    q = torch.randn(1, 128, 576, generator=g).to(torch.bfloat16)
    out = ops.sparse_mla_decode_paged(q.cuda(), cache.cuda(), table.cuda(), idx.cuda(), 0.06)
    with pytest.raises(ops.DsaError, match="out of range"):
        ops.check_status("cuda")
    ok = idx.clone()
    ok[0, 192:] = -1
    table[0, 3] = 3
    check(out, O.sparse_mla_decode_paged(q.float(), cache, table, ok, 0.06, round_bf16=True))


def test_decode_split_parts_match_the_single_part_path():
    """Few sequences with long slot lists take the split path (parts merged by a second kernel);
    a workspace too small for it forces the single-part path.  Both must agree."""
    from llmdivedeep_b200 import _lib
    B, H, P, K = 2, 128, 40, 2048
    g = torch.Generator().manual_seed(77)
    kv = torch.randn(B * P * 64, 576, generator=g).to(torch.bfloat16)
    cache = O.pack_latent_cache(kv).cuda()
    table = torch.randperm(B * P, generator=g).int().view(B, P).cuda()
    idx = torch.stack([torch.randperm(P * 64, generator=g)[:K] for _ in range(B)]).int()
    idx[1, 300:1500] = -1                                  # whole parts of sequence 1 are empty
    idx = idx.cuda()
    q = torch.randn(B, H, 576, generator=g).to(torch.bfloat16).cuda()
    assert _lib.load().dsa_sparse_mla_decode_workspace_bytes(B, H, K) > 0
    split = ops.sparse_mla_decode_paged(q, cache, table, idx, 0.06)
    single = ops.sparse_mla_decode_paged(q, cache, table, idx, 0.06, workspace=torch.empty(16, dtype=torch.uint8, device="cuda"))
    ops.check_status("cuda")
    assert float((split.float() - single.float()).abs().max()) <= 1e-2
    check(split, O.sparse_mla_decode_paged(q.float().cpu(), cache.cpu(), table.cpu(), idx.cpu(), 0.06, round_bf16=True))


@pytest.mark.parametrize("K", [1, 63, 64, 65, 128, 191, 193, 320, 321, 385, 640, 705])
@pytest.mark.parametrize("H", [128, 16])
def test_prefill_block_counts(H, K):
    """Slot lists around whole numbers of 64-key blocks: one and two blocks (one warp set has nothing to do), the number
    of KV buffers (five), and beyond."""
    q, kv, idx = make(3, H, 1500, K, seed=K + H, causal=False)
    out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), 0.06)
    ops.check_status("cuda")
    check(out, O.sparse_mla(q.float(), kv.float(), idx, 0.06))


@pytest.mark.parametrize("T,H", [(4096, 16), (2048, 128)])
def test_prefill_whole_output_and_repeats(T, H):
    """Many waves of CTA pairs, every output value: against float64 on the GPU, and bit for bit the same in every run (a
    hand-over between the two CTAs that comes too early shows here as a few wrong tokens in ten thousand)."""
    g = torch.Generator(device="cuda").manual_seed(T + H)
    S, K, scale = 8192, 1024, 192 ** -0.5
    kv = torch.randn(S, 576, device="cuda", generator=g).to(torch.bfloat16)
    q = torch.randn(T, H, 576, device="cuda", generator=g).to(torch.bfloat16)
    idx = torch.rand(T, S, device="cuda", generator=g).topk(K, dim=-1).indices.int()
    out = ops.sparse_mla_prefill(q, kv, idx, scale)
    for _ in range(12):
        assert torch.equal(ops.sparse_mla_prefill(q, kv, idx, scale), out)
    ops.check_status("cuda")
    worst = 0.0
    for a in range(0, T, 64):
        rows = kv[idx[a:a + 64].long()].double()
        p = (torch.bmm(q[a:a + 64].double(), rows.transpose(1, 2)) * scale).softmax(-1)
        worst = max(worst, float((out[a:a + 64].double() - torch.bmm(p, rows[..., :512])).abs().max()))
    assert worst <= MAX_ABS, worst


@pytest.mark.parametrize("B,H,K", [(74, 16, 512), (75, 128, 600), (80, 16, 2048), (111, 16, 700), (150, 40, 513), (37, 200, 640)])
def test_decode_rounds_of_queries_with_a_split_remainder(B, H, K):
    """Batches around whole rounds of CTA pairs: the queries of the last round are cut into parts and merged, the others
    are not; both against the oracle, and against the call whose workspace is too small to split anything."""
    g = torch.Generator().manual_seed(B + K)
    P = 40
    cache = O.pack_latent_cache(torch.randn(B * P * 64, 576, generator=g).to(torch.bfloat16))
    table = torch.randperm(B * P, generator=g).int().view(B, P)
    idx = torch.rand(B, P * 64, generator=g).topk(K, dim=-1).indices.int()
    idx[B - 1, K // 3:] = -1                               # some parts of the last query are empty
    idx[0, ::5] = -1
    q = torch.randn(B, H, 576, generator=g).to(torch.bfloat16)
    args = (q.cuda(), cache.cuda(), table.cuda(), idx.cuda(), 0.06)
    out = ops.sparse_mla_decode_paged(*args)
    one = ops.sparse_mla_decode_paged(*args, workspace=torch.empty(16, dtype=torch.uint8, device="cuda"))
    ops.check_status("cuda")
    assert float((out.float() - one.float()).abs().max()) <= MAX_ABS
    rows = [0, 1, B // 2, B - 2, B - 1]
    check(out[rows], O.sparse_mla_decode_paged(q[rows].float(), cache, table[rows], idx[rows], 0.06, round_bf16=True))


def _holes(idx, g):
    """Every second row: random empty slots, an empty block now and then, a tail of its own length."""
    T, K = idx.shape
    idx[::2].masked_fill_(torch.rand((T + 1) // 2, K, device="cuda", generator=g) < 0.2, -1)
    idx[::4, 64:128] = -1
    length = torch.randint(1, K + 1, (T, 1), device="cuda", generator=g)
    idx[::2].masked_fill_(torch.arange(K, device="cuda") >= length[::2], -1)
    return idx


@pytest.mark.parametrize("form", ["prefill", "decode"])
def test_ragged_lists_and_decode_repeat_bit_for_bit(form):
    """The hand-over between the two CTAs of a pair, where the masks of holes and ragged tails come between reading a tile and
    releasing it, and in the decode kernel: many waves of pairs, the same bits in every run, a sample against float64."""
    g = torch.Generator(device="cuda").manual_seed(71)
    T, H, K, P, scale = 1200, 128, 1024, 24, 192 ** -0.5
    q = torch.randn(T, H, 576, device="cuda", generator=g).to(torch.bfloat16)
    idx = _holes(torch.rand(T, P * 64, device="cuda", generator=g).topk(K, dim=-1).indices.int(), g)
    if form == "prefill":
        kv = torch.randn(P * 64, 576, device="cuda", generator=g).to(torch.bfloat16)
        run = lambda: ops.sparse_mla_prefill(q, kv, idx, scale)
        rows_of = lambda t, pos: kv[pos].double()
    else:
        records = O.pack_latent_cache(torch.randn(200 * 64, 576, generator=torch.Generator().manual_seed(72)).to(torch.bfloat16)).cuda()
        table = torch.randint(0, 200, (T, P), device="cuda", generator=g).int()
        run = lambda: ops.sparse_mla_decode_paged(q, records, table, idx, scale)

        def rows_of(t, pos):
            rec = records[table[t].long()[pos // 64] * 64 + pos % 64]
            lat = rec[:, :512].contiguous().view(torch.float8_e4m3fn).float().view(-1, 4, 128)
            lat = (lat * rec[:, 512:528].contiguous().view(torch.float32).unsqueeze(-1)).view(-1, 512).to(torch.bfloat16)
            return torch.cat((lat, rec[:, 528:].contiguous().view(torch.bfloat16)), -1).double()

    out = run()
    for _ in range(12):
        assert torch.equal(run(), out)
    ops.check_status("cuda")
    for t in range(0, T, 7):
        rows = rows_of(t, idx[t][idx[t] >= 0].long())
        ref = ((q[t].double() @ rows.T) * scale).softmax(-1) @ rows[:, :512] if rows.shape[0] else torch.zeros_like(out[t]).double()
        assert float((out[t].double() - ref).abs().max()) <= MAX_ABS, t


def test_decode_parts_are_weighted_with_the_sums_of_their_own_half():
    """The score of every key is about 6144 and comes from the second CTA's half of the contraction alone, so that CTA has it
    unrounded while the other receives it in fp16 (spacing 4, two units of the scaled score).  Output columns 256.. are the
    second CTA's: exact to bf16 whether the list is split or not, if its parts are weighted with its own sums."""
    B, H, P, K, scale = 2, 128, 40, 2048, 0.5
    g = torch.Generator().manual_seed(31)
    kv = torch.randn(B * P * 64, 576, generator=g)
    kv[:, 512:544] = 0
    kv[:, 544:] = 24
    cache = O.pack_latent_cache(kv.to(torch.bfloat16))
    table = torch.randperm(B * P, generator=g).int().view(B, P)
    idx = torch.stack([torch.randperm(P * 64, generator=g)[:K] for _ in range(B)]).int()
    q = torch.zeros(B, H, 576)
    q[:, :, 256:512] = torch.randn(B, H, 256, generator=g) / 2
    q[:, :, 544:] = 8
    q = q.to(torch.bfloat16)
    ref = O.sparse_mla_decode_paged(q.float(), cache, table, idx, scale, round_bf16=True)[..., 256:]
    args = (q.cuda(), cache.cuda(), table.cuda(), idx.cuda(), scale)
    split = ops.sparse_mla_decode_paged(*args)
    single = ops.sparse_mla_decode_paged(*args, workspace=torch.empty(16, dtype=torch.uint8, device="cuda"))
    ops.check_status("cuda")
    check(single[..., 256:], ref)
    check(split[..., 256:], ref)


@pytest.mark.parametrize("form", ["prefill", "decode"])
@pytest.mark.parametrize("K", [32, 33, 64, 700, 929, 1000, 1824, 2048])
def test_last_used_slot_anywhere_in_the_list(form, K):
    """The last used slot decides how many blocks a row walks: at both ends of the list, around its last 32 slots and around
    the 896 slots that the threads of a CTA look at together; alone, and behind holes."""
    last = sorted({p for p in (0, 31, 32, 63, 64, 863, 864, 895, 896, 897, 1791, 1792, K - 66, K - 34, K - 33, K - 32, K - 31, K - 1)
                   if 0 <= p < K})
    g = torch.Generator().manual_seed(K)
    T, H, P = 2 * len(last) + 1, 16, 34
    idx = torch.full((T, K), -1, dtype=torch.int32)
    for i, p in enumerate(last):                       # row T - 1 stays empty
        idx[2 * i, p] = 5 + i
        idx[2 * i + 1, :p + 1] = torch.randperm(P * 64, generator=g)[:p + 1].int()
        idx[2 * i + 1, 1:p:3] = -1
    q = torch.randn(T, H, 576, generator=g).to(torch.bfloat16)
    kv = torch.randn(P * 64, 576, generator=g).to(torch.bfloat16)
    if form == "prefill":
        out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), 0.06)
        ref = O.sparse_mla(q.float(), kv.float(), idx, 0.06)
    else:                                              # T < 74: the lists are cut into parts
        cache, table = O.pack_latent_cache(kv), torch.arange(P, dtype=torch.int32).repeat(T, 1)
        out = ops.sparse_mla_decode_paged(q.cuda(), cache.cuda(), table.cuda(), idx.cuda(), 0.06)
        ref = O.sparse_mla_decode_paged(q.float(), cache, table, idx, 0.06, round_bf16=True)
    ops.check_status("cuda")
    check(out, ref)
    assert float(out[T - 1].float().abs().max()) == 0.0


@pytest.mark.parametrize("H", [1, 8, 15, 16, 17, 31, 32])
@pytest.mark.parametrize("T,K", [(1, 1), (5, 64), (150, 65), (200, 177), (160, 2048)])
def test_prefill_of_few_heads(H, T, K):
    """Up to 32 heads go through the kernel with scores and output transposed (tiles of 16 and 32 heads): head counts around the
    tiles, blocks and their remainders, more tokens than CTAs, holes, empty lists, scores wide enough to raise the references.
    (The kernel of more heads sends partial scores as fp16: its bound at q x 8 also holds 2^-11 |partial| of the scores.)"""
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + T + K)
    S, scale = 2500, 192 ** -0.5
    kv = torch.randn(S, 576, device="cuda", generator=g).to(torch.bfloat16)
    for wide in (1, 8):
        q = (torch.randn(T, H, 576, device="cuda", generator=g) * wide).to(torch.bfloat16)
        idx = _holes(torch.rand(T, S, device="cuda", generator=g).topk(K, dim=-1).indices.int(), g)
        idx[T // 2] = -1
        out = ops.sparse_mla_prefill(q, kv, idx, scale)
        assert torch.equal(ops.sparse_mla_prefill(q, kv, idx, scale), out)
        # a row does not depend on the call's other rows
        assert torch.equal(ops.sparse_mla_prefill(q[-1:].contiguous(), kv, idx[-1:].contiguous(), scale), out[-1:])
        ops.check_status("cuda")
        rows = kv[idx.clamp_min(0).long()].double()
        s = (torch.bmm(q.double(), rows.transpose(1, 2)) * scale).masked_fill((idx < 0).unsqueeze(1), float("-inf"))
        ref = torch.bmm(s.softmax(-1).nan_to_num(0.0), rows[..., :512])
        # bf16 P and outputs: 2^-9 of the largest value each (|v| < 6), and their sums
        assert float((out.double() - ref).abs().max()) <= 6 * 2 ** -8 + 2 ** -9


def test_prefill_of_few_heads_flags_positions_out_of_range():
    q, kv, idx = make(9, 16, 300, 130, seed=4, causal=False)
    bad = idx.clone()
    bad[3, 70], bad[8, 129] = 300, 2 ** 31 - 1
    out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), bad.cuda(), 0.06)
    with pytest.raises(ops.DsaError, match="out of range"):
        ops.check_status("cuda")
    skipped = torch.where(bad >= 300, torch.full_like(bad, -1), bad)
    check(out, O.sparse_mla(q.float(), kv.float(), skipped, 0.06))


def _climbing(T, H, K, seed):
    """Rows whose scores climb from block to block of the list by far more than the softmax reference may lag.  In log2 units
    the blocks lie at 0, 31.5, 33, 66, 97.5, ...: where the reference is raised, the block before may still have a third of
    the new one's weight, so that the factor shows in the output.  A head takes them once, by half, not at all, or backwards.
    The levels (half-integers up to 1408 before the scale) come from the second CTA's rope dims, the random part from the
    first CTA's latent values: the level is exact in fp16 on its way between the two."""
    g = torch.Generator().manual_seed(seed)
    level = [0.0]
    for b in range((K - 1) // 64):
        level.append(level[-1] + 2 * (31.5, 1.5, 33.0)[b % 3])
    scale = 0.5 * math.log(2.0)                                # log2 units are half the raw score
    kv = torch.randn(K, 576, generator=g)
    lv = torch.tensor(level).repeat_interleave(64)[:K]
    kv[:, 512:] = 0
    kv[:, 544], kv[:, 545] = torch.div(lv, 8, rounding_mode="floor"), lv % 8
    q = torch.zeros(T, H, 576)
    q[:, :, :256] = torch.randn(T, H, 256, generator=g) / 16
    c = torch.tensor([1.0, 0.5, 1.0, 0.0, 1.0, -1.0]).repeat(H)[:H]
    q[:, :, 544], q[:, :, 545] = 8 * c, c
    idx = torch.empty(T, K, dtype=torch.int32)
    for t in range(T):
        for b in range(0, K, 64):
            n = min(64, K - b)
            idx[t, b:b + n] = b + torch.randperm(n, generator=g).int()
    return q.to(torch.bfloat16), kv.to(torch.bfloat16), idx, scale


def _raises(q, kv, idx, scale, first=0, last=None):
    """How often the reference of each row and head is raised after its first block, walking slots [first, last)."""
    src = open(os.path.join(os.path.dirname(ops.__file__), "csrc", "dsa_common.cuh")).read()
    lag = float(re.search(r"kMaxRaise = ([0-9.]+)f", src).group(1))
    s = torch.einsum("thd,tkd->thk", q.float(), kv.float()[idx.long()])[..., first:last] * (scale / math.log(2.0))
    m, n = torch.full(s.shape[:2], -math.inf), torch.zeros(s.shape[:2], dtype=torch.int32)
    for b in range(0, s.shape[2], 64):
        top = s[..., b:b + 64].amax(-1)
        up = top - m > lag
        n += up if b else 0
        m = torch.where(up, top, m)
    return n


@pytest.mark.parametrize("H,K", [(64, 1024), (128, 2048), (200, 700), (16, 2048), (32, 1000), (7, 321)])
def test_prefill_scores_that_outgrow_the_reference_many_times(H, K):
    q, kv, idx, scale = _climbing(3, H, K, seed=H + K)
    assert int(_raises(q, kv, idx, scale)[:, 0].min()) >= 2
    out = ops.sparse_mla_prefill(q.cuda(), kv.cuda(), idx.cuda(), scale)
    ops.check_status("cuda")
    check(out, O.sparse_mla(q.float(), kv.float(), idx, scale))


@pytest.mark.parametrize("H", [64, 128, 200])
@pytest.mark.parametrize("form", ["split", "whole"])
def test_decode_scores_that_outgrow_the_reference_many_times(form, H):
    """In a list that one pair walks, and in the parts of a split one (256 slots: the reference is raised in each)."""
    B, K = 2, 2048
    q, kv, idx, scale = _climbing(B, H, K, seed=H)
    for first in range(0, K, 256):
        assert int(_raises(q, kv, idx, scale, first, first + 256)[:, 0].min()) >= 1
    assert int(_raises(q, kv, idx, scale)[:, 0].min()) >= 2
    cache = O.pack_latent_cache(kv)
    table = torch.arange(K // 64, dtype=torch.int32).repeat(B, 1)
    ws = torch.empty(16, dtype=torch.uint8, device="cuda") if form == "whole" else None
    out = ops.sparse_mla_decode_paged(q.cuda(), cache.cuda(), table.cuda(), idx.cuda(), scale, workspace=ws)
    ops.check_status("cuda")
    check(out, O.sparse_mla_decode_paged(q.float(), cache, table, idx, scale, round_bf16=True))


@pytest.mark.parametrize("H", [1, 16, 17, 32])
@pytest.mark.parametrize("K", [129, 256, 257, 320, 700, 2048])
def test_rows_of_few_heads_have_the_same_bits_in_calls_of_any_size(H, K):
    """Up to one row for every two SMs a row's list is dealt to two CTAs, beyond that one CTA walks both halves: the same bits
    (a row may be computed by another rank, or in another chunk), over lists that end anywhere, holes and empty rows."""
    T, P = 160, 40
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    g = torch.Generator(device="cuda").manual_seed(H + K)
    kv = torch.randn(P * 64, 576, device="cuda", generator=g).to(torch.bfloat16)
    q = torch.randn(T, H, 576, device="cuda", generator=g).to(torch.bfloat16)
    idx = _holes(torch.rand(T, P * 64, device="cuda", generator=g).topk(K, dim=-1).indices.int(), g)
    for t, n in enumerate((0, 1, 64, 65, 128, 129, 192, 193, 256, 257, 321, 1024, 1025)):
        idx[2 * t, min(n, K):] = -1
    run = lambda a, b: ops.sparse_mla_prefill(q[a:b], kv, idx[a:b], 0.06)
    out = run(0, T)
    for a, n in ((0, 1), (0, pairs), (T - pairs, pairs), (5, pairs - 1), (3, pairs + 1)):
        for _ in range(3):
            assert torch.equal(run(a, a + n), out[a:a + n]), (a, n)
    ops.check_status("cuda")
    check(out, O.sparse_mla(q.float().cpu(), kv.float().cpu(), idx.cpu(), 0.06))


@pytest.mark.parametrize("H", [16, 32])
def test_halves_of_a_list_are_weighted_by_their_own_references(H):
    """Scores that climb by hundreds of log2 units along the list, fall, or stay: one CTA to a row and two, the same bits."""
    q, kv, idx, scale = (x.cuda() if torch.is_tensor(x) else x for x in _climbing(100, H, 1100, seed=H))
    out = ops.sparse_mla_prefill(q, kv, idx, scale)
    assert torch.equal(ops.sparse_mla_prefill(q[:40], kv, idx[:40], scale), out[:40])
    ops.check_status("cuda")
    check(out, O.sparse_mla(q.float().cpu(), kv.float().cpu(), idx.cpu(), scale))
