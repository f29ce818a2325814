"""dsa_topk_select (through the C ABI) against torch.topk / exact rules. Index work: bit-exact."""
import pytest
import torch

from llmdivedeep_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _sets_equal(x, idx, ks, ke, k):
    T = x.shape[0]
    for t in range(T):
        lo = int(ks[t]) if ks is not None else 0
        hi = int(ke[t]) if ke is not None else x.shape[1]
        kk = min(k, max(hi - lo, 0))
        got = idx[t].tolist()
        assert all(v == -1 for v in got[kk:]), f"row {t}: padding"
        if kk:
            ref = set((x[t, lo:hi].topk(kk).indices + lo).tolist())
            assert set(got[:kk]) == ref, f"row {t}"


@pytest.mark.parametrize("T,S,k", [(8, 1000, 16), (16, 4096, 256), (8, 65536, 2048), (4, 131072, 2048),
                                   (5, 5000, 2048), (3, 2049, 2048), (7, 300, 1), (2, 65537, 512)])
def test_random_rows_match_torch_topk(T, S, k):
    g = torch.Generator(device=DEV).manual_seed(S * 31 + k)
    x = torch.randn(T, S, device=DEV, generator=g)
    ke = torch.randint(S // 2, S + 1, (T,), device=DEV, dtype=torch.int32, generator=g)
    ks = torch.randint(0, max(S // 4, 1), (T,), device=DEV, dtype=torch.int32, generator=g)
    idx = ops.topk_select(x, k, ks, ke)
    _sets_equal(x, idx, ks, ke, k)
    assert torch.equal(idx, ops.topk_select(x, k, ks, ke)), "not deterministic"
    idx = ops.topk_select(x, k)            # no window
    _sets_equal(x, idx, None, None, k)


def test_short_windows_pad_with_minus_one():
    x = torch.randn(4, 512, device=DEV)
    ks = torch.tensor([0, 10, 500, 300], dtype=torch.int32, device=DEV)
    ke = torch.tensor([0, 13, 512, 200], dtype=torch.int32, device=DEV)   # empty, 3, 12, inverted
    idx = ops.topk_select(x, 16, ks, ke).cpu()
    assert idx[0].tolist() == [-1] * 16
    assert idx[1].tolist() == [10, 11, 12] + [-1] * 13
    assert idx[2].tolist() == list(range(500, 512)) + [-1] * 4
    assert idx[3].tolist() == [-1] * 16


def test_all_equal_rows_take_lowest_columns():
    x = torch.full((3, 10000), 2.5, device=DEV)
    idx = ops.topk_select(x, 2048)
    assert torch.equal(idx.sort(dim=1).values, torch.arange(2048, device=DEV, dtype=torch.int32).expand(3, -1))


def test_heavy_ties_break_towards_lower_columns():
    g = torch.Generator(device=DEV).manual_seed(5)
    x = torch.randint(0, 8, (4, 30000), device=DEV, generator=g).float()
    x[:, ::7] *= -1.0
    idx = ops.topk_select(x, 2048).long()
    for t in range(4):
        sel = torch.zeros(30000, dtype=torch.bool, device=DEV)
        sel[idx[t]] = True
        assert int(sel.sum()) == 2048
        thr = x[t][sel].min()
        assert x[t][~sel].max() <= thr
        tie = (x[t] == thr).nonzero().flatten()
        n_tie = int(sel[tie].sum())
        assert bool(sel[tie[:n_tie]].all()) and not bool(sel[tie[n_tie:]].any())


def test_special_values_and_signs():
    x = torch.randn(2, 4096, device=DEV)
    x[0, 100] = float("inf")
    x[0, 200:300] = float("-inf")
    x[1] = -x[1].abs() - 1.0            # all negative
    x[1, 7] = -0.0
    x[1, 9] = 0.0
    idx = ops.topk_select(x, 64)
    _sets_equal(x, idx, None, None, 64)
    assert 100 in idx[0].tolist() and 9 in idx[1].tolist() and 7 in idx[1].tolist()


def test_unaligned_leading_dimension_uses_scalar_loads():
    base = torch.randn(6, 1001, device=DEV)
    x = base[:, :999]                    # ld = 1001: rows are not 16-byte aligned
    idx = ops.topk_select(x, 50)
    _sets_equal(x, idx, None, None, 50)


def test_many_candidates_in_one_bin_takes_extra_passes():
    # values so close together that the threshold bin of the first pass overflows
    # the in-shared-memory finish (more than 2048 candidates share 12 key bits)
    g = torch.Generator(device=DEV).manual_seed(9)
    x = 1.0 + torch.rand(3, 50000, device=DEV, generator=g) * 1e-3
    idx = ops.topk_select(x, 2048)
    _sets_equal(x, idx, None, None, 2048)
    x = 1.0 + torch.rand(2, 50000, device=DEV, generator=g) * 1e-6   # few distinct floats, massive ties
    idx = ops.topk_select(x, 2048).long()
    for t in range(2):
        sel = torch.zeros(50000, dtype=torch.bool, device=DEV)
        sel[idx[t]] = True
        assert int(sel.sum()) == 2048 and x[t][~sel].max() <= x[t][sel].min()


def test_full_size_row_property():
    """Bench-size rows: selected minimum >= unselected maximum, count == k."""
    T, S, k = 64, 131072, 2048
    x = torch.randn(T, S, device=DEV)
    idx = ops.topk_select(x, k).long()
    sel = torch.zeros(T, S, dtype=torch.bool, device=DEV)
    sel.scatter_(1, idx, True)
    assert bool((sel.sum(1) == k).all())
    lo_sel = torch.where(sel, x, torch.full_like(x, float("inf"))).amin(1)
    hi_uns = torch.where(sel, torch.full_like(x, float("-inf")), x).amax(1)
    assert bool((lo_sel >= hi_uns).all())


def _two_pass(x, k, ks=None, ke=None):
    """The same call through the test hook that keeps every row on the two-pass path."""
    from llmdivedeep_b200 import _lib
    T, S = x.shape
    out = torch.empty(T, k, dtype=torch.int32, device=x.device)
    _lib.check(_lib.load().dsa_test_topk_select_two_pass(
        x.data_ptr(), x.stride(0), None if ks is None else ks.data_ptr(), None if ke is None else ke.data_ptr(),
        T, S, k, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return out


def _adversarial_rows(S, g):
    """Rows built to mislead a sample taken as one 128-column block in every 16: a ramp, the large
    values packed into few blocks, a two-level row with more ties than the candidate capacity, a
    near-constant row, and a row whose large values sit exactly in the sampled blocks."""
    rows = [torch.randn(S, device=DEV, generator=g),
            torch.arange(S, device=DEV, dtype=torch.float32),
            -torch.arange(S, device=DEV, dtype=torch.float32)]
    r = torch.randn(S, device=DEV, generator=g)
    r[4096:4096 + 3000] += 100.0                              # contiguous spike wider than k
    rows.append(r)
    r = torch.zeros(S, device=DEV)
    r[torch.randperm(S, device=DEV, generator=g)[:6000]] = 1.0   # 6000 tied maxima
    rows.append(r)
    rows.append(torch.full((S,), 3.0, device=DEV) + 1e-7 * torch.randn(S, device=DEV, generator=g))
    r = torch.randn(S, device=DEV, generator=g)
    blk = torch.arange(S, device=DEV) // 128
    r[(blk % 16) == 8] += 6.0                                 # only the sampled blocks are large
    rows.append(r)
    r = torch.randn(S, device=DEV, generator=g)
    r[(blk % 16) == 8] -= 6.0                                 # the sampled blocks are small
    rows.append(r)
    return torch.stack(rows)


@pytest.mark.parametrize("S,k", [(65536, 2048), (131072, 2048), (16384, 2048), (40000, 512), (300000, 2048)])
def test_sampled_pass_equals_two_pass_on_adversarial_rows(S, k):
    g = torch.Generator(device=DEV).manual_seed(S + k)
    x = _adversarial_rows(S, g)
    a = ops.topk_select(x, k)
    b = _two_pass(x, k)
    assert torch.equal(a.sort(dim=1).values, b.sort(dim=1).values)
    _sets_equal_with_ties(x, a, k)
    T = x.shape[0]
    # the output of a row does not depend on how many rows the call has
    many = ops.topk_select(x.repeat(10, 1), k)
    assert torch.equal(many[:T], a) and torch.equal(many[-T:], a)
    ks = torch.randint(0, S // 8, (T,), device=DEV, dtype=torch.int32, generator=g)
    ke = torch.randint(S - S // 8, S + 1, (T,), device=DEV, dtype=torch.int32, generator=g)
    a = ops.topk_select(x, k, ks, ke)
    assert torch.equal(a, ops.topk_select(x, k, ks, ke)), "not deterministic"
    assert torch.equal(a.sort(dim=1).values, _two_pass(x, k, ks, ke).sort(dim=1).values)


def _sets_equal_with_ties(x, idx, k):
    """Exact rule: everything above the k-th value is selected, the rest are the lowest columns equal to it."""
    for t in range(x.shape[0]):
        row = x[t]
        kth = row.topk(k).values[-1]
        above = (row > kth).nonzero().flatten()
        tied = (row == kth).nonzero().flatten()[: k - above.numel()]
        want = torch.cat([above, tied]).sort().values
        assert torch.equal(idx[t].long().sort().values, want), f"row {t}"


@pytest.mark.parametrize("n", [257, 2047, 4092, 4093, 4096, 4097, 8188, 8189, 8192, 12000, 16384])
@pytest.mark.parametrize("k", [1, 256, 2048])
def test_row_lengths_around_the_changes_of_path(n, k):
    """Rows kept in registers (one and two chunks of 4096 columns), read again, or staged behind a sample: lengths at the edges,
    windows that start inside a float4, calls of few rows (a larger CTA) and of many.  Sets against torch.topk with the tie rule,
    the same output, order included, whatever the number of rows, and against the two-pass path."""
    g = torch.Generator(device=DEV).manual_seed(n + k)
    rows = [torch.randn(n + 3, device=DEV, generator=g), torch.randn(n + 3, device=DEV, generator=g).exp() * -1,
            torch.randint(0, 50, (n + 3,), device=DEV, generator=g).float(), torch.full((n + 3,), -1.5, device=DEV),
            1e30 * torch.randn(n + 3, device=DEV, generator=g) ** 9]
    x = torch.zeros(len(rows), (n + 6) // 4 * 4, device=DEV)
    x[:, :n + 3] = torch.stack(rows)
    for lo in (0, 1, 3):
        ks = torch.full((len(rows),), lo, dtype=torch.int32, device=DEV)
        ke = ks + n
        a = ops.topk_select(x, min(k, n), ks, ke)
        _sets_equal_with_ties(x[:, lo:lo + n], a - lo, min(k, n))
        assert torch.equal(a.sort(1).values, _two_pass(x, min(k, n), ks, ke).sort(1).values)
        many = ops.topk_select(x.repeat(40, 1), min(k, n), ks.repeat(40), ke.repeat(40))
        assert torch.equal(many[:len(rows)], a) and torch.equal(many[-len(rows):], a)


@pytest.mark.parametrize("n", [3000, 6000, 9000, 40000])
def test_nan_and_infinities_keep_the_order_of_the_bits(n):
    """A NaN counts by its bits: above +inf with the sign bit clear, below -inf with it set; the oracle is the order-preserving
    map of the bit patterns to integers, lower column first among equals."""
    g = torch.Generator(device=DEV).manual_seed(n)
    x = torch.randn(6, n, device=DEV, generator=g)
    nan = torch.tensor([0x7fc00000, -0x400000], dtype=torch.int32, device=DEV).view(torch.float32)
    x[0, 5::97] = nan[0]
    x[1, 7::89] = nan[1]
    x[2, 11::101] = float("inf")
    x[3, 3::2] = float("-inf")
    x[4, ::3], x[4, 1::3] = nan[1], nan[0]
    x[5, 0] = 3e38
    bits = x.view(torch.int32).long()
    key = torch.where(bits < 0, -(bits & 0x7fffffff) - 1, bits)
    for k in (40, 2048):
        got = ops.topk_select(x, k)
        assert torch.equal(got, ops.topk_select(x.repeat(60, 1), k)[:6])
        for t in range(6):
            want = sorted(range(n), key=lambda c, kt=key[t].tolist(): (-kt[c], c))[:k]
            assert sorted(got[t].tolist()) == sorted(want), (t, k)


def _stretched_rows(n, g):
    """Rows of which a few values lie so far from the others that equal bins over the whole range say nothing about them."""
    rows = []
    for count, sigma in ((4, 100.0), (64, 100.0), (64, 300.0), (64, 1e4), (300, 1e6)):
        r = torch.randn(n, device=DEV, generator=g)
        r[torch.randperm(n, device=DEV, generator=g)[:count]] = sigma * (1 + 0.1 * torch.randn(count, device=DEV, generator=g))
        rows.append(r)
    rows += [(2.0 * torch.randn(n, device=DEV, generator=g)).exp(), (3.0 * torch.randn(n, device=DEV, generator=g)).exp(),
             torch.tan(3.14 * (torch.rand(n, device=DEV, generator=g) - 0.5))]
    return torch.stack(rows)


@pytest.mark.parametrize("n,k", [(9000, 2048), (33000, 2048), (131072, 2048), (131072, 256)])
def test_values_far_from_the_others_keep_long_rows_on_the_sampled_form(n, k):
    """The bin of the sample's rank is cut into bins in turn, and the candidates are binned by their keys.  Which form a row took
    shows in the order of its output: the sampled one ends with the threshold bin's elements by value, the two-pass form lists
    them by column."""
    g = torch.Generator(device=DEV).manual_seed(n + k)
    x = torch.zeros(8, (n + 3) // 4 * 4, device=DEV)
    x[:, :n] = _stretched_rows(n, g)
    x = x[:, :n]
    a, b = ops.topk_select(x, k), _two_pass(x, k)
    _sets_equal_with_ties(x, a, k)
    assert not (a == b).all(dim=1).any(), (a == b).all(dim=1).tolist()
    many = ops.topk_select(x.repeat(20, 1) if n % 4 == 0 else torch.cat([x] * 20), k)
    assert torch.equal(many[:8], a) and torch.equal(many[-8:], a)


@pytest.mark.parametrize("n", [2048, 3000, 8188, 8192, 33000])
@pytest.mark.parametrize("share", [0.05, 0.3, 0.6])
def test_rows_of_zeros_and_a_few_others(n, share):
    """What a ReLU leaves: the k-th value may be the zero that most columns hold (lower columns first), of either sign."""
    g = torch.Generator(device=DEV).manual_seed(n)
    k = min(2048, n // 2)
    x = torch.randn(6, n, device=DEV, generator=g)
    x = torch.where(torch.rand(6, n, device=DEV, generator=g) < share, x, torch.zeros_like(x))
    x[1] = x[1].relu()
    x[2] = torch.where(x[2] == 0, -x[2], x[2])                  # -0.0
    x[3] *= 1e-38
    x[4] = x[4].abs() * 1e30
    a = ops.topk_select(x, k)
    _sets_equal_with_ties(x, a, k)
    assert torch.equal(a.sort(1).values, _two_pass(x, k).sort(1).values)
    assert torch.equal(ops.topk_select(x.repeat(30, 1), k)[-6:], a)
