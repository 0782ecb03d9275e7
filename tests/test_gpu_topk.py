"""cpg_select_topk: the final select-and-sort step on its own, through the
C ABI on device buffers, against numpy."""
import numpy as np
import pytest

import cpg_b200

pytestmark = pytest.mark.gpu


def _costs(n, seed, zeros=0.1, ties=False):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-5.0, 500.0, size=n).astype(np.float32)
    if ties:
        c = np.round(c).astype(np.float32)
    c[rng.random(n) < zeros] = 0.0
    return c


@pytest.mark.parametrize("n,k,ties", [(1, 1, False), (1000, 10, False), (100_000, 4096, True),
                                      (3_000_000, 1_000_000, False), (50_000, 200_000, True)])
def test_select_topk_matches_numpy(n, k, ties):
    import torch
    c = _costs(n, n + k, ties=ties)
    d = torch.from_numpy(c).cuda()
    out = torch.empty(max(k, 1), dtype=torch.float32, device="cuda")
    got = cpg_b200.select_topk(d.data_ptr(), n, k, out.data_ptr())
    want = np.sort(c[c != 0.0])[:k]
    assert got == len(want)
    assert np.array_equal(out[:got].cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_select_topk_all_zero_and_empty():
    import torch
    d = torch.zeros(1000, dtype=torch.float32, device="cuda")
    out = torch.empty(10, dtype=torch.float32, device="cuda")
    assert cpg_b200.select_topk(d.data_ptr(), 1000, 10, out.data_ptr()) == 0
    assert cpg_b200.select_topk(d.data_ptr(), 0, 10, out.data_ptr()) == 0


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("values", ["one", "two_bits", "few", "narrow", "signs", "inf", "all_bits"])
@pytest.mark.parametrize("n,k", [(1, 3), (5, 2), (2047, 2048), (8193, 2049), (300_001, 70_000)])
def test_select_topk_over_key_ranges_and_alignments(n, k, values, offset):
    """Inputs whose keys differ in no bit, few bits or all 32, values of both
    signs and infinities, at every offset from a 16-byte boundary."""
    import torch
    rng = np.random.default_rng(n + offset)
    c = {"one": lambda: np.full(n, 7.25),
         "two_bits": lambda: rng.choice([1.0, 1.0000001, 1.0000002], n),
         "few": lambda: rng.integers(1, 5, n),
         "narrow": lambda: rng.uniform(40.0, 40.01, n),
         "signs": lambda: rng.normal(0.0, 3.0, n),
         "inf": lambda: rng.choice([-np.inf, np.inf, 1.0, 0.0, -0.0, 3e38], n),
         "all_bits": lambda: rng.choice([-3e38, -1e-40, 1e-40, 2.0, 3e38], n)}[values]().astype(np.float32)
    d = torch.zeros(n + offset, dtype=torch.float32, device="cuda")
    d[offset:] = torch.from_numpy(c).cuda()
    out = torch.full((k,), -1.0, dtype=torch.float32, device="cuda")
    got = cpg_b200.select_topk(d.data_ptr() + 4 * offset, n, k, out.data_ptr())
    want = np.sort(c[c != 0.0])[:k]
    assert got == want.size
    assert np.array_equal(out[:got].cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("n", [40, 5000, 100_003])
def test_select_topk_keeps_the_other_costs_apart_from_nans(n, noalloc):
    """NaNs are no costs, but they count as non-zero values and must not
    disturb the others.  (A NaN's own place and bits are not defined: the key
    transform may pass it through the float unit.)"""
    import ctypes as C
    import torch
    rng = np.random.default_rng(n)
    u = rng.choice(np.array([0x7fc00000, 0x7f800001, 0x7fffffff, 0xffc00000, 0xff800001, 0x7f800000,
                             0xff800000, 0x3f800000, 0xbf800000, 0x42280000, 0, 0x80000000], np.uint32), n)
    c = u.view(np.float32)
    d = torch.from_numpy(u.view(np.int32)).cuda()
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    fn = cpg_b200.lib.cpg_select_topk_noalloc if noalloc else cpg_b200.lib.cpg_select_topk
    got = C.c_int64(-1)
    assert fn(d.data_ptr(), n, n, out.data_ptr(), C.byref(got), None) == 0
    assert got.value == np.count_nonzero(c != 0.0)
    x = out[:got.value].cpu().numpy().view(np.float32)
    x = x[(x != 0.0) & ~np.isnan(x)]
    want = np.sort(c[(c != 0.0) & ~np.isnan(c)])
    assert np.array_equal(x.view(np.uint32), want.view(np.uint32))
