"""The window of x of each CTA of the row-segment stream is the best one: no
other saves more (a 32-byte sector an entry) over its own length in bytes; a
CTA without entries has none."""
import ctypes

import numpy as np
import pytest


def _best(cols, vsz, longest):
    """The largest saving minus cost over all windows from one column of the
    CTA's entries to another (first columns move down to a multiple of 4)."""
    c = np.sort(cols)
    best = 0
    for lo in range(len(c)):
        last = np.searchsorted(c, (c[lo] & ~3) + longest)
        hi = np.arange(lo, last)
        if len(hi):
            best = max(best, int((32 * (hi - lo + 1) - vsz * (c[hi] - c[lo] + 1)).max()))
    return best


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("n,spread", [(70001, 1), (70001, 40), (9000, 3), (900001, 1)])
@pytest.mark.parametrize("warps", [32, 160])
def test_best_window(f32, n, spread, warps):
    import cbspmv
    from cbspmv import gen
    from layout_decode import rowseg_arrays
    rng = np.random.default_rng(n + spread)
    m = 150
    key = np.unique(rng.integers(0, m, 1500) * n + (n * rng.random(1500) ** spread).astype(int))
    coo = gen.Coo(m, n, (key // n).astype(np.int32), (key % n).astype(np.int32),
                  rng.standard_normal(key.size))
    plan = cbspmv.Plan(coo, value_type=int(f32))
    rs = rowseg_arrays(plan, warps)
    nch, M, nseg, nord, G, W = (int(v) for v in rs["sizes"])
    wlen = np.zeros(G, np.int32)
    assert cbspmv.lib().cbspmv_export(plan._h, f"rs_wlen:{warps}".encode(),
                                      wlen.ctypes.data_as(ctypes.c_void_p)) == G
    words = rs["chunks"].reshape(nch, -1)[:, :512].copy().view(np.uint32).reshape(-1)[:coo.nnz]
    cols = (words & ((1 << 30) - 1)).astype(np.int64)
    vsz = 4 if f32 else 8
    some = 0
    for b in range(G):
        e0, e1 = ((q * nseg // G) * M * 128 for q in (b, b + 1))
        c, wb, wl = cols[e0:e1], int(rs["wbase"][b]), int(wlen[b])
        best = _best(c, vsz, W)
        inside = c[(c >= wb) & (c < wb + wl)]
        assert (wl > 0) == (best > 0)
        assert np.array_equal((words[e0:e1] >> 30) & 1, (c >= wb) & (c < wb + wl))
        if wl:
            some += 1
            assert inside.max() == wb + wl - 1 and inside.min() & ~3 == wb
            assert 32 * len(inside) - vsz * (inside.max() - inside.min() + 1) == best
    assert some > 0
