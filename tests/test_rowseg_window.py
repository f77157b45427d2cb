"""The windows of x of the row-segment stream: every entry marked as inside
its CTA's window lies in it, and every window lies in x, on the alignment its
copies need.  (Column counts around the alignment and the largest window.)"""
import ctypes

import numpy as np
import pytest


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("n", [1, 3, 5, 16383, 16386, 32769, 70001])
@pytest.mark.parametrize("warps", [32, 160])
def test_windows_hold_their_entries(f32, n, warps):
    import cbspmv
    from cbspmv import gen
    from layout_decode import rowseg_arrays
    rng = np.random.default_rng(n)
    nnz = 30000
    key = np.unique(rng.integers(0, 2000, nnz) * n + (n * rng.random(nnz) ** 3).astype(np.int64))
    coo = gen.Coo(2000, n, (key // n).astype(np.int32), (key % n).astype(np.int32),
                  rng.standard_normal(key.size))
    plan = cbspmv.Plan(coo, value_type=int(f32))
    rs = rowseg_arrays(plan, warps)
    nch, M, nseg, nord, G, W = (int(v) for v in rs["sizes"])
    wlen = np.zeros(G, np.int32)
    assert cbspmv.lib().cbspmv_export(plan._h, f"rs_wlen:{warps}".encode(),
                                      wlen.ctypes.data_as(ctypes.c_void_p)) == G
    wbase = rs["wbase"]
    assert np.all(wlen >= 0) and np.all(wlen <= W)
    assert np.all(wbase % 4 == 0) and np.all(wbase + wlen <= n)
    words = rs["chunks"].reshape(nch, -1)[:, :512].copy().view(np.uint32)
    cols, win = (words & ((1 << 30) - 1)).astype(np.int64), (words >> 30) & 1
    assert win.any() or n == 70001
    for b in range(G):
        c0, c1 = (b * nseg // G) * M, min(nch, ((b + 1) * nseg // G) * M)
        c = cols[c0:c1][win[c0:c1] == 1]
        assert np.all((c >= wbase[b]) & (c < wbase[b] + wlen[b]))
