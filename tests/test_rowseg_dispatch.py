"""The automatic kernel of one right-hand side on layouts with CSR and DENSE
blocks: which layouts keep the tile kernels (host rule, at a full device's
segmentation), and, on a GPU, that both kernels give the oracle's product
there."""
import ctypes

import numpy as np
import pytest

WARPS = 4736


def _rows(n, half, per, frac, seed=3):
    """A band of 2 half + 1 over the first frac of the rows, per random columns
    in every row."""
    from cbspmv import gen
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    cols = i[:, None] + np.arange(-half, half + 1)[None]
    ok = (cols >= 0) & (cols < n) & (i[:, None] < int(n * frac))
    key = np.concatenate([(i[:, None] * n + cols)[ok],
                          np.repeat(i, per) * n + rng.integers(0, n, n * per)])
    key = np.unique(key)
    return gen.Coo(n, n, (key // n).astype(np.int32), (key % n).astype(np.int32),
                   rng.standard_normal(key.size))


def _tiles(coo, unit, f32, bs):
    import cbspmv
    from cbspmv import gen
    val = np.ones(coo.nnz) if unit else coo.val
    plan = cbspmv.Plan(gen.Coo(coo.m, coo.n, coo.row, coo.col, val), value_type=int(f32),
                       block_size=bs)
    out = np.full(1, -1, np.int32)
    assert cbspmv.lib().cbspmv_export(plan._h, f"rs_tiles:{WARPS}".encode(),
                                      out.ctypes.data_as(ctypes.c_void_p)) == 1
    return int(out[0])


# (rows, half band, random a row, share of banded rows): unit 16, unit 32,
# FP32 16, FP64 16
RULE = [
    ((20000, 64, 0, 1.0), (0, 0, 0, 0)),      # few entries
    ((40000, 64, 0, 1.0), (1, 1, 0, 0)),      # bitmasks
    ((150000, 24, 8, 0.15), (1, 0, 0, 0)),    # uneven scatter
    ((60000, 24, 8, 0.15), (0, 0, 0, 0)),     # the same, few entries
    ((300000, 0, 12, 0.0), (0, 0, 0, 0)),     # no DENSE block
    ((100000, 16, 40, 1.0), (0, 0, 0, 0)),    # even scatter
]


@pytest.mark.parametrize("shape,want", RULE, ids=[str(r[0]) for r in RULE])
def test_which_layouts_keep_the_tiles(shape, want):
    coo = _rows(*shape)
    got = (_tiles(coo, True, False, 16), _tiles(coo, True, False, 32),
           _tiles(coo, False, True, 16), _tiles(coo, False, False, 16))
    assert got == want


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(40000, 64, 0, 1.0), (150000, 24, 8, 0.15)])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("bs", [16, 32])
def test_both_kernels_give_the_product(cuda, shape, f32, bs):
    import torch
    import cbspmv
    import cbdump as cd
    from cbspmv import gen
    coo = _rows(*shape)
    coo = gen.Coo(coo.m, coo.n, coo.row, coo.col, np.ones(coo.nnz))
    dt = torch.float32 if f32 else torch.float64
    x = gen.uniform_x(coo.n, 5)
    if f32:
        x = x.astype(np.float32).astype(np.float64)
    xd = torch.from_numpy(x).to(cuda, dt)
    ref, ab = cd.oracle_spmm_ld(coo, x[None, :])
    for kernel in (0, 5):
        plan = cbspmv.Plan(coo, value_type=int(f32), block_size=bs, kernel=kernel)
        for _ in range(2):
            y = torch.full((coo.m,), float("nan"), device=cuda, dtype=dt)
            plan.spmv(xd, y)
            assert np.all(np.abs(y.cpu().numpy() - ref[0]) <=
                          (1e-5 if f32 else 1e-12) * ab[0] + 1e-30), kernel
