"""Vectors at any element of a buffer (GPU): the windows of x are copied 16
bytes at a time where x allows it and value by value where it does not, with
window lengths that are no multiple of either; several right-hand sides load
rows of x likewise.  The same values are added in the same order, so the
products are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _coo(kind):
    from cbspmv import gen
    if kind == "grid":  # every gather inside a window
        return gen.laplacian_2d(101, 77)
    rng = np.random.default_rng(5)
    m, n = 3001, {"mixed": 40003, "scattered": 900001}[kind]
    cols = rng.integers(0, n, (m, 12))
    if kind == "mixed":  # some inside, some outside
        cols[:, :8] = (np.arange(m)[:, None] * 13 + rng.integers(0, 300, (m, 8))) % n
    key = np.unique(np.arange(m)[:, None] * n + cols)
    return gen.Coo(m, n, (key // n).astype(np.int32), (key % n).astype(np.int32),
                   rng.standard_normal(key.size))


@pytest.mark.parametrize("kind", ["grid", "mixed", "scattered"])
@pytest.mark.parametrize("f32,offset", [(False, 1), (True, 1), (True, 2), (True, 3)])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_offset_vectors(cuda, kind, f32, offset, nrhs):
    import torch
    import cbspmv
    coo = _coo(kind)
    dt = torch.float32 if f32 else torch.float64
    plan = cbspmv.Plan(coo, value_type=int(f32), kernel=5)
    shape = (coo.n,) if nrhs == 1 else (coo.n, nrhs)
    x = torch.randn(shape, device=cuda, dtype=dt)
    want = plan.spmv(x)
    buf = torch.full((x.numel() + 8,), float("nan"), device=cuda, dtype=dt)
    xo = buf[offset:offset + x.numel()].view(shape)
    xo.copy_(x)
    out = torch.full((want.numel() + 8,), float("nan"), device=cuda, dtype=dt)
    yo = out[offset:offset + want.numel()].view(want.shape)
    assert xo.data_ptr() % 16 and torch.equal(plan.spmv(xo, yo), want)
    assert out[:offset].isnan().all() and out[offset + want.numel():].isnan().all()
