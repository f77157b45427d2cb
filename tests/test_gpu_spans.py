"""Rows that cross segment boundaries (GPU): one boundary (the two parts meet
in an exchange word) and several (slots and a counter), one and several
right-hand sides and batches, repeated: each launch leaves the words empty for
the next.  Parts that are infinite or NaN, the empty word's own bits among
them, still give NaN rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {False: 1e-12, True: 1e-5}


def _rows(per_row, m=60, n=6000):
    from cbspmv import gen
    rng = np.random.default_rng(per_row)
    cols = np.stack([np.sort(rng.choice(n, per_row, replace=False)) for _ in range(m)])
    return gen.Coo(m, n, np.repeat(np.arange(m), per_row).astype(np.int32),
                   cols.reshape(-1).astype(np.int32), rng.standard_normal(m * per_row))


# chunks of 128 entries, one per segment here: rows inside a chunk, ending on
# its boundary, over one boundary, over several
@pytest.mark.parametrize("per_row", [1, 127, 128, 129, 200, 256, 257, 900])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 3, 8, 16])
def test_rows_across_segments(cuda, per_row, f32, nrhs):
    import torch
    import cbspmv
    import cbdump as cd
    from cbspmv import gen
    coo = _rows(per_row)
    plan = cbspmv.Plan(coo, value_type=int(f32), kernel=5)
    dt = torch.float32 if f32 else torch.float64
    X = gen.uniform_x(coo.n, 7, nrhs=nrhs).reshape(nrhs, coo.n)
    if f32:
        X = X.astype(np.float32).astype(np.float64)
    xd = torch.from_numpy(np.ascontiguousarray(X.T)).to(cuda, dt)
    ref, ab = cd.oracle_spmm_ld(coo, X)
    first = None
    for _ in range(3):
        y = torch.full((coo.m, nrhs), float("nan"), device=cuda, dtype=dt)
        plan.spmv(xd if nrhs > 1 else xd[:, 0].contiguous(), y if nrhs > 1 else y[:, 0])
        got = y.cpu().numpy().astype(np.float64)
        assert np.all(np.abs(got.T - ref) <= TOL[f32] * ab + 1e-300)
        assert first is None or np.array_equal(got, first)
        first = got
    batch = cbspmv.Batch([plan, plan], [nrhs, 1])
    ys = [torch.empty(coo.m, nrhs, device=cuda, dtype=dt),
          torch.empty(coo.m, 1, device=cuda, dtype=dt)]
    batch.bind([xd, xd[:, :1].contiguous()], ys)
    for _ in range(2):
        batch.run()
        assert np.all(np.abs(ys[0].cpu().numpy().T - ref) <= TOL[f32] * ab + 1e-300)
        assert np.all(np.abs(ys[1].cpu().numpy().T - ref[:1]) <= TOL[f32] * ab[:1] + 1e-300)


@pytest.mark.parametrize("f32", [False, True])
def test_parts_without_a_number(cuda, f32):
    import torch
    import cbspmv
    coo = _rows(200)
    plan = cbspmv.Plan(coo, value_type=int(f32), kernel=5)
    t = torch.float32 if f32 else torch.float64
    bits = np.uint32(0xffffdead) if f32 else np.uint64(0xffffdeadffffdead)
    x = np.ones(coo.n, np.float32 if f32 else np.float64)
    ref = plan.spmv(torch.from_numpy(x).to(cuda, t))
    bad = x.copy()
    bad[::3] = bits.view(np.float32 if f32 else np.float64)
    bad[1::3] = np.inf
    bd = torch.from_numpy(bad).to(cuda, t)
    assert torch.isnan(plan.spmv(bd)).all() and torch.isnan(plan.spmv(bd)).all()
    assert torch.equal(plan.spmv(torch.from_numpy(x).to(cuda, t)), ref)
