"""Graphs captured before a product with more right-hand sides (GPU): the
split-row partials that they hold stay allocated (here several MB, a mapping of
their own), and each replay gives the captured product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _coo(per_row=200, m=400, n=6000):
    from cbspmv import gen
    rng = np.random.default_rng(per_row)
    cols = np.stack([np.sort(rng.choice(n, per_row, replace=False)) for _ in range(m)])
    return gen.Coo(m, n, np.repeat(np.arange(m), per_row).astype(np.int32),
                   cols.reshape(-1).astype(np.int32), rng.standard_normal(m * per_row))


@pytest.mark.parametrize("how", ["batch", "own"])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [3, 20])
def test_replays_after_more_right_hand_sides(cuda, how, f32, nrhs):
    import torch
    import cbspmv
    import cbdump as cd
    dt = torch.float32 if f32 else torch.float64
    coo = _coo()
    plan = cbspmv.Plan(coo, value_type=int(f32), kernel=3, tile_entries=64)
    assert plan.info()["split_rows"] > 0
    x = torch.randn(coo.n, nrhs, device=cuda, dtype=dt)
    y = plan.spmv(x)
    ref, ab = cd.oracle_spmm_ld(coo, np.ascontiguousarray(x.cpu().numpy().astype(np.float64).T))
    if how == "batch":
        batch = cbspmv.Batch([plan], [nrhs]).bind([x], [y])
        batch.graph_launch(True)
        replay = lambda: batch.graph_launch(True)  # noqa: E731
    else:
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            plan.spmv(x, y)
        replay = g.replay
    for more in (1, 2, 3, 7):
        plan.spmv(torch.randn(coo.n, more * nrhs, device=cuda, dtype=dt))
        torch.cuda.synchronize()
        y.fill_(float("nan"))
        replay()
        torch.cuda.synchronize()
        tol = 1e-5 if f32 else 1e-12
        assert np.all(np.abs(y.cpu().numpy().T - ref) <= tol * ab + 1e-30), more
