"""Batches that list one plan several times (GPU): its launches share its
scratch, so none of them may overlap another.  Rows over one segment boundary
(exchange words) and over several (slots and a counter); the plan's own product
afterwards is what it was before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _coo(per_row, m=400, n=6000):
    from cbspmv import gen
    rng = np.random.default_rng(per_row)
    cols = np.stack([np.sort(rng.choice(n, per_row, replace=False)) for _ in range(m)])
    return gen.Coo(m, n, np.repeat(np.arange(m), per_row).astype(np.int32),
                   cols.reshape(-1).astype(np.int32), rng.standard_normal(m * per_row))


def _modes(batch):
    return (("run", batch.run), ("run_each", batch.run_each),
            ("graph", lambda: batch.graph_launch(False)),
            ("graph_each", lambda: batch.graph_launch(True)))


@pytest.mark.parametrize("per_row", [200, 900])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_one_plan_on_every_entry(cuda, per_row, f32, nrhs):
    import torch
    import cbspmv
    dt = torch.float32 if f32 else torch.float64
    coo = _coo(per_row)
    plan = cbspmv.Plan(coo, value_type=int(f32))
    other = cbspmv.Plan(_coo(129), value_type=int(f32))
    plans = [plan, plan, other, plan, other, plan, plan, plan, plan, plan, plan]
    xs = [torch.randn(coo.n, nrhs, device=cuda, dtype=dt) for _ in plans]
    ys = [torch.empty(coo.m, nrhs, device=cuda, dtype=dt) for _ in plans]

    def own(p, x):  # a product of the plan by itself, waited for
        y = p.spmv(x if nrhs > 1 else x[:, 0].contiguous()).reshape(-1, nrhs)
        torch.cuda.synchronize()
        return y

    want = [own(p, x) for p, x in zip(plans, xs)]
    scale = max(float(w.abs().max()) for w in want)
    batch = cbspmv.Batch(plans, [nrhs] * len(plans)).bind(xs, ys)
    for how, fn in _modes(batch):
        for _ in range(3):
            for y in ys:
                y.fill_(float("nan"))
            fn()
            torch.cuda.synchronize()
            for y, w in zip(ys, want):
                # run_each and its graph launch the plan's own product; the one
                # launch cuts other segments, so it adds in another order
                if how.endswith("each"):
                    assert torch.equal(y, w), how
                else:
                    tol = (1e-4 if f32 else 1e-12) * scale
                    assert float((y - w).abs().max()) <= tol, how
        assert torch.equal(own(plan, xs[0]), want[0]), how


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 5, 20])
def test_one_plan_on_every_entry_over_tiles(cuda, f32, nrhs):
    """The same over the tiles, with block rows split over several (their
    partial sums and arrival counters are the entry's own), and after a
    product with more right-hand sides has given the plan larger partials."""
    import torch
    import cbspmv
    import cbdump as cd
    dt = torch.float32 if f32 else torch.float64
    coo = _coo(200)
    plan = cbspmv.Plan(coo, value_type=int(f32), kernel=3, tile_entries=64)
    assert plan.info()["split_rows"] > 0
    plans = [plan] * 6
    X = [torch.randn(coo.n, nrhs, device=cuda, dtype=dt) for _ in plans]
    ys = [torch.empty(coo.m, nrhs, device=cuda, dtype=dt) for _ in plans]
    refs = [cd.oracle_spmm_ld(coo, np.ascontiguousarray(x.cpu().numpy().astype(np.float64).T))
            for x in X]
    batch = cbspmv.Batch(plans, [nrhs] * len(plans)).bind(X, ys)
    for rep in range(2):
        for how, fn in _modes(batch):
            for y in ys:
                y.fill_(float("nan"))
            fn()
            torch.cuda.synchronize()
            for y, (ref, ab) in zip(ys, refs):
                tol = 1e-5 if f32 else 1e-12
                assert np.all(np.abs(y.cpu().numpy().T - ref) <= tol * ab + 1e-30), (how, rep)
        plan.spmv(torch.randn(coo.n, 3 * nrhs, device=cuda, dtype=dt))


@pytest.mark.parametrize("per_matrix", [False, True])
@pytest.mark.parametrize("ahead", ["own", "batch"])
def test_first_graph_launch_waits_for_the_stream(cuda, per_matrix, ahead):
    """The first graph launch runs the plans once before it captures them:
    after the products already on the stream, not beside them."""
    import torch
    import cbspmv
    coo = _coo(900, m=4000)
    plan = cbspmv.Plan(coo)
    x = torch.randn(coo.n, device=cuda, dtype=torch.float64)
    want = plan.spmv(x)
    torch.cuda.synchronize()
    for _ in range(3):
        y = torch.empty_like(want)
        xs, ys = [x[:, None].contiguous()], [torch.empty(coo.m, 1, device=cuda, dtype=x.dtype)]
        batch = cbspmv.Batch([plan], [1]).bind(xs, ys)
        batch.run()
        torch.cuda.synchronize()
        once = ys[0].clone()
        for _ in range(300):
            plan.spmv(x, y) if ahead == "own" else batch.run()
        batch.graph_launch(per_matrix)
        torch.cuda.synchronize()
        assert torch.equal(ys[0][:, 0], want) if per_matrix else torch.equal(ys[0], once)
        assert ahead == "batch" or torch.equal(y, want)
        assert torch.equal(plan.spmv(x), want)
        batch.run()
        assert torch.equal(ys[0], once)
