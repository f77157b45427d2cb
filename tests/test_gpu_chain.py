"""Dependent products issued one after another (GPU): each launch is set up
while the one before still writes its input, so a chain of products, each
reading what the last one wrote, gives bit for bit what the same chain gives
when every call is waited for.  (Products of one plan are reproducible bit for
bit, so no tolerance.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(f32, n=3001, per_row=9):
    from cbspmv import gen
    import cbspmv
    rng = np.random.default_rng(n)
    cols = np.stack([np.sort(rng.choice(n, per_row, replace=False)) for _ in range(n)])
    # every row sums to at most 1 in magnitude, so that long chains stay finite
    coo = gen.Coo(n, n, np.repeat(np.arange(n), per_row).astype(np.int32),
                  cols.reshape(-1).astype(np.int32),
                  rng.uniform(-1, 1, n * per_row) / per_row)
    return coo, cbspmv.Plan(coo, value_type=int(f32), want_transpose=1, keep_values=1)


def _both(chain):
    import torch
    outs = []
    for wait in (False, True):
        def step(fn, *a):
            fn(*a)
            if wait:
                torch.cuda.synchronize()
        bufs = chain(step)
        torch.cuda.synchronize()
        outs.append([b.clone() for b in bufs])
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 3, 8, 16])
def test_products_of_products(cuda, f32, nrhs):
    import torch
    coo, plan = _plan(f32)
    dt = torch.float32 if f32 else torch.float64
    shape = (coo.n,) if nrhs == 1 else (coo.n, nrhs)
    x0 = torch.randn(shape, device=cuda, dtype=dt)
    plan.spmv(x0), plan.spmv_t(x0)

    def chain(step):
        x, y = x0.clone(), torch.empty_like(x0)
        for _ in range(40):
            step(plan.spmv, x, y)
            step(plan.spmv_t, y, x)
        return [x, y]

    _both(chain)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_new_values_between_products(cuda, f32, nrhs):
    import torch
    coo, plan = _plan(f32)
    dt = torch.float32 if f32 else torch.float64
    shape = (coo.n,) if nrhs == 1 else (coo.n, nrhs)
    x0 = torch.randn(shape, device=cuda, dtype=dt)
    sets = [torch.from_numpy(s * np.asarray(coo.val)).to(cuda, dt) for s in (1.0, -0.5, 0.75)]
    plan.spmv(x0), plan.spmv_t(x0)

    def chain(step):
        x, y = x0.clone(), torch.empty_like(x0)
        for i in range(30):
            step(plan.set_values, sets[i % 3])
            step(plan.spmv, x, y)
            step(plan.spmv_t, y, x)
        return [x, y]

    _both(chain)


@pytest.mark.parametrize("f32", [False, True])
def test_batches_of_batches(cuda, f32):
    import torch
    import cbspmv
    plans = [_plan(f32, n)[1].upload() for n in (257, 1000, 3001)]
    rhs = [1, 4, 7]
    dt = torch.float32 if f32 else torch.float64
    x0 = [torch.randn(p.n, k, device=cuda, dtype=dt) for p, k in zip(plans, rhs)]
    ends = [[torch.empty_like(x) for x in x0] for _ in range(2)]
    there, back = (cbspmv.Batch(plans, rhs) for _ in range(2))
    there.bind(ends[0], ends[1])
    back.bind(ends[1], ends[0])

    def chain(step):
        for a, x in zip(ends[0], x0):
            a.copy_(x)
        for _ in range(30):
            step(there.run)
            step(back.run)
        return ends[0] + ends[1]

    _both(chain)
