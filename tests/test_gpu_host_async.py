"""cbspmv_spmv_host_async beside other work on the caller's stream (GPU): its
kernels run on a stream of the plan's own, with scratch of their own, after the
caller's value updates.  Rows over one segment boundary (exchange words), over
several (slots and counters), and split block rows over the tiles."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(per_row, f32, kernel, m=2000, n=6000):
    from cbspmv import gen
    import cbspmv
    rng = np.random.default_rng(per_row)
    cols = np.stack([np.sort(rng.choice(n, per_row, replace=False)) for _ in range(m)])
    coo = gen.Coo(m, n, np.repeat(np.arange(m), per_row).astype(np.int32),
                  cols.reshape(-1).astype(np.int32), rng.standard_normal(m * per_row))
    return coo, cbspmv.Plan(coo, value_type=int(f32), keep_values=1, kernel=kernel,
                            tile_entries=64 if kernel == 3 else 0)


def _call(plan, xh, yh, nrhs):
    import torch
    import cbspmv
    rc = cbspmv.lib().cbspmv_spmv_host_async(
        plan._h, ctypes.c_void_p(xh.data_ptr()), ctypes.c_void_p(yh.data_ptr()), nrhs,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, cbspmv.last_error()


@pytest.mark.parametrize("per_row,kernel", [(200, 0), (900, 0), (200, 3)])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_beside_products_of_the_plan(cuda, per_row, kernel, f32, nrhs):
    import torch
    coo, plan = _plan(per_row, f32, kernel)
    dt = torch.float32 if f32 else torch.float64
    shape = (coo.n,) if nrhs == 1 else (coo.n, nrhs)
    x = torch.randn(shape, device=cuda, dtype=dt)
    y = plan.spmv(x)
    torch.cuda.synchronize()
    want = y.clone()
    xh, calls = x.cpu().pin_memory(), 6
    yhs = [torch.empty_like(want, device="cpu").pin_memory() for _ in range(calls)]
    for _ in range(3):
        y.fill_(float("nan"))
        for yh in yhs:
            yh.fill_(float("nan"))
        for _ in range(60):
            plan.spmv(x, y)
        for yh in yhs:
            _call(plan, xh, yh, nrhs)
        torch.cuda.synchronize()
        assert torch.equal(y, want)
        assert all(torch.equal(yh, want.cpu()) for yh in yhs)
    plan.spmv(x, y)
    assert torch.equal(y, want)


@pytest.mark.parametrize("f32", [False, True])
def test_after_new_values(cuda, f32):
    import torch
    coo, plan = _plan(900, f32, 0)
    dt = torch.float32 if f32 else torch.float64
    x = torch.randn(coo.n, device=cuda, dtype=dt)
    xh = x.cpu().pin_memory()
    sets = [torch.from_numpy(s * np.asarray(coo.val)).to(cuda, dt) for s in (1.0, -0.5, 0.25)]
    want = []
    for v in sets:
        plan.upload().set_values(v)
        want.append(plan.spmv(x).cpu())
    big = torch.randn(4096, 4096, device=cuda)
    yhs = [torch.empty_like(want[0]).pin_memory() for _ in range(9)]
    for yh in yhs:
        yh.fill_(float("nan"))
    for i, yh in enumerate(yhs):
        big = big @ big * 1e-4  # the update waits its turn on the caller's stream
        plan.set_values(sets[i % 3])
        _call(plan, xh, yh, 1)
    torch.cuda.synchronize()
    for i, yh in enumerate(yhs):
        assert torch.equal(yh, want[i % 3]), i
