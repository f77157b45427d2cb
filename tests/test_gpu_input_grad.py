"""The value gradient in input order (GPU): its rows and columns, gathered on
the device by the first call, over every kind of layout and count of input
nonzeros around a block of threads; and the captured call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _coo(kind, nnz):
    from cbspmv import gen
    rng = np.random.default_rng(nnz)
    if kind == "band":  # CSR and DENSE blocks
        return gen.banded(rng, max(3, nnz // 60), 40)
    if kind == "dups":  # several inputs in one stored value
        return gen.random_small(rng, 60, 50, nnz, dup=True)
    m, n = 400, 700
    key = np.sort(rng.choice(m * n, nnz, replace=False))
    val = np.ones(nnz) if kind == "unit" else rng.standard_normal(nnz)
    return gen.Coo(m, n, (key // n).astype(np.int32), (key % n).astype(np.int32), val)


@pytest.mark.parametrize("kind,nnz", [("random", k) for k in (1, 255, 256, 257, 5000)] +
                         [("unit", 700), ("band", 9000), ("dups", 2500)])
@pytest.mark.parametrize("bs", [16, 32])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_every_input_has_its_own_product(cuda, kind, nnz, bs, nrhs):
    import torch
    import cbspmv
    coo = _coo(kind, nnz)
    plan = cbspmv.Plan(coo, block_size=bs, want_transpose=1)
    shape = (nrhs,) if nrhs > 1 else ()
    # small whole numbers: every product and sum is exact
    x = torch.randint(-9, 10, (coo.n,) + shape, device=cuda).double()
    g = torch.randint(-9, 10, (coo.m,) + shape, device=cuda).double()
    _, gin = plan.adjoint_input(g, x, want_gx=False)
    r = torch.from_numpy(np.asarray(coo.row)).long().to(cuda)
    c = torch.from_numpy(np.asarray(coo.col)).long().to(cuda)
    want = (g[r] * x[c]).reshape(coo.nnz, -1).sum(1)
    assert torch.equal(gin, want)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 8])
def test_captured(cuda, f32, nrhs):
    import torch
    import cbspmv
    dt = torch.float32 if f32 else torch.float64
    coo = _coo("random", 5000)
    plan = cbspmv.Plan(coo, value_type=int(f32), want_transpose=1, keep_values=1)
    shape = (nrhs,) if nrhs > 1 else ()
    x = torch.randn((coo.n,) + shape, device=cuda, dtype=dt)
    g = torch.randn((coo.m,) + shape, device=cuda, dtype=dt)
    gx, gin = plan.adjoint_input(g, x)  # before the capture: streams, coordinates
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.adjoint_input(g, x, gx, gin)
    for _ in range(3):
        x.normal_(), g.normal_()
        graph.replay()
        torch.cuda.synchronize()
        got = gx.clone(), gin.clone()
        want = plan.adjoint_input(g, x)
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
