"""Value updates and gradients in input order (GPU): a plan given new values
gives bit for bit what a plan built with them gives, from the stream and from
the tiles, forward and transposed; the input-order gradient is the stored
values' gradient, value for value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kind, nnz):
    from cbspmv import gen
    rng = np.random.default_rng(nnz)
    if kind == "band":  # CSR and DENSE blocks
        coo = gen.banded(rng, max(3, nnz // 60), 40)
    elif kind == "dups":  # several inputs in one stored value
        coo = gen.random_small(rng, 60, 50, nnz, dup=True)
    else:
        m, n = 400, 700
        key = np.sort(rng.choice(m * n, nnz, replace=False))
        coo = gen.Coo(m, n, (key // n).astype(np.int32), (key % n).astype(np.int32),
                      rng.standard_normal(nnz))
    return coo, gen.Coo(coo.m, coo.n, coo.row, coo.col, rng.standard_normal(coo.nnz))


# one value, the ends of a thread's and of a block's share, several blocks
CASES = [("random", k) for k in (1, 127, 128, 255, 257, 1023, 1024, 1025, 4097)] + [
    ("band", 1024), ("band", 9000), ("dups", 2500)]


@pytest.mark.parametrize("kind,nnz", CASES, ids=[f"{k}-{n}" for k, n in CASES])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("kernel", [0, 1, 2])
def test_new_values_as_if_built_with_them(cuda, kind, nnz, f32, kernel):
    import torch
    import cbspmv
    if kind == "dups" and f32:
        pytest.skip("FP32 inputs of one value are added in another precision at build time")
    coo, new = _case(kind, nnz)
    dt = torch.float32 if f32 else torch.float64
    opts = dict(value_type=int(f32), want_transpose=1, keep_values=1, kernel=kernel)
    p, q = cbspmv.Plan(coo, **opts), cbspmv.Plan(new, **opts)
    p.upload()
    p.set_values(torch.from_numpy(np.asarray(new.val)).to(cuda, dt))
    x = torch.randn(coo.n, device=cuda, dtype=dt)
    g = torch.randn(coo.m, device=cuda, dtype=dt)
    assert torch.equal(p.spmv(x), q.spmv(x))
    assert torch.equal(p.spmv_t(g), q.spmv_t(g))


@pytest.mark.parametrize("kind,nnz", [("random", 1), ("random", 1025), ("band", 1024),
                                      ("dups", 2500)])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs", [1, 3, 8])
def test_adjoint_in_input_order(cuda, kind, nnz, f32, nrhs):
    import torch
    import cbspmv
    coo, _ = _case(kind, nnz)
    dt = torch.float32 if f32 else torch.float64
    plan = cbspmv.Plan(coo, value_type=int(f32), want_transpose=1, keep_values=1)
    shape = (nrhs,) if nrhs > 1 else ()
    x = torch.randn((coo.n,) + shape, device=cuda, dtype=dt)
    g = torch.randn((coo.m,) + shape, device=cuda, dtype=dt)
    gx, gslots = plan.adjoint(g, x)
    hx, gin = plan.adjoint_input(g, x)
    slots = torch.from_numpy(plan.input_slots()).to(cuda)
    assert torch.equal(gx, hx) and torch.equal(gslots[slots], gin)
    none, only = plan.adjoint_input(g, x, want_gx=False)
    assert none is None and torch.equal(only, gin)
