"""The tuner's choice among kernels that launching bounds alike (GPU): the
automatic choice, every time."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("bs", [16, 32])
def test_ties_go_to_the_automatic_choice(cuda, f32, bs):
    import cbspmv
    from test_gpu_spmv import _patterned
    plan = cbspmv.Plan(_patterned(), value_type=int(f32), block_size=bs)
    assert [plan.autotune(1)[0] for _ in range(16)] == [4] * 16
