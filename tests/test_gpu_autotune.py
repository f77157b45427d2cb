"""The tuner's choice among kernels of small products (GPU), which all take the
host's time a launch when launched one by one: by their device time, the same
every time (pattern reuse 2.6 us here, row segments 4.4)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("bs", [16, 32])
def test_small_products_are_told_apart(cuda, f32, bs):
    import cbspmv
    from test_gpu_spmv import _patterned
    plan = cbspmv.Plan(_patterned(), value_type=int(f32), block_size=bs)
    assert [plan.autotune(1)[0] for _ in range(16)] == [4] * 16
