"""Preparing the tensor-core capacitance allocates twice, whatever the number of
levels: the slices and one block of tables."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def _allocations(lib, call):
    from dplr_gb300 import _native
    for k in range(200):
        lib.dplr_gpu_debug_fail_alloc(k)
        try:
            call()
            return k
        except _native.NativeError as e:
            assert "(-3)" in str(e)
        finally:
            lib.dplr_gpu_debug_fail_alloc(-1)
    raise AssertionError("never succeeds")


@pytest.mark.parametrize("ranks", [24, [128, 100, 64, 30, 20], [64, 0, 40, 23]])
def test_two_allocations_whatever_the_levels(ranks):
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(4096, 128, ranks, seed=1, diag_shift=64.0))
    p.factor()
    p.prepare_sliced()
    lib = _native.lib()
    fp64 = _allocations(lib, lambda: p.prepare_mixed(7, fp64_capacitance=True))
    both = _allocations(lib, lambda: p.prepare_mixed(7))
    assert both - fp64 == 2, (fp64, both)
    p.close()
