"""What a factorisation and its solves allocate: the tables of both ops belong to
the factorisation, and its numeric pass allocates nothing."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _bytes(lib, p):
    return lib.dplr_gpu_factor_device_bytes(p.handle)


@pytest.mark.parametrize("n,leaf,rank", [(1024, 64, 8), (4096, 256, 64), (1200, 75, [9, 0, 4])])
def test_solves_of_either_op_bring_no_tables(n, leaf, rank):
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    lib = _native.lib()
    p = GpuPlan(gen.random_tree(n, leaf, rank, seed=1))
    p.factor()
    b = torch.randn(1, n, dtype=torch.float64, device="cuda")
    before = _bytes(lib, p)
    p.solve(b)
    assert _bytes(lib, p) == before
    p.solve(b, trans="T")                     # (the copy of B that op T sweeps over: n doubles)
    assert _bytes(lib, p) == before + 8 * n
    p.close()


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("n,leaf,rank", [(1024, 64, 8), (4096, 256, 64), (1200, 75, [9, 0, 4]), (1024, 128, 100)])
def test_every_allocation_is_the_layout_s(n, leaf, rank, transposed):
    """A failed allocation of the layout leaves no layout; one of the numeric pass
    would leave it behind."""
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    lib = _native.lib()
    p = GpuPlan(gen.random_tree(n, leaf, rank, seed=2))
    failures = 0
    for k in range(100):
        lib.dplr_gpu_debug_fail_alloc(k)
        try:
            p.factor(transposed=transposed)
            break
        except _native.NativeError as e:
            assert "(-3)" in str(e)
            assert _bytes(lib, p) == 0, k
            failures += 1
        finally:
            lib.dplr_gpu_debug_fail_alloc(-1)
    assert failures >= 4
    p.close()
