"""A profiled solve reports the algorithmic FP64 work of its sweep, whatever kernels
form it: leaves, each level's panel and update, and the capacitance."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,leaf,rank,k", [(4096, 64, 8, 1), (4096, 64, 8, 40), (1024, 64, 16, 3), (65536, 128, 16, 5),
                                           (2048, 128, 100, 4)])
def test_flops_of_a_solve(n, leaf, rank, k):
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(n, leaf, rank, seed=1))
    p.factor()
    b = torch.randn(k, n, dtype=torch.float64, device="cuda")
    levels = (n // leaf).bit_length() - 1
    nodes = sum(1 << lv for lv in range(levels))
    want = 2.0 * k * (n * leaf + levels * 2 * n * rank + nodes * (2 * rank) ** 2)
    for op in "NT":
        x = p.solve(b, trans=op)
        _native.profile_start()
        p.solve(b, trans=op, out=x)
        prof = _native.profile_stop()
        got = sum(v[1] for name, v in prof.items() if name != "reduce")
        assert abs(got - want) <= 1e-9 * want, (op, got, want, prof)
    p.close()
