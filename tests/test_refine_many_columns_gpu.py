"""A refined solve whose unconverged columns, at most a third of all, are more
than a grid's limit in y (65535): each ends as the same column solved alone."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("live", [65535, 65536, 70001])
def test_unconverged_columns_past_the_grid_limit(live):
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(128, 64, 8, seed=9))
    p.factor()
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    b = torch.zeros(210003, p.m, dtype=torch.float64, device="cuda")      # columns of zeros have converged
    b[:live] = torch.randn(live, p.m, dtype=torch.float64, device="cuda", generator=g)
    x, _, its = p.solve_refined(b, tol=0.0, maxiter=1, strict=False, precise=False)
    assert its == 1
    cols = [0, 1, 65534, live - 1]
    want, _, _ = p.solve_refined(b[cols].contiguous(), tol=0.0, maxiter=1, strict=False, precise=False)
    for c, w in zip(cols, want):
        assert (torch.linalg.norm(x[c] - w) / torch.linalg.norm(w)).item() <= 1e-12, c
    assert not bool(x[live:].any())
    p.close()
