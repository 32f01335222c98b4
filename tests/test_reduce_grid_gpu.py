"""The reduce of a product with many elements in blocks of many chunks: on both
sides of the grid's limit in y (65535 CTAs of 32 elements, rank 512 and 4095 / 4096
right-hand sides), every column is the same column's product on its own, to 1e-12
(relative, the tolerance of the apply tests)."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 1e-12


def test_reduce_on_both_sides_of_the_grid_limit():
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(65536, 64, [512, 1], seed=5))      # 64 chunks of 512 rows
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(4100, p.m, dtype=torch.float64, device="cuda", generator=g)
    cols = [0, 1, 2049, 4094, 4099]
    for trans in "NT":
        want = p.apply(x[cols].contiguous(), trans=trans)
        for n in (4095, 4100):
            y = p.apply(x[:n], trans=trans)
            for c, w in zip(cols, want):
                if c < n:
                    assert (torch.linalg.norm(y[c] - w) / torch.linalg.norm(w)).item() <= TOL, (trans, n, c)
    p.close()


@pytest.mark.parametrize("n", [262140, 262141, 1048577])
def test_products_of_more_columns_than_a_grid_takes(n):
    """Rank 64: 262140 right-hand sides are one pass, one more are two, and the
    panel's and the expand's grids end at 1048560."""
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(128, 64, 64, seed=6))
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    x = torch.randn(n, p.m, dtype=torch.float64, device="cuda", generator=g)
    cols = [0, 1, 262139, 262140, n - 1]
    cols = [c for c in cols if c < n]
    for trans in "NT":
        want = p.apply(x[cols].contiguous(), trans=trans)
        y = p.apply(x, trans=trans)
        for c, w in zip(cols, want):
            assert (torch.linalg.norm(y[c] - w) / torch.linalg.norm(w)).item() <= TOL, (trans, c)
    p.close()
