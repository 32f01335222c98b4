"""Sweeps of 2 to 33 right-hand sides: every column is its own solve, at tile heights
of 8 to 64 rows and ranks up to 64, and a few columns cost about what they are."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,leaf,ranks", [(1024, 8, [64, 33, 17, 8, 5]), (1088, 17, [64, 40, 20, 9]),
                                          (800, 25, [64, 31, 12]), (1600, 50, [50, 64, 1, 7]), (4096, 64, [64, 48, 3]),
                                          (6400, 100, 37), (8192, 256, [60, 64, 64])])
def test_every_column_is_its_own_solve(n, leaf, ranks):
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(n, leaf, ranks, seed=leaf))
    p.factor()
    g = torch.Generator(device="cuda").manual_seed(n)
    b = torch.randn(33, n, dtype=torch.float64, device="cuda", generator=g)
    for op in "NT":
        alone = torch.cat([p.solve(b[c:c + 1], trans=op) for c in range(33)])
        for k in list(range(2, 18)) + [20, 31, 33]:
            x = p.solve(b[:k], trans=op)
            err = (torch.linalg.norm(x - alone[:k], dim=1) / torch.linalg.norm(alone[:k], dim=1)).max().item()
            assert err <= 1e-12, (op, k, err)
    p.close()


def test_four_columns_cost_at_most_two_and_a_half_times_two():
    """Twice the work, and fewer launches' latencies; with four predicated multiply-adds
    for every column they took 2.9 times as long."""
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(65536, 256, 32, seed=1))
    p.factor()
    ms = {}
    for k in (2, 4):
        b = torch.randn(k, p.m, dtype=torch.float64, device="cuda")
        x = torch.empty_like(b)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ms[k] = float("inf")
        for _ in range(6):
            for _ in range(2):
                p.solve(b, out=x)
            e0.record()
            for _ in range(10):
                p.solve(b, out=x)
            e1.record()
            torch.cuda.synchronize()
            ms[k] = min(ms[k], e0.elapsed_time(e1) / 10)
    assert ms[4] <= 2.3 * ms[2], ms
    p.close()
