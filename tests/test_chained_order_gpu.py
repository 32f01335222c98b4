"""Chained launches back to back on changing inputs: every product and solve of a
single right-hand side has the bits it has alone, whatever ran before it."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,leaf,rank", [(1024, 64, 8), (16384, 128, 16), (131072, 64, 4)])
def test_alternating_inputs(n, leaf, rank):
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(n, leaf, rank, seed=n))
    p.factor()
    g = torch.Generator(device="cuda").manual_seed(1)
    xs = [s * torch.randn(1, n, dtype=torch.float64, device="cuda", generator=g) for s in (1.0, 1e3, -1e-3)]
    calls = [lambda x, y: p.apply(x, out=y), lambda x, y: p.apply(x, trans="T", out=y),
             lambda x, y: p.solve(x, out=y), lambda x, y: p.solve(x, trans="T", out=y)]
    want = []
    for c in calls:
        for x in xs:
            y = torch.empty_like(x)
            c(x, y)
            torch.cuda.synchronize()
            want.append(y)
    got = [torch.empty_like(x) for _ in calls for x in xs]
    for rep in range(40):
        order = torch.randperm(len(got), generator=torch.Generator().manual_seed(rep)).tolist()
        for y in got:
            y.fill_(float("nan"))
        for k in order:
            calls[k // len(xs)](xs[k % len(xs)], got[k])
        torch.cuda.synchronize()
        for k in order:
            assert torch.equal(got[k], want[k]), (rep, k)
    p.close()
