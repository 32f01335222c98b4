"""Kernels launched while the ones in front of them in the stream still run: the
same results as one after the other (as in a profiled run, which launches every
kernel plainly), on both sides of the lines where they are chained, repeated
without a pause between the calls, on inputs that the kernel in front has just
written, and replayed from a graph.

The results are compared bit for bit: the launches only change when a kernel
starts, never the order of a sum.
"""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# tiles: 64 of 16 rows; 1024 and 2048 of 24 rows, on either side of the expand's line
TREES = {"small": (1024, 64, [8, 4, 2, 3]), "below": (24 * 1024, 24, [4] * 10), "above": (24 * 2048, 24, [3] * 11),
         "rank0": (2048, 128, [0, 3, 0, 5]), "leaf": (128, 128, [1])}


def _plain(f):
    from dplr_gb300 import _native
    _native.profile_start()
    try:
        y = f()
        torch.cuda.synchronize()
    finally:
        _native.profile_stop()
    return y


@pytest.mark.parametrize("name", sorted(TREES))
@pytest.mark.parametrize("nrhs", [1, 2])
def test_chained_launches(name, nrhs):
    from dplr_gb300.plan import GpuGraph, GpuPlan
    n, leaf, ranks = TREES[name]
    p = GpuPlan(gen.random_tree(n, leaf, ranks, seed=1, diag_shift=8.0, decay=0.9))
    p.factor(transposed=True)
    x = torch.randn(nrhs, n, generator=torch.Generator().manual_seed(2), dtype=torch.float64).cuda()
    for op, call in (("A", p.apply), ("S", p.solve)):
        for trans in "NT":
            def chain():
                v = x
                for _ in range(6):
                    v = call(v * 0.125, trans=trans)      # reads what has just been written
                return v
            want = _plain(chain)
            assert bool(torch.isfinite(want).all())
            assert torch.equal(chain(), want)
            one = _plain(lambda: call(x, trans=trans))
            y = torch.full_like(x, float("nan"))
            g = GpuGraph(p, op, x, y, trans=trans)
            for _ in range(3):
                y.fill_(float("nan"))
                g.launch()
            assert torch.equal(y, one)
            g.close()
    p.close()
