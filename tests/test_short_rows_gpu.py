"""One column under op T, whose leaves are read by rows: tiles and leaves on both sides
of the line between the two ways (tiles of 32 rows, leaves of 64) against the dense
product, alone and in batches, and op T about as fast as op N on a batch of small trees."""
import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _rand(m, seed):
    return torch.randn(1, m, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def _check(y, x, t):
    d = torch.tensor(tree.to_dense(t), device="cuda")
    want = x @ d
    assert ((y - want).norm() / want.norm()).item() <= 1e-13


@pytest.mark.parametrize("n,leaf", [(64, 64), (48, 48), (512, 8), (400, 25), (512, 32), (1024, 64), (1040, 65),
                                    (1024, 128), (2048, 32), (2048, 64), (2048, 256), (4096, 64), (4096, 32)])
def test_one_column_against_the_dense_product(n, leaf):
    from dplr_gb300.plan import GpuPlan
    t = gen.random_tree(n, leaf, 5, seed=leaf)
    p = GpuPlan(t)
    p.factor()
    x = _rand(n, n)
    _check(p.apply(x, trans="T"), x, t)
    z = p.solve(x, trans="T")
    assert ((p.apply(z, trans="T") - x).norm() / x.norm()).item() <= 1e-10
    p.close()


@pytest.mark.parametrize("sizes", [[(512, 32), (256, 64), (1024, 64)], [(512, 32), (4096, 64), (256, 128)]])
def test_batches(sizes):
    from dplr_gb300.plan import GpuPlan
    ts = [gen.random_tree(n, leaf, 4, seed=n) for n, leaf in sizes]
    p = GpuPlan.batch(ts)
    x = _rand(p.m, 3)
    y = p.apply(x, trans="T")
    for t, o in zip(ts, p.offsets()):
        _check(y[:, o:o + t.size], x[:, o:o + t.size], t)
    p.close()


def test_op_t_of_small_trees_is_about_as_fast_as_op_n():
    """600 trees of 256 rows: 79 us under op N, 90 under op T (127 by dot products)."""
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan.batch([gen.random_tree(256, 32, 2, seed=1)] * 600)
    x = _rand(p.m, 1)
    y = torch.empty_like(x)
    ms = []
    for op in "NT":
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = float("inf")
        for _ in range(8):
            for _ in range(3):
                p.apply(x, trans=op, out=y)
            e0.record()
            for _ in range(20):
                p.apply(x, trans=op, out=y)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        ms.append(best)
    assert ms[1] <= 1.35 * ms[0], ms
    p.close()
