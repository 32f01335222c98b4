"""The Woodbury sweep by row tiles (csrc/sweep.cuh): both ops, levels of uneven
and zero rank, leaves that are no power of two, trees of different depth in one
plan, W formed by the tiles (few CTAs) and by its own launches (many tiles, or
many right-hand sides), more right-hand sides than one pass takes, ranks at its
limit and beyond it (the launches per level).  Against numpy's dense solve, at
the bound of a backward stable solver, 1e-13 m cond(A).
"""
import numpy as np
import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TREES = {
    "uneven": lambda: [gen.random_tree(1024, 32, [40, 0, 7, 16, 1], seed=2)],
    "leaf100": lambda: [gen.random_tree(800, 100, [11, 5, 30], seed=3)],
    "rank64": lambda: [gen.random_tree(512, 128, [64, 33], seed=4)],
    "rank65": lambda: [gen.random_tree(512, 128, [65, 33], seed=5)],
    "one_level": lambda: [gen.random_tree(130, 65, [9], seed=6)],
    "forest": lambda: [gen.random_tree(256, 64, [5, 3], seed=7), tree.Dense(np.eye(10) * 3.0),
                       gen.random_tree(1024, 64, [4, 0, 2, 1], seed=8), gen.random_tree(96, 48, [6], seed=9)],
    "many_tiles": lambda: [gen.random_tree(512, 8, [3, 2, 2, 1, 1, 1], seed=s) for s in range(12)],
}


@pytest.mark.parametrize("name", list(TREES))
def test_solves(name):
    from dplr_gb300.plan import GpuPlan
    trees = TREES[name]()
    dense = [tree.to_dense(t) for t in trees]
    p = GpuPlan.batch(trees)
    p.factor()
    rng = np.random.default_rng(11)
    for n in (1, 2, 3, 16, 33, 70):
        b = rng.standard_normal((n, p.m))
        for trans in ("N", "T"):
            x = p.solve(torch.tensor(b, device="cuda"), trans=trans).cpu().numpy()
            for a, o in zip(dense, p.offsets()):
                m = len(a)
                want = np.linalg.solve(a if trans == "N" else a.T, b[:, o:o + m].T).T
                err = np.linalg.norm(x[:, o:o + m] - want) / np.linalg.norm(want)
                assert err <= 1e-13 * m * np.linalg.cond(a), (n, trans, m)
    p.close()


def test_new_values_reuse_the_sweep():
    """Refactorisation after new values, and both ops again."""
    from dplr_gb300.plan import GpuPlan
    a, b = (gen.random_tree(512, 64, [12, 6, 3], seed=s) for s in (20, 21))
    p, q = GpuPlan(a), GpuPlan(b)
    rhs = torch.tensor(np.random.default_rng(3).standard_normal((4, 512)), device="cuda")
    p.factor()
    p.solve(rhs)
    p.solve(rhs, trans="T")
    p.write_pool(q.read_pool())
    p.factor()
    q.factor()
    for trans in ("N", "T"):
        assert torch.equal(p.solve(rhs, trans=trans), q.solve(rhs, trans=trans))
    p.close()
    q.close()
