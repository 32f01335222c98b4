"""The FP64 tile products (csrc/fp64tile.cuh) where their cuts can go wrong:
leaves that are no power of two (tiles of unequal height, leaves below, at and
above 64 rows), ranks around the rank tile of 64 and up to 130, every number of
right-hand sides around the column tile of 16, both ops, accumulation, and both
forms of the apply; the transposed single right-hand side too.  Against numpy
on the dense matrix, at n u |A| |X| (the bound of any summation order).
"""
import numpy as np
import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = {
    "leaf50": lambda: gen.random_tree(400, 50, [12, 7, 3], seed=1),
    "leaf75": lambda: gen.random_tree(600, 75, [20, 9, 1], seed=2),
    "leaf127": lambda: gen.random_tree(508, 127, [43, 5], seed=3),
    "leaf3": lambda: gen.random_tree(48, 3, [2, 1, 0, 3], seed=4),
    "leaf1": lambda: gen.random_tree(8, 1, [1, 1, 1], seed=5),
    "leaf65": lambda: gen.random_tree(520, 65, [64, 65, 33], seed=6),
    "rank130": lambda: gen.random_tree(1024, 256, [130, 100], seed=7),
    "dense": lambda: tree.Dense(np.random.default_rng(8).standard_normal((70, 70))),
}


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("form", ["persistent", "launches"])
def test_apply_of_every_cut(name, trans, form, monkeypatch):
    from dplr_gb300.plan import GpuPlan
    monkeypatch.setenv("DPLR_GB300_APPLY", form)
    t = SHAPES[name]()
    a = tree.to_dense(t)
    op = a if trans == "N" else a.T
    p = GpuPlan(t)
    rng = np.random.default_rng(9)
    for n in (1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 50):
        x, y = rng.standard_normal((n, t.size)), rng.standard_normal((n, t.size))
        got = torch.tensor(y, device="cuda")
        p.apply(torch.tensor(x, device="cuda"), trans=trans, alpha=-1.5, beta=0.5, out=got)
        want = -1.5 * (op @ x.T).T + 0.5 * y
        # the products go through the factors: |U||S||V^T| <= sqrt(rank)-ish |block|
        bound = 8 * t.size * 2.0 ** -53 * (np.abs(op) @ np.abs(x).T).max()
        assert np.abs(got.cpu().numpy() - want).max() <= bound, n
    p.close()


@pytest.mark.parametrize("name", ["leaf50", "leaf127", "leaf65", "rank130"])
def test_solve_of_every_cut(name):
    from dplr_gb300.plan import GpuPlan
    t = SHAPES[name]()
    a = tree.to_dense(t)
    p = GpuPlan(t)
    p.factor()
    rng = np.random.default_rng(10)
    for n in (1, 3, 16, 21):
        for trans in ("N", "T"):
            b = rng.standard_normal((n, t.size))
            x = p.solve(torch.tensor(b, device="cuda"), trans=trans).cpu().numpy()
            want = np.linalg.solve(a if trans == "N" else a.T, b.T).T
            assert np.linalg.norm(x - want) <= 1e-13 * t.size * np.linalg.cond(a) * np.linalg.norm(want)
    p.close()
