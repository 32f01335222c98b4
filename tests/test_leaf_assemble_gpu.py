"""The inverse's leaves at the edges of the tiles that assemble them: leaves of
1 to 100 rows, ancestors' ranks around the slab of 16, none at all, and trees
whose leaves differ in size, against the dense inverse.

Tolerance: with the diagonal at 4 sqrt(n) times the entries the condition number
is below 10; every leaf entry is a sum of at most 200 products, so an error of
200 * 10 * 2^-53 = 2.2e-13 of the inverse's norm per step, over at most 5 levels
1.1e-12.
"""
import numpy as np
import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu

SHAPES = {
    "leaf1": (8, 1, [2, 1, 1]),
    "leaf32": (512, 32, [17, 16, 15, 1]),
    "leaf33": (528, 33, [33, 32, 31, 16]),
    "leaf50": (400, 50, [2, 0, 40]),
    "leaf65": (260, 65, [48, 17]),
    "leaf100": (400, 100, [0, 5]),
    "uneven": (560, 70, [12, 20, 9, 3]),        # the nw quarter one leaf of 140 rows
}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_leaves_of_the_inverse(name):
    from dplr_gb300 import _native
    n, leaf, ranks = SHAPES[name]
    t = gen.random_tree(n, leaf, ranks, seed=2, diag_shift=4.0 * np.sqrt(n), decay=0.9)
    if name == "uneven":
        t.nw.nw = tree.Dense(tree.to_dense(t.nw.nw))
    a, b = tree.to_c(t), tree.new_empty()
    try:
        assert _native.api().geinv(t.size, a, b, 0.0) == 0
        got = tree.to_dense(tree.from_c(b))
    finally:
        tree.free_c(a)
        tree.free_c(b)
    want = np.linalg.inv(tree.to_dense(t))
    assert np.linalg.norm(got - want, 2) <= 1.1e-12 * np.linalg.norm(want, 2)
