"""The batched FP64 GEMM behind the PLR x PLR product, at the edges of its 32 x 32
tiles: leaves and ranks around 8, 16, 32 and 64, inner lengths that end inside a
slab of 16, and long skinny products cut along K, with every transposition.

Tolerance: an entry of the product sums n <= 1040 terms of each of a few products,
n 2^-53 times sum |a| |b| <= sqrt(n) max |c| at random signs: 1.2e-13 * 32 = 4e-12
of the largest entry would be the worst case, a tenth of it is allowed.
"""
import numpy as np
import pytest

from dplr_gb300 import gen, tree
from test_ppmm import _gpu_ppmm

pytestmark = pytest.mark.gpu

SHAPES = {
    "leaf33": (528, 33, [33, 17, 9, 8], [7, 16, 32, 1]),
    "leaf50": (800, 50, [1, 33, 31, 2], [40, 32, 15, 24]),
    "leaf65": (1040, 65, [64, 31, 16, 7], [65, 8, 0, 33]),
    "leaf7": (56, 7, [3, 5, 7], [1, 7, 2]),
}


@pytest.mark.parametrize("ta", "NT")
@pytest.mark.parametrize("tb", "NT")
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_product_is_the_dense_product(name, ta, tb):
    n, leaf, ra, rb = SHAPES[name]
    a = gen.random_tree(n, leaf, ra, seed=3, diag_shift=1.0, decay=0.97)
    b = gen.random_tree(n, leaf, rb, seed=4, diag_shift=1.0, decay=0.97)
    c = gen.random_tree(n, leaf, 2, seed=5, diag_shift=1.0)
    got = tree.to_dense(_gpu_ppmm(ta, tb, 1.3, a, b, 0.4, c, 0.0))
    da, db = tree.to_dense(a), tree.to_dense(b)
    want = 1.3 * (da.T if ta == "T" else da) @ (db.T if tb == "T" else db) + 0.4 * tree.to_dense(c)
    assert np.abs(got - want).max() <= 4e-13 * np.abs(want).max()
