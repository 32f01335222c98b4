"""A drop-in product into new trees: the pages of its result are the first to be
touched, and cost about as much as pages used before (each is faulted in once, by
a write; read first, the products took 4 times as long)."""
import time

import numpy as np
import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu


def test_product_into_untouched_pages():
    from dplr_gb300 import _native
    api = _native.api()
    n = 8192
    t = gen.random_tree(n, 256, 32, seed=1)
    a = tree.to_c(t)

    def product(c):
        t0 = time.perf_counter()
        api.geppmm("N", "N", n, 1.0, a, a, 0.0, c, 1e-10)
        return time.perf_counter() - t0

    again, fresh, kept = [], [], []
    for _ in range(8):                            # the heap gives the same pages again
        c = tree.to_c(t)
        again.append(product(c))
        tree.free_c(c)
    for _ in range(10):                           # and has none left after the first of these
        kept.append(tree.to_c(t))
        fresh.append(product(kept[-1]))
    want = tree.flatten(tree.from_c(kept[0]))
    for c in kept[1:]:
        got = tree.flatten(tree.from_c(c))
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    for c in kept + [a]:
        tree.free_c(c)
    assert np.median(fresh[4:]) <= 2.0 * np.median(again), (again, fresh)
