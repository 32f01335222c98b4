"""The drop-ins that reshape a tree (dplrgeinv, dplrgeppmm) leave it as it was when
an allocation fails, the pinned staging of results above 128 MB among them, whose
allocation is the last one (made to fail on the host, as in test_faults_gpu.py)."""
import numpy as np
import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu


def _state(c):
    meta, data = tree.flatten(tree.from_c(c))
    return meta, data.view(np.int64)              # bits: NaN compare equal


def _last_failure(lib, call, limit):
    """The largest k for which call(), its k-th allocation failing, reports a
    failure (bisection: call(k) is True where it succeeded)."""
    lo, hi = 0, limit
    assert not call(lo)
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if call(mid):
            hi = mid
        else:
            lo = mid
    return lo


@pytest.mark.parametrize("what", ["geinv", "geppmm"])
def test_tree_untouched_by_a_failed_allocation(what, capfd):
    from dplr_gb300 import _native
    lib, api = _native.lib(), _native.api()
    t = gen.random_tree(16384, 1024, 1, seed=1)               # leaves of 2^24 doubles: just above 128 MB
    m = t.size
    a = tree.to_c(t)
    old = tree.to_c(gen.random_tree(16384, 1024, [0, 3, 1], seed=2))
    before = _state(old)
    messages = {}

    def call(k):
        nonlocal old
        lib.dplr_gpu_release_staging()
        lib.dplr_gpu_debug_fail_alloc(k)
        try:
            if what == "geinv":
                api.geinv(m, a, old, 1e-10)
            else:
                api.geppmm("N", "N", m, 1.0, a, a, 0.5, old, 1e-10)
        finally:
            lib.dplr_gpu_debug_fail_alloc(-1)
        messages[k] = capfd.readouterr().err
        after = _state(old)
        same = np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
        if "allocate" in messages[k]:
            assert same, (k, messages[k])
            return False
        assert not same, (k, messages[k])
        tree.free_c(old)
        old = tree.to_c(gen.random_tree(16384, 1024, [0, 3, 1], seed=2))
        return True

    last = _last_failure(lib, call, 2000)
    assert "pinned staging" in messages[last], messages[last]
    lib.dplr_gpu_release_staging()
    tree.free_c(a)
    tree.free_c(old)
