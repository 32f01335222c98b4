"""The batched Gauss-Jordan inverse (csrc/gjinverse.cuh) behind the leaf and
capacitance inverses: orders around its panels of 16, its warps of 32 rows and
its block sizes, one matrix (a cluster of CTAs) and many (one CTA each), mixed
orders, random matrices that pivot in every column and kernel matrices that
never do.  A plan of dense leaves alone makes solve(I) the inverses.

Tolerance: the forward error bound of elimination with partial pivoting,
c n u cond(A) with c = 8 for the growth of these matrices.
"""
import numpy as np
import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
U = 2.0 ** -53


def _matrix(n, seed):
    if seed % 3 == 2:
        return gen.exp_kernel_1d(gen.sorted_uniform(n, seed), 0.1, 1e-2)
    a = np.random.default_rng(seed).standard_normal((n, n))
    return a + 0.5 * np.sqrt(n) * np.eye(n) if seed % 3 else a


def _check(mats):
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan.batch([tree.Dense(a) for a in mats])
    p.factor()
    offs, w = p.offsets(), max(len(a) for a in mats)
    B = np.zeros((w, p.m))
    for a, o in zip(mats, offs):
        B[:len(a), o:o + len(a)] = np.eye(len(a))
    X = p.solve(torch.tensor(B, device="cuda")).cpu().numpy()
    p.close()
    for a, o in zip(mats, offs):
        n = len(a)
        got, want = X[:n, o:o + n].T, np.linalg.inv(a)
        err = np.linalg.norm(got - want) / np.linalg.norm(want)
        assert err <= 8 * n * U * np.linalg.cond(a), (n, err)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 48, 100, 127, 128, 129, 160, 255, 256, 257, 300, 512,
                               513, 800, 1000, 1024])
def test_single_matrix(n):
    for seed in (0, 1, 2):
        _check([_matrix(n, seed)])


def test_mixed_orders():
    _check([_matrix(n, s) for s, n in enumerate([1, 5, 16, 40, 17, 64, 130, 33, 96, 200, 128, 7, 256, 75] * 3)])


@pytest.mark.parametrize("n", [24, 50, 128])
def test_many_matrices(n):
    _check([_matrix(n, s) for s in range(320)])


@pytest.mark.parametrize("n,col", [(8, 0), (40, 20), (128, 127), (200, 16)])
def test_zero_column_reports_its_pivot(n, col):
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    a = _matrix(n, 1)
    a[:, col] = 0.0
    p = GpuPlan(tree.Dense(a))
    with pytest.raises(_native.NativeError, match=rf"zero pivot {col + 1}\)"):
        p.factor()
    p.close()
