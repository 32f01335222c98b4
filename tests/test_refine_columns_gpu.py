"""Refined solves correct only the columns that have not converged once those
are at most a third: columns that have are left bit for bit, the others end
below the tolerance, whatever their number and wherever they are, on strided
arrays and through the host entry point too.

The inner solve runs on 3 slices (22 bits), so that the first residuals are
about 1e-5 and one or two corrections pass any tolerance between them.
"""
import ctypes

import numpy as np
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def plan():
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(2048, 128, [24, 16, 8, 4], seed=1, diag_shift=4.0))
    p.factor()
    p.prepare_sliced()
    p.prepare_mixed(3)
    yield p
    p.close()


def _solve(p, b, tol, maxiter):
    return p.solve_refined(b, tol=tol, maxiter=maxiter, strict=False, precise=True, mixed=True)


@pytest.mark.parametrize("n", [3, 16, 64, 130])
@pytest.mark.parametrize("late", [1, 2, 5, 21])
def test_only_unconverged_columns_change(plan, n, late):
    if 3 * late > n:
        pytest.skip("more than a third: every column is corrected")
    p = plan
    b = torch.tensor(np.random.default_rng(n + late).standard_normal((n, p.m)), device="cuda")
    x0, _, _ = _solve(p, b, 0.0, 0)
    r0 = p.residual(x0, b).norm(dim=1) / b.norm(dim=1)
    top = torch.sort(r0, descending=True).values
    tol = float((top[late - 1] * top[late]).sqrt())
    x, res, its = _solve(p, b, tol, 6)
    assert its >= 1 and res <= tol
    hard = r0 > tol
    assert int(hard.sum()) == late
    assert torch.equal(x[~hard], x0[~hard])
    r = p.residual(x, b).norm(dim=1) / b.norm(dim=1)
    assert float(r[hard].max()) <= 0.1 * tol            # corrected, not just kept
    # the host entry point returns the same iterate
    from dplr_gb300 import _native
    hb, hx = b.cpu().numpy(), np.zeros((n, p.m))
    out, k = ctypes.c_double(), ctypes.c_int()
    rc = _native.lib().dplr_gpu_solve_refined_host(p.handle, n, hb.ctypes.data, p.m, hx.ctypes.data, p.m, tol, 6, 3,
                                                   ctypes.byref(out), ctypes.byref(k), None)
    assert rc == 0 and k.value == its
    assert np.array_equal(hx, x.cpu().numpy())


def test_strided_arrays(plan):
    from dplr_gb300 import _native
    p, n, ld = plan, 12, plan.m + 7
    b = torch.tensor(np.random.default_rng(5).standard_normal((n, ld)), device="cuda")
    bc = b[:, :p.m].contiguous()
    x0, _, _ = _solve(p, bc, 0.0, 0)
    top = torch.sort(p.residual(x0, bc).norm(dim=1) / bc.norm(dim=1), descending=True).values
    tol = float((top[2] * top[3]).sqrt())
    want, _, its = _solve(p, bc, tol, 6)
    x = torch.full((n, ld), 7.0, dtype=torch.float64, device="cuda")
    out, k = ctypes.c_double(), ctypes.c_int()
    rc = _native.lib().dplr_gpu_solve_refined(p.handle, n, b.data_ptr(), ld, x.data_ptr(), ld, tol, 6, 3,
                                              ctypes.byref(out), ctypes.byref(k),
                                              torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and k.value == its
    assert torch.equal(x[:, :p.m], want) and bool((x[:, p.m:] == 7.0).all())
