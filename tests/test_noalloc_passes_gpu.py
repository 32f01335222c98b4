"""dplr_gpu_apply_noalloc where a call takes several passes over its blocks or
columns: small trees, whose own panels are shorter than the 512 rows that a call
is counted with.  The result is the ordinary apply's to 1e-12 (relative, the
tolerance of the apply tests)."""
import ctypes

import pytest

from dplr_gb300 import gen, tree

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 1e-12


def _check(plan, n, trans, seed):
    from dplr_gb300 import _native
    f = _native.lib().dplr_gpu_apply_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p, ctypes.c_char, ctypes.c_int, ctypes.c_double, ctypes.c_void_p,
                  ctypes.c_int, ctypes.c_double, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    m = plan.m
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g)
    y = torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g)
    want = plan.apply(x, trans=trans, alpha=0.7, beta=-0.3, out=y.clone())
    rc = f(plan.handle, trans.encode(), n, 0.7, x.data_ptr(), m, -0.3, y.data_ptr(), m,
           torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0, _native.last_error()
    assert (torch.linalg.norm(y - want) / torch.linalg.norm(want)).item() <= TOL


@pytest.mark.parametrize("leaf,ranks,n", [(64, 32, 4300), (512, 512, 4096), (64, [7, 0, 31, 5], 12000)])
def test_columns_and_blocks_in_passes(leaf, ranks, n):
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(1024, leaf, ranks, seed=leaf))
    for trans in "NT":
        _check(p, n, trans, 3)
    p.close()


def test_one_column_of_a_large_batch_in_passes():
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    count = 2800                       # counted with 5.4 M doubles, 8.4 M with the plan's own panels
    a = tree.to_c(gen.random_tree(1024, 64, 32, seed=7))
    h = ctypes.c_void_p()
    rc = _native.lib().dplr_gpu_batch_create(count, (ctypes.c_int * count)(*[1024] * count),
                                             (tree.PDPlrMtx * count)(*[a] * count), None, ctypes.byref(h))
    tree.free_c(a)
    assert rc == 0, _native.last_error()
    p = GpuPlan(None, _handle=h)
    for trans in "NT":
        _check(p, 1, trans, 4)
    p.close()
