"""The persistent apply by name (DPLR_GB300_APPLY=persistent): a plan takes the three
launches unless its autotuner timed the other form faster, so the tests that ask for no
form run those.  Against the oracle and the three launches, in a batch and in a captured
graph."""
import os

import numpy as np
import pytest

from dplr_gb300 import gen, tree
from oracle import pyoracle
from test_persist_gpu import TREES, _apply

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _want(t, x, trans, alpha, beta, y0):
    a = tree.to_c(t)
    want = y0.cpu().numpy().reshape(-1).copy()
    pyoracle.oracle("best").gepdmm(trans, "N", t.size, x.shape[0], alpha, a,
                                   np.ascontiguousarray(x.cpu().numpy()).reshape(-1), t.size, beta, want, t.size)
    tree.free_c(a)
    return torch.tensor(want.reshape(x.shape[0], t.size), device="cuda")


def test_an_untuned_plan_takes_the_three_launches():
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(TREES["exp1d"]())
    x = torch.randn(3, p.m, dtype=torch.float64, device="cuda")
    p.apply(x)
    before = _native.launch_count()
    p.apply(x)
    assert _native.launch_count() - before == 3
    assert _native.lib().dplr_gpu_apply_form(p.handle) == 1
    p.close()


@pytest.mark.parametrize("name", list(TREES))
@pytest.mark.parametrize("nrhs", [1, 2, 3, 5, 16, 17, 40])
@pytest.mark.parametrize("trans", ["N", "T"])
def test_persistent_form_matches_the_oracle(name, nrhs, trans):
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    t = TREES[name]()
    p = GpuPlan(t)
    g = torch.Generator(device="cpu").manual_seed(nrhs)
    x = torch.randn(nrhs, t.size, generator=g, dtype=torch.float64).cuda()
    y0 = torch.randn(nrhs, t.size, generator=g, dtype=torch.float64).cuda()
    for alpha, beta in ((1.0, 0.0), (-0.75, 1.25)):
        before = _native.launch_count()
        y = _apply(p, x, trans, alpha, beta, y0, "persistent")
        assert _native.launch_count() - before == 1
        want = _want(t, x, trans, alpha, beta, y0)
        assert float((y - want).norm()) <= 1e-12 * float(want.norm())
        yl = _apply(p, x, trans, alpha, beta, y0, "launches")
        assert float((y - yl).norm()) <= 1e-13 * float(want.norm())
    p.close()


def test_persistent_form_on_a_batch_and_in_a_graph(monkeypatch):
    from dplr_gb300.plan import GpuGraph, GpuPlan
    monkeypatch.setenv("DPLR_GB300_APPLY", "persistent")
    assert os.environ["DPLR_GB300_APPLY"] == "persistent"
    ts = [TREES["small_ranks"](), gen.random_tree(512, 32, [5, 3, 1], seed=9)]
    p = GpuPlan.batch(ts)
    x = torch.randn(5, p.m, dtype=torch.float64, device="cuda")
    y, z = p.apply(x), torch.empty_like(x)
    g = GpuGraph(p, "A", x, z)
    assert g.kernels == 1
    z.zero_()
    g.launch()
    torch.cuda.synchronize()
    assert torch.equal(y, z)
    for o, t in zip(p.offsets(), ts):
        xs = x[:, o:o + t.size].contiguous()
        want = _want(t, xs, "N", 1.0, 0.0, torch.zeros_like(xs))
        assert float((y[:, o:o + t.size] - want).norm()) <= 1e-12 * float(want.norm())
    p.close()
