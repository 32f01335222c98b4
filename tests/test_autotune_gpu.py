"""The autotuner keeps the plan's own launch shapes where they are the fastest, and
leaves the plan as it came when a trial fails."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _small_trees():
    from dplr_gb300.plan import GpuPlan
    return GpuPlan.batch([gen.random_tree(1024 << (s % 3), 64, 4, seed=s) for s in range(64)])


def test_a_failed_trial_leaves_the_plan_as_it_came():
    from dplr_gb300 import _native
    lib = _native.lib()
    p = _small_trees()
    x = torch.randn(5, p.m, dtype=torch.float64, device="cuda")
    want = p.apply(x)
    form = lib.dplr_gpu_apply_form(p.handle)
    failures = 0
    for k in range(100):
        lib.dplr_gpu_debug_fail_alloc(k)
        try:
            p.autotune(5)
            break
        except _native.NativeError as e:
            assert "(-3)" in str(e)
            failures += 1
        finally:
            lib.dplr_gpu_debug_fail_alloc(-1)
        assert lib.dplr_gpu_apply_form(p.handle) == form
        assert torch.equal(p.apply(x), want), k           # the same panels and tiles: the same bits
    assert failures >= 4
    p.close()


def _ms(graph):
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(6):
        for _ in range(3):
            graph.launch()
        e0.record()
        for _ in range(20):
            graph.launch()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) / 20)
    return best


@pytest.mark.parametrize("n", [1, 5, 16])
def test_a_tuned_plan_is_not_slower(n):
    """Trials of three products each scatter by a few percent; panels of 256 rows and
    more in place of the plan's own, or no tile of 5 columns, cost 20 to 40."""
    from dplr_gb300.plan import GpuGraph
    p, q = _small_trees(), _small_trees()
    cfg = q.autotune(n)
    x = torch.randn(n, p.m, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    gp, gq = GpuGraph(p, "A", x, y), GpuGraph(q, "A", x, y)
    before, after = _ms(gp), _ms(gq)
    assert after <= 1.12 * before, (before, after, cfg)
    p.close()
    q.close()
