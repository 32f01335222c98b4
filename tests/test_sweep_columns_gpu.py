"""Solves of many right-hand sides: every column is the same column's solve among a
few, on both sides of the passes' limit (8192 columns for N = 16384, rank 64), and
columns share launches."""
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,leaf,rank,k", [(16384, 256, 64, 8191), (16384, 256, 64, 8233), (1024, 64, 8, 131072 + 65),
                                           (256, 64, 0, 700), (2048, 128, [64, 0, 17, 33], 517)])
def test_columns_in_one_pass_and_in_several(n, leaf, rank, k):
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(n, leaf, rank, seed=3))
    p.factor()
    g = torch.Generator(device="cuda").manual_seed(k)
    b = torch.randn(k, n, dtype=torch.float64, device="cuda", generator=g)
    cols = [c for c in (0, 15, 16, 63, 64, 8191, 8192, 131071, 131072, k - 1) if c < k]
    for op in "NT":
        x = p.solve(b, trans=op)
        want = p.solve(b[cols].contiguous(), trans=op)
        for c, w in zip(cols, want):
            assert (torch.linalg.norm(x[c] - w) / torch.linalg.norm(w)).item() <= 1e-12, (op, c)
    p.close()


def test_columns_share_launches():
    from dplr_gb300 import _native
    from dplr_gb300.plan import GpuPlan
    p = GpuPlan(gen.random_tree(2048, 128, 32, seed=4))
    p.factor()
    counts = []
    for k in (64, 512):
        b = torch.randn(k, p.m, dtype=torch.float64, device="cuda")
        p.solve(b)
        before = _native.launch_count()
        p.solve(b)
        counts.append(_native.launch_count() - before)
    assert counts[0] > 0 and counts[1] <= 2 * counts[0], counts
    p.close()
