"""The tensor-core capacitance of the inner solve against the FP64 kernel
(`fp64_capacitance`), at the edges of its tiles: node orders around the line
between the two kernels, one output tile (two blocks of up to 64 ranks, or
unequal ones), tiles per block, blocks of more than 128 and odd ranks, levels
that mix both kernels and rank-0 blocks, and right-hand sides around the tiles
of 64 columns; 1030 of them take the tensor cores on every level that has the
work.

Both build the same solve on 7 slices.  A capacitance output differs by the
FP64 kernel's rounding, about r 2^-53 of the row's sum (r <= 512), and the
slices that carry it on hold 50 bits: over 5 levels the solutions differ by
less than 5 512 2^-50 = 2e-12 of the largest entry times the growth of a level,
which the dominant diagonal keeps near 1; 1e-10 leaves a factor 40.  A misplaced
row or term is an error of the order of the update itself.
"""
import numpy as np
import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _mixed_ranks(level, rng):
    return int(rng.choice([0, 1, 5, 16, 23, 24, 25, 40, 63, 64, 65, 100, 127, 128]))


RANKS = {
    "below": [64, 40, 30, 25, 23],
    "line": [25, 24, 23, 25, 24],
    "one_tile": [33, 40, 49, 63, 64],
    "two_tiles": [128, 127, 100, 66, 65],
    "wide": [256, 255, 129, 130, 128],
    "unequal": lambda level, rng: int(rng.choice([20, 30, 90, 100, 129, 200])),
    "mixed": _mixed_ranks,
}


@pytest.mark.parametrize("name", sorted(RANKS))
def test_capacitance_on_the_tensor_cores_matches_fp64(name):
    from dplr_gb300.plan import GpuPlan
    t = gen.random_tree(4096, 128, RANKS[name], seed=3, diag_shift=256.0, decay=0.95)
    rng = np.random.default_rng(8)
    b = torch.tensor(rng.standard_normal((1030, t.size)), device="cuda")
    got = {}
    p = GpuPlan(t)
    p.factor()
    p.prepare_sliced()
    for fp64 in (True, False):
        p.prepare_mixed(7, fp64_capacitance=fp64)
        got[fp64] = [p.solve_refined(b[:n].contiguous(), tol=1e-30, maxiter=0, precise=True, mixed=True, strict=False)
                     for n in (1, 65, 130, 1030)]
    p.close()
    for (x, r, _), (xf, rf, _) in zip(got[False], got[True]):
        assert float((x - xf).abs().max() / xf.abs().max()) <= 1e-10
        assert r <= 4 * rf and rf <= 4 * r, (r, rf)
