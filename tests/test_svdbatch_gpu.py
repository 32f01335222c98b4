"""The batched truncated SVD (csrc/svdbatch.cuh) at the sizes where its split
can go wrong: blocks of one chunk, one row more than a chunk, uneven chunks,
many chunks, the largest rank, ranks of 1 and odd ranks; graded columns,
repeated columns and a scale of 1e120.  Each block against numpy's SVD of its
core (QR of both factors) at the tolerance of the other recompression tests,
1e-12 of the largest singular value.
"""
import numpy as np
import pytest

from dplr_gb300 import tree

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _factors(n, r, rng, kind):
    u, v = rng.standard_normal((n, r)), rng.standard_normal((n, r))
    sig = np.sort(10.0 ** -rng.uniform(0, 9, r))[::-1].copy()
    if kind == "repeated" and r > 1:
        h = r // 2
        u[:, h:2 * h], v[:, h:2 * h] = u[:, :h], v[:, :h]
    if kind == "huge":
        sig *= 1e120
    return u, sig, v


def _tree(n, leaf, top, r0=0):
    """A tree of 2n rows whose top blocks are `top`; deeper blocks of rank 0."""
    def sub(m):
        if m <= leaf:
            return tree.Dense(np.eye(m))
        h = m // 2
        zero = tree.LowRank(np.zeros((h, 0)), np.zeros(0), np.zeros((h, 0)))
        return tree.HNode(sub(h), zero, sub(h), zero)
    return tree.HNode(sub(n), top[0], sub(n), top[1])


@pytest.mark.parametrize("n,leaf,r", [(64, 64, 16), (16, 16, 16), (64, 64, 64), (320, 80, 64), (336, 84, 64),
                                      (1024, 64, 64), (912, 57, 49), (512, 64, 16), (528, 66, 16), (1040, 65, 16),
                                      (8192, 64, 16), (1024, 64, 8), (1056, 66, 7), (2080, 65, 1), (4096, 64, 31),
                                      (16384, 64, 3)])
@pytest.mark.parametrize("kind", ["graded", "repeated", "huge"])
def test_truncated_svd_of_every_chunking(n, leaf, r, kind):
    from dplr_gb300.plan import GpuPlan
    rng = np.random.default_rng(n + r)
    blocks = [_factors(n, r, rng, kind) for _ in range(2)]
    big = 1e120 if kind == "huge" else 1.0
    eps = 1e-6 * big
    p = GpuPlan(_tree(n, leaf, [tree.LowRank(*b) for b in blocks]))
    q = p.reduce_svd(4.0 * eps)                       # eps at the top level's blocks
    pool = q.read_pool().cpu().numpy()
    got = [b for b in q.pool_blocks() if b["kind"] == "lowrank" and b["n"] == n]
    for (u, s, v), b in zip(blocks, got):
        qu, ru = np.linalg.qr(u * (s / big))
        qv, rv = np.linalg.qr(v)
        uc, sc, vct = np.linalg.svd(ru @ rv.T)
        assert np.abs(np.log(sc[sc > 0] * big / eps)).min() > 1e-3       # ranks are decided by the matrix
        k = int(np.sum(sc * big >= eps))
        assert b["rank"] == k
        gu = pool[b["u"]:b["u"] + n * k].reshape(k, n).T
        gv = pool[b["v"]:b["v"] + n * k].reshape(k, n).T
        gs = pool[b["sig"]:b["sig"] + k] / big
        tol = 1e-12 * sc[0]
        assert np.abs(gs - sc[:k]).max() <= tol
        np.testing.assert_allclose(gu.T @ gu, np.eye(k), atol=1e-12)
        np.testing.assert_allclose(gv.T @ gv, np.eye(k), atol=1e-12)
        # the truncated products, through their action on the exact factors
        want = (qu @ (uc[:, :k] * sc[:k])) @ (vct[:k] @ (qv.T @ v))
        have = (gu * gs) @ (gv.T @ v)
        assert np.linalg.norm(have - want) <= 1e-12 * sc[0] * np.linalg.norm(v)
    p.close()
    q.close()
