"""The batched SVD kernels' algorithm (dplr_gb300/csrc/svdbatch.cuh: row chunks, QR
of the stacked R's, Jacobi with FP32 angles and power-of-two scaling), checked on
the CPU through a numpy mirror of the three launches: the chunks, the accuracy of
a rotation, the sweep bound and the truncated SVD.  The kernels themselves are held
to the recompression and compression restatements in test_svdbatch_gpu.py,
test_recompress.py and test_compress.py.

Tolerances: a rotation is orthogonal to a few roundings (4 u); the SVD's as for the
one-CTA mirror of test_svdbatch_cpu.py (1e-13 of the largest singular value, 1e-12
for the vectors' orthogonality), of which the chunked QR's and the core's backward
errors, a few r u each, take a tenth.
"""
import os
import re

import numpy as np
import pytest

from dplr_gb300 import gen

HDR = os.path.join(os.path.dirname(__file__), "..", "dplr_gb300", "csrc", "svdbatch.cuh")
U = 1.1102230246251565e-16


def _constant(name):
    m = re.search(r"constexpr int %s = (\d+);" % name, open(HDR).read())
    assert m, name
    return int(m.group(1))


MAX_RANK, MAX_SWEEPS, CHUNK_MAX = _constant("kSvdBatchRank"), _constant("kSvdSweeps"), _constant("kSvdChunkMax")


def _chunk_rows(r):
    return 320 if r > 48 else CHUNK_MAX if 8192 // r > CHUNK_MAX else max(8192 // r, 256)


def _head(x):
    """The leading 21 bits in [1, 2) as a float, signed, and the exponent."""
    m, e = np.frexp(np.abs(x))
    return np.copysign(np.floor(m * 2.0 ** 21) / 2.0 ** 20, x).astype(np.float32), e - 1


def _rotation(a, b, g):
    """svd_rotation, for arrays of pairs."""
    one = np.float32(1)
    d = b - a
    md, ed = _head(np.where(d == 0, 1.0, d))
    mg, eg = _head(g)
    z = (md / mg) * np.exp2(np.clip(ed - eg - 1, -126, 120).astype(np.float32))
    az = np.abs(z)
    zs = np.where(az > 1e6, one, z)
    t = np.where(az > 1e6, np.float32(0.5) / az, one / (np.abs(zs) + np.sqrt(zs * zs + one)))
    t = np.where(d == 0, one, np.copysign(t, z)).astype(np.float32)
    td = t.astype(np.float64)
    y = 1.0 + td * td
    my, ey = _head(y)
    h = 0.5 * y
    x = (one / np.sqrt(np.where(ey > 0, 2 * my, my))).astype(np.float32).astype(np.float64)
    for _ in range(2):
        x = x * (0.5 - h * x * x) + x
    return x, x * td


def _qr(s):
    """(reflectors with unit diagonal, tau, R) of a chunk, scaled by a power of two."""
    n, r = s.shape
    top = np.max(np.abs(s), initial=0.0)
    e = 0 if top == 0 or not np.isfinite(top) else int(np.clip(np.frexp(top)[1] - 1, -1000, 1000))
    a = s * 2.0 ** -e
    neg2 = 2.0 ** -120 * np.sum(a * a)
    v, tau, rr = np.zeros((n, r)), np.zeros(r), np.zeros((r, r))
    for j in range(r):
        alpha, ss = a[j, j], np.sum(a[j + 1:, j] ** 2)
        nn = alpha * alpha + ss
        beta, scl = alpha, 0.0
        if ss > 0.0 and nn > neg2:
            beta = -np.copysign(np.sqrt(nn), alpha)
            tau[j], scl = (beta - alpha) / beta, 1.0 / (alpha - beta)
            w = tau[j] * (scl * (a[j + 1:, j] @ a[j + 1:, j + 1:]) + a[j, j + 1:])
            a[j + 1:, j + 1:] -= np.outer(a[j + 1:, j] * scl, w)
            a[j, j + 1:] -= w
        v[j, j], v[j + 1:, j] = 1.0, a[j + 1:, j] * scl
        rr[:j, j], rr[j, j] = a[:j, j], beta
    return v, tau, rr * 2.0 ** e


def _apply(v, tau, y):
    for j in range(len(tau) - 1, -1, -1):
        if tau[j] != 0.0:
            y[j:] -= np.outer(v[j:, j], tau[j] * (v[j:, j] @ y[j:]))
    return y


def _jacobi(c):
    """(C J, J, sweeps) of svd_core_kernel, c of order 1."""
    r = c.shape[0]
    j = np.eye(r)
    tol2, z2 = (4.0 * r * U) ** 2, np.sum(c * c) * (r * U) ** 2
    rp = r + (r & 1)
    m = rp - 1
    for sweep in range(1, MAX_SWEEPS + 1):
        rotated = False
        for k in range(m):
            pi = np.arange(rp // 2)
            p, q = (k + pi) % m, (k - pi + m) % m
            p[0], q[0] = k, m
            ok = (p < r) & (q < r)
            p, q = p[ok], q[ok]
            x, y = c[:, p], c[:, q]
            a, b, g = np.sum(x * x, 0), np.sum(y * y, 0), np.sum(x * y, 0)
            ok = (a > z2) & (b > z2) & (g * g > tol2 * a * b)
            if not ok.any():
                continue
            rotated = True
            p, q = p[ok], q[ok]
            cs, sn = _rotation(a[ok], b[ok], g[ok])
            for w in (c, j):
                x, y = w[:, p].copy(), w[:, q].copy()
                w[:, p], w[:, q] = cs * x - sn * y, sn * x + cs * y
        if not rotated:
            return c, j, sweep
    raise AssertionError("not converged")


def _svd_batch(u, sig, v, eps):
    """(U', sig', V', sweeps) as the three launches compute them."""
    n, r = u.shape
    nch = -(-n // _chunk_rows(r))
    cut = [k * n // nch for k in range(nch + 1)]
    sides = []
    for s in (u * sig, v):
        chunks = [_qr(s[lo:hi]) for lo, hi in zip(cut, cut[1:])]
        if nch == 1:
            sides.append((chunks, None, chunks[0][2]))
        else:
            v2, t2, rr = _qr(np.vstack([c[2] for c in chunks]))
            sides.append((chunks, (v2, t2), rr))
    core = sides[0][2] @ sides[1][2].T
    top = np.max(np.abs(core), initial=0.0)
    e = 0 if top == 0 else int(np.clip(np.frexp(top)[1] - 1, -1000, 1000))
    c, j, sweeps = _jacobi(core * 2.0 ** -e)
    sv = np.sqrt(np.sum(c * c, 0))
    order = sorted(range(r), key=lambda i: (-sv[i], i))
    rank = 0
    while rank < r and not sv[order[rank]] * 2.0 ** e < eps:
        rank += 1
    keep = order[:rank]
    inv = np.array([1.0 / sv[i] if sv[i] > 0 else 0.0 for i in keep])
    out = []
    for (chunks, stack, _), top in zip(sides, (c[:, keep] * inv, j[:, keep])):
        if stack is not None:
            y = np.zeros((nch * r, rank))
            y[:r] = top
            coef = _apply(*stack, y)
        else:
            coef = top
        res = np.zeros((n, rank))
        for k, (lo, hi) in enumerate(zip(cut, cut[1:])):
            y = np.zeros((hi - lo, rank))
            y[:r] = coef[k * r:(k + 1) * r]
            res[lo:hi] = _apply(chunks[k][0], chunks[k][1], y)
        out.append(res)
    return out[0], sv[keep] * 2.0 ** e, out[1], sweeps


@pytest.mark.parametrize("r", range(1, MAX_RANK + 1))
def test_chunks_cover_the_rows_and_hold_a_triangle(r):
    text = open(HDR).read()
    assert "return r > 48 ? 320 : 8192 / r > kSvdChunkMax ? kSvdChunkMax : 8192 / r > 256 ? 8192 / r : 256;" in text
    rows = _chunk_rows(r)
    for n in [r, r + 1, rows - 1, rows, rows + 1, 2 * rows + 1, 7 * rows + 3, (1 << 22) // (r * r)]:
        if n < r or n * r * r > 1 << 22:
            continue
        nch = -(-n // rows)
        cut = [k * n // nch for k in range(nch + 1)]
        size = np.diff(cut)
        assert cut[-1] == n and size.max() <= rows and size.min() >= r


def test_rotations_are_orthogonal_and_annihilate():
    rng = np.random.default_rng(4)
    m = 20000
    a, b = 10.0 ** rng.uniform(-30, 0, m), 10.0 ** rng.uniform(-30, 0, m)
    b[:50] = a[:50]
    g = np.sqrt(a) * np.sqrt(b) * rng.uniform(-1, 1, m) * 10.0 ** rng.uniform(-14, 0, m)
    cs, sn = _rotation(a, b, g)
    assert np.max(np.abs(cs * cs + sn * sn - 1.0)) <= 4 * 2 * U
    # what is left of g: the angle's relative error, 2^-20 of the heads and a few of FP32
    left = cs * sn * (a - b) + (cs * cs - sn * sn) * g
    assert np.max(np.abs(left) / (np.abs(g) + 8 * U * np.maximum(a, b))) <= 8e-6


def _cases():
    rng = np.random.default_rng(21)
    u, v = rng.standard_normal((900, 64)), rng.standard_normal((900, 64))
    yield "random64", u, 10.0 ** -rng.uniform(0, 12, 64), v, 1e-10
    u, v = rng.standard_normal((700, 11)), rng.standard_normal((700, 11))
    s = np.abs(rng.standard_normal(11)) * 10.0 ** -rng.uniform(0, 6, 11)
    yield "repeated", np.hstack([u] * 6)[:, :64], np.concatenate([s] * 6)[:64], np.hstack([v] * 6)[:, :64], 1e-9
    u, v = (np.linalg.qr(rng.standard_normal((1500, 40)))[0] for _ in range(2))
    yield "decay", u, 0.5 ** np.arange(40), v, 1e-8
    yield "equal", u, np.ones(40), v, 1e-8                     # one cluster of singular values
    yield "pairs", u, np.repeat(0.3 ** np.arange(20), 2) * (1 + 1e-12 * np.arange(40)), v, 1e-9
    yield "tall2", rng.standard_normal((2500, 2)), np.array([1.0, 1e-3]), rng.standard_normal((2500, 2)), 1e-10
    yield "rank1", rng.standard_normal((70, 1)), np.array([2.0]), rng.standard_normal((70, 1)), 1e-10
    x = gen.sorted_uniform(128, seed=11)
    yield "dense", gen.exp_kernel_1d(x, 0.1, 1e-2)[:64, 64:].copy(), np.ones(64), np.eye(64), 1e-10
    p = np.random.default_rng(5).random((128, 2))
    d2 = np.sum((p[:64, None] - p[None, 64:]) ** 2, axis=2)
    yield "gaussian", np.exp(-d2 / 0.02), np.ones(64), np.eye(64), 1e-10
    yield "tiny", 1e-160 * rng.standard_normal((100, 20)), np.full(20, 1e-100), rng.standard_normal((100, 20)), 0.0
    yield "odd", rng.standard_normal((333, 33)), 2.0 ** -np.arange(33), rng.standard_normal((333, 33)), 1e-7


@pytest.mark.parametrize("name,u,s,v,eps", list(_cases()), ids=[c[0] for c in _cases()])
def test_mirror_is_the_truncated_svd_within_the_sweep_bound(name, u, s, v, eps):
    uo, so, vo, sweeps = _svd_batch(u.copy(), s.copy(), v.copy(), eps)
    assert sweeps <= MAX_SWEEPS // 2, sweeps
    # the reference through QRs of the library (the blocks are tall)
    qu, ru = np.linalg.qr(u * s)
    qv, rv = np.linalg.qr(v)
    uf, sf, vtf = np.linalg.svd(ru @ rv.T)
    uf, vf = qu @ uf, qv @ vtf.T
    k = int(np.sum(sf >= eps))
    assert len(so) == k
    scale = sf[0]
    np.testing.assert_allclose(so, sf[:k], rtol=0, atol=1e-13 * scale)
    got, want = (uo * (so / scale)) @ vo.T, (uf[:, :k] * (sf[:k] / scale)) @ vf[:, :k].T
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-13)
    np.testing.assert_allclose(uo.T @ uo, np.eye(k), atol=1e-12)
    np.testing.assert_allclose(vo.T @ vo, np.eye(k), atol=1e-12)


def test_random_and_appended_cores_within_half_the_sweep_bound():
    worst = 0
    for seed in range(40):
        rng = np.random.default_rng(100 + seed)
        r = int(rng.choice([8, 17, 32, 48, 64]))
        s = 10.0 ** -rng.uniform(0, rng.choice([1, 6, 14]), r)
        u, v = rng.standard_normal((r + 30, r)), rng.standard_normal((r + 30, r))
        if seed % 2:                                           # appended copies
            w = max(r // int(rng.integers(2, 7)), 1)
            u, v, s = (np.concatenate([x[..., :w]] * 8, axis=-1)[..., :r] for x in (u, v, s))
        worst = max(worst, _svd_batch(u, s, v, 0.0)[3])
    assert worst <= MAX_SWEEPS // 2, worst


def test_mirror_keeps_zero_blocks_at_rank_zero():
    rng = np.random.default_rng(3)
    _, so, _, _ = _svd_batch(rng.standard_normal((32, 5)), np.zeros(5), rng.standard_normal((32, 5)), 1e-12)
    assert len(so) == 0
