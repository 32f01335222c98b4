"""What the framework's speed is measured on: its public entry points over the
sizes that its configurations, tests and benchmarks use.

Every matrix is a partitioned low-rank (PLR) matrix of a kernel on sorted
random points of [0, 1]: K(x, y) = sum_k w_k exp(-|x - y| / l_k) + shift I.  Each
exponential makes every off-diagonal block exactly rank one, so a sum of r of
them gives blocks of rank r with smooth columns and decaying weights; ranks
above that carry columns at rounding level, the shape a truncated SVD of such a
block has (as gen.exp1d_tree does it).  Matrices, right-hand sides and weights
come from the seed alone and are made on the GPU.

``exact`` restates each case in 64 bits with torch only: products block by
block, solves by the Woodbury identity with two refinement steps, truncated SVDs
by QR and torch.linalg.svd.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dplr_gb300 import _native, autograd, tree
from dplr_gb300.plan import GpuGraph, GpuPlan

DEV = "cuda"
F64 = torch.float64

# shift (nugget) of the kernel matrix by kind: the refined solve takes the
# benchmark's 1e-2, on which refinement has something to correct
SHIFT = {"refined": 1e-2}
LEARNING_RATE = 1e-10


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # one matrix-vector product of a small operator inside an iterative
        # method: launches and the host path count, not the factors
        {"name": "apply_small", "kind": "apply", "n": 1024, "leaf": 64, "rmax": 8, "rhs": 1, "trans": "N"},
        # a transposed, accumulated product on a mesh whose size is no power
        # of two (leaves of 50 points), with a handful of right-hand sides
        {"name": "apply_ragged_t", "kind": "apply", "n": 25600, "leaf": 50, "rmax": 12, "rhs": 5, "trans": "T"},
        # the matrix-vector product of the large operator (N = 131072, rank
        # 32, leaf 256): every factor is streamed once
        {"name": "apply_large_1", "kind": "apply", "n": 131072, "leaf": 256, "rmax": 32, "rhs": 1, "trans": "N"},
        # the block product with 64 right-hand sides (block Krylov methods,
        # multiple load cases)
        {"name": "apply_block_64", "kind": "apply", "n": 65536, "leaf": 256, "rmax": 32, "rhs": 64, "trans": "N"},
        # one right-hand side through a factorisation that is kept: the
        # preconditioner application and the time-stepping solve
        {"name": "solve_1", "kind": "solve", "n": 16384, "leaf": 128, "rmax": 16, "rhs": 1, "trans": "N"},
        # the benchmark's refined solve of a block of right-hand sides on the
        # tensor cores (leaf 256, ranks up to 128, tolerance 1e-12)
        {"name": "refined_256", "kind": "refined", "n": 131072, "leaf": 256, "rmax": 128, "rhs": 256, "trans": "N"},
        # new factor values in a plan, factorisation and first solve: each
        # step of a parameter sweep or a nonlinear iteration
        {"name": "refactor_256", "kind": "refactor", "n": 32768, "leaf": 256, "rmax": 64, "rhs": 16, "trans": "N"},
        # a gradient step through the solve with respect to every factor and
        # the right-hand side (leaf 128, rank 16)
        {"name": "adjoint_step", "kind": "adjoint", "n": 32768, "leaf": 128, "rmax": 16, "rhs": 1, "trans": "N"},
        # many small independent matrices in one plan: products and refined
        # solves replayed from graphs (N = 1024 to 8192, ranks 1 to 4, leaf 64)
        {"name": "batch_64", "kind": "batch", "n": 64, "leaf": 64, "rmax": 4, "rhs": 8, "trans": "N"},
        # the drop-in route of a program written against dplr.h, host trees
        # in and out: the explicit inverse, then its product with a block
        {"name": "dropin_inverse", "kind": "inverse", "n": 8192, "leaf": 128, "rmax": 16, "rhs": 16, "trans": "N"},
        # ranks that grew by an update (A + alpha B) brought down again by
        # truncated SVDs on the device, then used
        {"name": "recompress", "kind": "recompress", "n": 16384, "leaf": 64, "rmax": 8, "rhs": 16, "trans": "N"},
        # the drop-in PLR x PLR product, host trees in and out, then used
        {"name": "dropin_product", "kind": "product", "n": 8192, "leaf": 256, "rmax": 32, "rhs": 16, "trans": "N"},
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, leaf, lo, hi):
    """leaf 2^L of [lo, hi], L >= 1."""
    least = max(1, math.ceil(math.log2(lo / leaf)))
    return leaf << rng.randint(least, max(least, int(math.log2(hi / leaf))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "solve", "solve", "refined", "refactor", "refactor", "adjoint",
                       "batch", "inverse", "recompress", "product"])
    trans = rng.choice("NT") if kind in ("apply", "solve") else "N"
    if kind == "batch":
        return {"kind": kind, "n": _between(rng, 12, 96), "leaf": 64, "rmax": 4, "rhs": rng.randint(1, 16), "trans": trans}
    leaf = {"apply": [50, 64, 75, 96, 128, 200, 256], "solve": [50, 64, 75, 96, 128, 192, 256],
            "refined": [128, 256], "refactor": [64, 100, 128, 160, 192, 256], "adjoint": [64, 96, 128, 150],
            "inverse": [64, 100, 128, 256], "recompress": [64, 80, 128], "product": [64, 100, 128, 256]}[kind]
    leaf = rng.choice(leaf)
    lo, hi = {"apply": (1024, 131072), "solve": (1024, 65536), "refined": (8192, 65536), "refactor": (4096, 32768),
              "adjoint": (4096, 32768), "inverse": (1024, 8192), "recompress": (2048, 16384),
              "product": (1024, 8192)}[kind]
    n = _size(rng, leaf, lo, hi)
    if kind == "apply":
        rhs = _between(rng, 1, 96 if n <= 40000 else 32)
    else:
        rhs = _between(rng, *{"solve": (1, 32), "refined": (16, 256), "refactor": (1, 64), "adjoint": (1, 4),
                              "inverse": (1, 64), "recompress": (1, 32), "product": (1, 32)}[kind])
    rmax = _between(rng, *{"apply": (4, 48), "solve": (4, 48), "refined": (16, 128), "refactor": (8, 64),
                           "adjoint": (4, 24), "inverse": (4, 32), "recompress": (4, 16), "product": (4, 32)}[kind])
    return {"kind": kind, "n": n, "leaf": leaf, "rmax": rmax, "rhs": rhs, "trans": trans}


# --------------------------------------------------------------- matrices --

class Matrix:
    """A PLR matrix as stacked tensors.  Level l has 2^l nodes of half size h
    and rank r: U[l], V[l] (2^l, 2, r, h) with [q, 0] the ne block's and [q, 1]
    the sw block's columns, sig[l] (2^l, 2, r); D (leaves, b, b)."""

    def __init__(self, n, leaf, rmax, shift, seed, length=0.1, ranks=None):
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        self.n, self.leaf = n, leaf
        self.levels = int(round(math.log2(n / leaf)))
        assert leaf << self.levels == n
        halves = [n >> (l + 1) for l in range(self.levels)]
        self.ranks = ranks or [min(rmax, max(h // 4, 4)) for h in halves]
        terms = min([24] + self.ranks)
        x = torch.sort(torch.rand(n, generator=gen, device=DEV, dtype=F64)).values
        w = 0.5 ** torch.arange(terms, device=DEV, dtype=F64)
        w = w / w.sum()
        ell = length * 0.7 ** torch.arange(terms, device=DEV, dtype=F64)
        self.U, self.V, self.sig = [], [], []
        for l, (h, r) in enumerate(zip(halves, self.ranks)):
            a, b = x.view(1 << l, 2, h).unbind(1)              # first and second half of every node
            left = torch.exp(-(a[:, -1:] - a)[:, None] / ell[:, None])        # (q, terms, h), 1 at the border
            right = torch.exp(-(b - b[:, :1])[:, None] / ell[:, None])
            gap = torch.exp(-(b[:, 0] - a[:, -1])[:, None] / ell)
            ln, rn = left.norm(dim=2), right.norm(dim=2)
            s = w * gap * ln * rn
            left, right = left / ln[..., None], right / rn[..., None]
            U = torch.stack([left, right], 1)
            V = torch.stack([right, left], 1)
            S = torch.stack([s, s], 1)
            if r > terms:                                      # columns at rounding level
                k = r - terms
                tail = torch.randn(2, 1 << l, 2, k, h, generator=gen, device=DEV, dtype=F64) / math.sqrt(h)
                U, V = torch.cat([U, tail[0]], 2), torch.cat([V, tail[1]], 2)
                S = torch.cat([S, S[..., :1] * 1e-14 * 0.9 ** torch.arange(k, device=DEV, dtype=F64)], 2)
            self.U.append(U)
            self.V.append(V)
            self.sig.append(S)
        xl = x.view(-1, leaf)
        d = (xl[:, :, None] - xl[:, None, :]).abs()
        self.D = sum(w[k] * torch.exp(-d / ell[k]) for k in range(terms))
        self.D += shift * torch.eye(leaf, device=DEV, dtype=F64)

    def host(self):
        """The tree the framework takes."""
        U, V, S = ([t.cpu().numpy() for t in v] for v in (self.U, self.V, self.sig))
        D = self.D.cpu().numpy()

        def block(l, q, s):
            return tree.LowRank(U[l][q, s].T, S[l][q, s], V[l][q, s].T)

        def build(l, q):
            if l == self.levels:
                return tree.Dense(D[q].T)
            return tree.HNode(build(l + 1, 2 * q), block(l, q, 0), build(l + 1, 2 * q + 1), block(l, q, 1))

        return build(0, 0)

    def transposed(self):
        t = object.__new__(Matrix)
        t.n, t.leaf, t.levels, t.ranks = self.n, self.leaf, self.levels, self.ranks
        t.U, t.V, t.sig = [v.flip(1) for v in self.V], [u.flip(1) for u in self.U], [s.flip(1) for s in self.sig]
        t.D = self.D.transpose(1, 2)
        return t

    # ---- in 64 bits, with torch alone -------------------------------------

    def times(self, X):
        """A X for X of shape (n, k) (columns are vectors)."""
        b, k = self.leaf, X.shape[1]
        Y = torch.bmm(self.D, X.view(-1, b, k)).view(self.n, k)
        for U, V, S in zip(self.U, self.V, self.sig):
            q, _, r, h = U.shape
            T = torch.matmul(V, X.view(q, 2, h, k).flip(1)) * S[..., None]
            Y += torch.matmul(U.transpose(2, 3), T).view(self.n, k)
        return Y

    def factor(self):
        self.Dinv = torch.linalg.inv(self.D)
        self.Z, self.Kinv = [None] * self.levels, [None] * self.levels
        for l in reversed(range(self.levels)):
            U, V, S = self.U[l], self.V[l], self.sig[l]
            q, _, r, h = U.shape
            Z = self._below(U.transpose(2, 3).reshape(self.n, r), l + 1).view(q, 2, h, r)
            T = torch.matmul(V, Z.flip(1)) * S[..., None]
            K = torch.eye(2 * r, device=DEV, dtype=F64).repeat(q, 1, 1)
            K[:, :r, r:], K[:, r:, :r] = T[:, 0], T[:, 1]
            self.Z[l], self.Kinv[l] = Z, torch.linalg.inv(K)

    def _below(self, X, lowest):
        k = X.shape[1]
        X = torch.bmm(self.Dinv, X.reshape(-1, self.leaf, k)).view(self.n, k)
        for l in reversed(range(lowest, self.levels)):
            V, S = self.V[l], self.sig[l]
            q, _, r, h = V.shape
            T = torch.matmul(V, X.view(q, 2, h, k).flip(1)) * S[..., None]
            W = torch.bmm(self.Kinv[l], T.view(q, 2 * r, k)).view(q, 2, r, k)
            X = X - torch.matmul(self.Z[l], W).view(self.n, k)
        return X

    def solved(self, B):
        """A^-1 B, refined twice."""
        self.factor()
        X = self._below(B, 0)
        for _ in range(2):
            X = X + self._below(B - self.times(X), 0)
        return X


def _matrix(case, seed):
    return Matrix(case["n"], case["leaf"], case["rmax"], SHIFT.get(case["kind"], 0.5), seed)


def _other(case, seed):
    """The second operand of an update: another length scale."""
    return Matrix(case["n"], case["leaf"], case["rmax"], 0.5, seed + 500_009, length=0.03)


def _batch(case, seed):
    rng = np.random.default_rng(seed)
    shapes = np.random.default_rng(case["n"])                  # sizes and ranks belong to the case
    out = []
    for _ in range(case["n"]):
        L, r = int(shapes.integers(4, 8)), int(shapes.integers(1, case["rmax"] + 1))
        out.append(Matrix(64 << L, 64, r, 0.1, int(rng.integers(1 << 40)), length=float(rng.uniform(0.05, 0.5)),
                          ranks=[r] * L))
    return out


def _rows(n, k, seed, mark):
    """k right-hand sides as the rows of a (k, n) tensor."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 8 + mark)
    return torch.randn(k, n, generator=gen, device=DEV, dtype=F64)


class _HostTree:
    """A malloc-owned C tree, freed with its holder."""

    def __init__(self, node=None):
        self.c = tree.to_c(node) if node is not None else tree.new_empty()

    def __del__(self):
        tree.free_c(self.c)


# ---------------------------------------------------------------- prepare --

def prepare(case, seed):
    kind, k = case["kind"], case["rhs"]
    s = {"kind": kind, "trans": case["trans"]}
    if kind == "batch":
        mats = _batch(case, seed)
        plan = GpuPlan.batch([a.host() for a in mats])
        plan.factor()
        s.update(plan=plan, x=_rows(plan.m, k, seed, 1))
        s["y"], s["z"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
        s["product"] = GpuGraph(plan, "A", s["x"], s["y"])
        s["solve"] = GpuGraph(plan, "C", s["x"], s["z"])
        return s
    n = case["n"]
    a = _matrix(case, seed)
    if kind in ("inverse", "product"):
        s.update(n=n, a=_HostTree(a.host()), c=_HostTree(), x=_rows(n, k, seed, 1).cpu().numpy(),
                 y=np.zeros((k, n)))
        if kind == "product":
            s["b"] = _HostTree(_other(case, seed).host())
            s["c"] = _HostTree(_other(case, seed + 1).host())
        return s
    plan = GpuPlan(a.host())
    s.update(plan=plan, x=_rows(n, k, seed, 1))
    if kind == "apply":
        s["y"] = _rows(n, k, seed, 2)
        s["base"] = s["y"].clone()
    elif kind == "solve":
        plan.factor()
    elif kind == "refined":
        plan.factor()
        plan.prepare_sliced()
        plan.prepare_mixed(7)
    elif kind == "refactor":
        s["pool"] = plan.read_pool()
    elif kind == "adjoint":
        s["pool"] = plan.read_pool().requires_grad_()
        s["x"].requires_grad_()
        s["target"] = _rows(n, k, seed, 3)
    elif kind == "recompress":
        s["other"] = GpuPlan(_other(case, seed).host())
    return s


# -------------------------------------------------------------------- run --

def run(s):
    kind, plan, x = s["kind"], s.get("plan"), s.get("x")
    if kind == "apply":
        if s["trans"] == "N":
            return plan.apply(x)
        s["y"].copy_(s["base"])                                # y := -0.5 A^T x + 2 y
        return plan.apply(x, trans="T", alpha=-0.5, beta=2.0, out=s["y"])
    if kind == "solve":
        return plan.solve(x, trans=s["trans"])
    if kind == "refined":
        return plan.solve_refined(x, tol=1e-12, maxiter=6, strict=False, precise=True, mixed=True)[0]
    if kind == "refactor":
        plan.write_pool(s["pool"])
        plan.factor()
        return plan.solve(x)
    if kind == "adjoint":
        pool = s["pool"]
        pool.grad = x.grad = None
        got = autograd.plr_solve(plan, pool, x)
        loss = ((got - s["target"]) ** 2).sum()
        loss.backward()
        with torch.no_grad():                                  # the factors change from step to step
            pool.add_(pool.grad, alpha=-LEARNING_RATE)
        return {"x": got.detach(), "loss": loss.detach(), "pool_grad": pool.grad, "b_grad": x.grad}
    if kind == "batch":
        s["product"].launch()
        s["solve"].launch()
        return s["y"], s["z"]
    if kind == "recompress":
        grown = plan.axpy(0.5, s["other"])
        small = grown.reduce_svd(1e-8)
        return small.apply(x)
    api, n, k = _native.api(), s["n"], x.shape[0]
    if kind == "inverse":
        api.geinv(n, s["a"].c, s["c"].c, 1e-13)
    else:
        api.geppmm("N", "N", n, 1.0, s["a"].c, s["b"].c, 0.0, s["c"].c, 1e-12)
    api.gepdmm("N", "N", n, k, 1.0, s["c"].c, x.reshape(-1), n, 0.0, s["y"].reshape(-1), n)
    return s["y"]


# ------------------------------------------------------------------- work --

def _stored(n, leaf, ranks):
    """Factor entries of U, V and the leaves."""
    return n * leaf + sum(2 * n * r for r in ranks)


def _ranks(case):
    n, leaf = case["n"], case["leaf"]
    levels = int(round(math.log2(n / leaf)))
    return [min(case["rmax"], max((n >> (l + 1)) // 4, 4)) for l in range(levels)]


def _sweep(n, leaf, ranks):
    """Multiplications of one solve sweep for one right-hand side: the leaf
    inverses, V^T x, the capacitance inverses, Z w."""
    return n * leaf + sum(2 * n * r + (1 << l) * 4 * r * r for l, r in enumerate(ranks))


def _factorisation(n, leaf, ranks):
    mul = n * leaf * leaf + sum((1 << l) * 8 * r ** 3 for l, r in enumerate(ranks))
    for l, r in enumerate(ranks):                              # Z of level l through the deeper levels, then V^T Z
        mul += r * (n * leaf + sum(2 * n * s + (1 << j) * 4 * s * s for j, s in enumerate(ranks) if j > l)) + n * r * r
    return mul


def work(case):
    kind, k = case["kind"], case["rhs"]
    if kind == "batch":
        shapes = np.random.default_rng(case["n"])
        flops = data = 0
        for _ in range(case["n"]):
            L, r = int(shapes.integers(4, 8)), int(shapes.integers(1, case["rmax"] + 1))
            n, ranks = 64 << L, [r] * L
            e = _stored(n, 64, ranks)
            # the product; two sweeps and one residual
            flops += 2 * k * (2 * e + 2 * _sweep(n, 64, ranks))
            data += 8 * (2 * e + n * 64 + sum(n * r for r in ranks)) + 8 * 3 * n * k
        return {"bytes": data, "flops": flops}
    n, leaf, ranks = case["n"], case["leaf"], _ranks(case)
    e, sweep = _stored(n, leaf, ranks), _sweep(n, leaf, ranks)
    if kind == "apply":
        return {"bytes": 8 * e + 8 * n * k * (2 if case["trans"] == "N" else 3), "flops": 2 * e * k}
    if kind == "solve":
        return {"bytes": 8 * sweep + 16 * n * k, "flops": 2 * sweep * k}
    if kind == "refined":                                      # two solves and two residuals
        return {"bytes": 8 * (sweep + e) + 16 * n * k, "flops": 4 * (sweep + e) * k}
    if kind == "refactor":
        return {"bytes": 16 * e + 16 * n * k, "flops": 2 * (_factorisation(n, leaf, ranks) + sweep * k)}
    if kind == "adjoint":
        return {"bytes": 8 * 4 * e + 8 * 5 * n * k, "flops": 2 * (_factorisation(n, leaf, ranks) + (2 * sweep + 2 * e) * k)}
    if kind == "recompress":                                   # two QRs and two products of each factor pair
        flops = sum(8 * n * (2 * r) ** 2 for r in ranks)
        return {"bytes": 8 * 3 * e + 16 * n * k, "flops": flops + 2 * e * k}
    grown = [sum(ranks[: l + 1]) for l in range(len(ranks))]
    if kind == "inverse":
        big = _stored(n, leaf, grown)
        return {"bytes": 8 * (e + 2 * big + 2 * n * k), "flops": 2 * (2 * _factorisation(n, leaf, ranks) + big * k)}
    big = _stored(n, leaf, [r + g for r, g in zip(ranks, grown)])
    mul = n * leaf * leaf + sum(2 * r * (n * leaf + sum(2 * n * s for s in ranks[l + 1:])) for l, r in enumerate(ranks))
    return {"bytes": 8 * (2 * e + 2 * big + 2 * n * k), "flops": 2 * (mul + big * k)}


# ------------------------------------------------------------------ exact --

def exact(case, seed):
    kind, k = case["kind"], case["rhs"]
    if kind == "batch":
        mats = _batch(case, seed)
        x = _rows(sum(a.n for a in mats), k, seed, 1)
        parts = x.split([a.n for a in mats], dim=1)
        return (torch.cat([a.times(p.T.contiguous()).T for a, p in zip(mats, parts)], 1),
                torch.cat([a.solved(p.T.contiguous()).T for a, p in zip(mats, parts)], 1))
    n = case["n"]
    a = _matrix(case, seed)
    x = _rows(n, k, seed, 1)
    xt = x.T.contiguous()
    if kind == "apply":
        if case["trans"] == "N":
            return a.times(xt).T.contiguous()
        return -0.5 * a.transposed().times(xt).T.contiguous() + 2.0 * _rows(n, k, seed, 2)
    if kind == "solve" and case["trans"] == "T":
        a = a.transposed()
    if kind in ("solve", "refined", "refactor"):
        return a.solved(xt).T.contiguous()
    if kind == "inverse":
        return a.solved(xt).T.cpu().numpy()
    if kind == "product":
        return a.times(_other(case, seed).times(xt)).T.cpu().numpy()
    if kind == "recompress":
        b = _other(case, seed)
        return _recompressed(a, b, 0.5, 1e-8).times(xt).T.contiguous()
    got = a.solved(xt)
    g = 2 * (got - _rows(n, k, seed, 3).T)
    lam = a.transposed().solved(g.contiguous())
    return {"x": got.T.contiguous(), "loss": ((got - _rows(n, k, seed, 3).T) ** 2).sum(),
            "pool_grad": _pool_gradient(a, got, -lam), "b_grad": lam.T.contiguous()}


def _recompressed(a, b, alpha, eps):
    """alpha a + b with every block truncated below eps / 4^(depth + 1)."""
    out = object.__new__(Matrix)
    out.n, out.leaf, out.levels, out.D = a.n, a.leaf, a.levels, alpha * a.D + b.D
    out.U, out.V, out.sig = [], [], []
    for l in range(a.levels):
        U = torch.cat([b.U[l] * b.sig[l][..., None], alpha * a.U[l] * a.sig[l][..., None]], 2)
        V = torch.cat([b.V[l], a.V[l]], 2)
        qu, ru = torch.linalg.qr(U.transpose(2, 3))
        qv, rv = torch.linalg.qr(V.transpose(2, 3))
        u, s, vh = torch.linalg.svd(torch.matmul(ru, rv.transpose(2, 3)))
        out.sig.append(torch.where(s >= eps / 4.0 ** (l + 1), s, torch.zeros_like(s)))
        out.U.append(torch.matmul(qu, u).transpose(2, 3))
        out.V.append(torch.matmul(qv, vh.transpose(2, 3)).transpose(2, 3))
    return out


def _pool_gradient(a, X, G):
    """d<G, A X>/d(U, V, sig, leaves) in the order the factors are stored in:
    at each node ne (U, V, sig), sw (U, V, sig), then the first and the second
    diagonal child; every array column by column, padded to 32 entries."""
    k = X.shape[1]
    dU, dV, dS = [], [], []
    for U, V, S in zip(a.U, a.V, a.sig):
        q, _, r, h = U.shape
        xc, gr = X.view(q, 2, h, k).flip(1), G.view(q, 2, h, k)
        tx, tg = torch.matmul(V, xc), torch.matmul(U, gr)                   # (q, 2, r, k)
        dU.append(torch.matmul(tx * S[..., None], gr.transpose(2, 3)))
        dV.append(torch.matmul(tg * S[..., None], xc.transpose(2, 3)))
        dS.append((tx * tg).sum(3))
    dD = torch.bmm(X.view(-1, a.leaf, k), G.view(-1, a.leaf, k).transpose(1, 2))   # columns first
    parts = []

    def put(t):
        parts.append(t.reshape(-1))
        parts.append(t.new_zeros(-t.numel() % 32))

    def walk(l, q):
        if l == a.levels:
            put(dD[q])
            return
        for s in (0, 1):
            for d in (dU, dV, dS):
                put(d[l][q, s])
        walk(l + 1, 2 * q)
        walk(l + 1, 2 * q + 1)

    walk(0, 0)
    return torch.cat(parts)
