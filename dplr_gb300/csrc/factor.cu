// factor.cu -- recursive Woodbury factorisation and FP64 solves.
//
// For an H node with diagonal children A1, A2 and off-diagonal blocks
// ne = U1 S1 V1^T, sw = U2 S2 V2^T, DPLR's inverse (src/dplrinv.c:93-450)
// uses  A^-1 = D^-1 - D^-1 W (S^-1 + V~^T D^-1 W)^-1 V~^T D^-1  with
// D = diag(A1, A2), W = diag(U1, U2), V~^T = [[0, V1^T], [V2^T, 0]].
// Here the same identity is kept in factored form, without 1/sig:
//   Z  = D^-1 W          (panels Z1 = A1^-1 U1, Z2 = A2^-1 U2)
//   K  = I + S V~^T Z = [[I, S1 V1^T Z2], [S2 V2^T Z1, I]]
//   A^-1 b = z - Z K^-1 S V~^T z,       z = D^-1 b
// Its transpose A^-T = D^-T (I - V~ S K^-T Z^T) reuses the same factors:
// the transposed solve sweeps top-down, g -= V~ S K^-T Z^T g per level
// (root first, every node of a level at once), then applies the leaf
// inverses transposed; nothing per level is stored.  The explicit inverse
// also needs Zt = D^-T V~ (Zt1 = A2^-T V1, Zt2 = A1^-T V2, built with
// DPLR_GPU_FACTOR_TRANSPOSED by the same top-down sweep truncated to the
// deeper levels).
//
// Device layout: per H level l one m x r_l matrix Z_l (ld m; rows of the
// ne block of node p hold Z1(p), rows of its sw block hold Z2(p)), the
// same for Zt_l, one (r1+r2)^2 inverse K^-1 per node, and the explicit
// inverses of the dense leaves.  Solves sweep bottom-up: leaves, then the
// deepest H level to the root, each level as one panel / reduce /
// capacitance / update launch sequence over all of its nodes at once.
#include "factor.cuh"
#include "gjinverse.cuh"
#include "hoststage.cuh"
#include "sweep.cuh"

#include <algorithm>
#include <cmath>

namespace dg {

static long long align32(long long x) { return (x + 31) & ~31LL; }

// ------------------------------------------------------------- kernels

// Place one factor per block into the rows of a level right-hand side:
// dst[row0 + i, k] = src[i + k*n] for i < n, k < rank (ld of dst = m).
struct ScatterItem {
    long long src;
    int row0, n, rank;
};

__global__ void scatter_kernel(const ScatterItem *items, const double *src, double *dst, int ldd)
{
    const ScatterItem it = items[blockIdx.y];
    const long long cnt = (long long)it.n * it.rank;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt;
         e += (long long)gridDim.x * blockDim.x) {
        int i = (int)(e % it.n), k = (int)(e / it.n);
        dst[it.row0 + i + (long long)k * ldd] = src[it.src + e];
    }
}

// K = I with off-diagonal blocks from T_ne (r1 x width) and T_sw (r2 x width):
// K[0:r1, r1:r] = T_ne[:, 0:r2],  K[r1:r, 0:r1] = T_sw[:, 0:r1].
__global__ void assemble_k_kernel(const CapItem *items, const double *T, int width, double *kbase)
{
    const CapItem c = items[blockIdx.x];
    const int r = c.r1 + c.r2;
    double *K = kbase + c.k;
    for (long long e = threadIdx.x; e < (long long)r * r; e += blockDim.x) {
        int i = (int)(e % r), j = (int)(e / r);
        double v = i == j ? 1.0 : 0.0;
        if (i < c.r1 && j >= c.r1) v = T[c.t1 * width + i + (long long)(j - c.r1) * c.r1];
        else if (i >= c.r1 && j < c.r1) v = T[c.t2 * width + (i - c.r1) + (long long)j * c.r2];
        K[e] = v;
    }
}

__global__ void zero_kernel(double *p, long long n)
{
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x)
        p[e] = 0.0;
}

// ------------------------------------------------------------- helpers

static int zero_device(double *p, long long n, cudaStream_t st)
{
    if (n <= 0) return 0;
    int grid = (int)std::min<long long>((n + 255) / 256, 152LL * 32);
    zero_kernel<<<grid, 256, 0, st>>>(p, n);
    note_launch();
    DG_CUDA(cudaGetLastError());
    return 0;
}

// Inverts `count` matrices (offsets d_off, orders d_size; nmax the largest,
// host side) and writes each one's info to d_info[i]; asynchronous: the
// caller reads the infos back once the whole factorisation has run.  With
// d_soff the values are read from sbase + d_soff[i] instead of in place.
static int batched_inverse(double *base, const long long *d_off, const int *d_size, const double *sbase,
                           const long long *d_soff, int count, int nmax, int *d_info, int sms, cudaStream_t st,
                           double flops)
{
    if (count == 0 || nmax == 0) return 0;
    ProfScope ps("inverse", st, flops, 0.0);       // 2 n^3 per matrix
    DG_CUDA(gj_launch(base, d_off, d_size, sbase, d_soff, d_info, count, nmax, sms, st));
    note_launch();
    return 0;
}

static int ensure_work(Fact *F, const Plan *p, int nrhs)
{
    // T, W and partials for the widest level schedule, or two levels' parts of
    // the sweep by row tiles.
    long long part = 0;
    for (int v = 0; v < F->nsets; ++v) part = std::max({part, 2 * F->sw[v][0].parts, 2 * F->sw[v][1].parts});
    for (const LevelOps &L : F->lv) part = std::max({part, L.n.partial_per_rhs, L.t.partial_per_rhs});
    size_t need = (size_t)(2 * p->total_rank + part) * std::max(nrhs, 1);
    return ensure_buffer(&F->work, &F->work_doubles, need);
}

// ---------------------------------------------------- the sweep by row tiles

// Right-hand sides of one pass: as many as two levels' parts (each up to rank / 64
// of x's size) allow in 2 GB, a multiple of 64, and as the grids' limits in y allow.
// Fewer only cost: passes of 64 left a small matrix's launches nearly empty (512
// columns, N = 2048, leaf 128, rank 32 2148 us, 1137 in one pass; N = 16384, leaf
// 256, rank 64 19.4 and 15.3 ms; N = 131072, leaf 256, rank 32 96.6 and 94.0).
static int sweep_cols(const Fact *F)
{
    long long parts = 1;
    for (int v = 0; v < F->nsets; ++v) parts = std::max({parts, F->sw[v][0].parts, F->sw[v][1].parts});
    return (int)std::min<long long>(1 << 17, std::max<long long>(64, (1LL << 27) / parts / 64 * 64));
}

// Levels of larger rank would leave one CTA on an SM (two 64 x rank tiles in
// shared memory).
static bool sweep_by_tiles(const Fact *F)
{
    for (const LevelOps &L : F->lv)
        if (L.width > kSweepRank) return false;
    return true;
}

static void add_phase(const std::vector<SweepTile> &tiles, SweepPhase &ph, TableBlock &tb)
{
    ph.count = (int)tiles.size();
    for (const SweepTile &t : tiles) {
        ph.rmax = std::max(ph.rmax, t.urank);
        ph.pmax = std::max(ph.pmax, t.prank);
        ph.rows += t.h;
        ph.urows += (double)t.h * t.urank;
        ph.prows += (double)t.h * t.prank;
    }
    tb.add(tiles, &ph.d);
}

// Most rows of a tile of the factorisation's kernels, by the rows of the whole
// plan: a batch's solves need not sum as each matrix alone does, since their levels
// have the batch's widths, and tiles of 16 rows in a batch of 64 trees of 1024 rows
// only cost (rank 8, 1 / 16 / 64 right-hand sides 170 / 533 / 1909 us; 98 / 317 /
// 1047 with tiles of 64).  Set 1 has tiles of 64 rows (sweep_tiles); levels that
// do not go by row tiles have the one set.
static int sweep_rows(const Plan *p, int set, bool by_tiles = true)
{
    return set == 1 || p->m > (by_tiles ? 4096 : 2048) ? 64 : p->m > 1024 ? 32 : 16;
}

// The tables of one op's sweep, added to tb.
static void build_sweep(Plan *p, Fact *F, int set, int trans, TableBlock &tb)
{
    SweepOp &S = F->sw[set][trans];
    std::vector<int> starts;
    tile_starts(p, starts, sweep_rows(p, set));
    const int nt = (int)starts.size() - 1, m = p->m;
    for (size_t l = 0; l < F->lv.size(); ++l)
        if (F->lv[l].width > 0) S.act.push_back((int)l);
    const int na = (int)S.act.size();
    S.lv.resize(na);
    SweepTile none = {};
    none.cap = -1;
    std::vector<std::vector<SweepTile>> upd(na), pan(na);       // per level and tile: its update, its panel
    for (int k = 0; k < na; ++k) {
        const int l = S.act[k];
        SweepLevel &V = S.lv[k];
        upd[k].assign(nt, none);
        pan[k].assign(nt, none);
        long long off = 0;
        std::vector<int> red_of(p->lr.size(), -1);
        for (int b : F->lv[l].blocks) {
            const LRDesc &D = p->lr[b];
            if (D.rank == 0) continue;
            const auto in = tile_range(starts, trans ? D.row0 : D.col0, D.n);
            red_of[b] = (int)V.red.reduces.size();
            V.red.reduces.push_back(ReduceItem{off, D.toff, trans ? -1 : D.sig, D.rank, in.second - in.first});
            V.red.max_rank = std::max(V.red.max_rank, D.rank);
            V.red.max_nch = std::max(V.red.max_nch, in.second - in.first);
            for (int t = in.first; t < in.second; ++t) {
                SweepTile &x = pan[k][t];
                x.pf = trans ? F->zoff[l] + starts[t] : D.v + (starts[t] - D.col0);
                x.pld = trans ? m : D.n;
                x.prank = D.rank;
                x.pp = off + (long long)(t - in.first) * D.rank;
            }
            off += (long long)(in.second - in.first) * D.rank;
        }
        S.parts = std::max(S.parts, off);
        std::vector<ReduceItem> pair;
        for (int nd : F->lv[l].nodes) {
            const HDesc &H = p->nodes[nd];
            const LRDesc *bl[2] = {&p->lr[H.ne], &p->lr[H.sw]};
            const int r = bl[0]->rank + bl[1]->rank, cap = (int)pair.size() / 2;
            if (r == 0) continue;
            long long sum = 0;
            for (int s = 0; s < 2; ++s) {
                const LRDesc &D = *bl[s];
                const int ri = red_of[s == 0 ? H.ne : H.sw];
                pair.push_back(ri >= 0 ? V.red.reduces[ri] : ReduceItem{0, 0, -1, 0, 0});
                sum += (long long)pair.back().nch * D.rank;
                V.rank_order = std::max(V.rank_order, D.rank * r);
                if (D.rank == 0) continue;
                const auto out = tile_range(starts, trans ? D.col0 : D.row0, D.n);
                for (int t = out.first; t < out.second; ++t) {
                    SweepTile &x = upd[k][t];
                    x.ua = trans ? D.v + (starts[t] - D.col0) : F->zoff[l] + starts[t];
                    x.ulda = trans ? D.n : m;
                    x.urank = D.rank;
                    x.ut = D.toff;
                    x.urow = s == 0 ? 0 : bl[0]->rank;
                    x.cap = cap;
                }
            }
            V.sum = std::max(V.sum, sum);
            V.order = std::max(V.order, r);
        }
        tb.add(V.red.reduces, &V.red.d_reduces);
        tb.add(pair, &V.d_pair);
    }
    auto join = [&](const std::vector<SweepTile> *u, const std::vector<SweepTile> *q, int t) {
        SweepTile x = u ? (*u)[t] : none;
        x.row0 = starts[t];
        x.h = starts[t + 1] - starts[t];
        if (q) {
            x.pf = (*q)[t].pf;
            x.pld = (*q)[t].pld;
            x.prank = (*q)[t].prank;
            x.pp = (*q)[t].pp;
        }
        return x;
    };
    std::vector<SweepTile> tiles;
    for (int k = 0; k < na; ++k) {
        const int nx = trans ? k + 1 : k - 1;
        const std::vector<SweepTile> *q = nx >= 0 && nx < na ? &pan[nx] : nullptr;
        tiles.clear();
        for (int t = 0; t < nt; ++t) {
            const SweepTile x = join(&upd[k], q, t);
            if (x.urank > 0 || x.prank > 0) tiles.push_back(x);
        }
        add_phase(tiles, S.lv[k].level, tb);
        if (!trans) continue;
        tiles.clear();
        for (int t = 0; t < nt; ++t) tiles.push_back(join(nullptr, &pan[k], t));
        add_phase(tiles, S.lv[k].first, tb);
    }
    if (!trans) {
        tiles.clear();
        int t = 0;
        for (size_t i = 0; i < p->leaves.size(); ++i) {
            const LeafDesc &Lf = p->leaves[i];
            for (; t < nt && starts[t] < Lf.row0 + Lf.b; ++t) {
                SweepTile x = join(nullptr, na ? &pan[na - 1] : nullptr, t);
                x.ua = F->leafoff[i] + (starts[t] - Lf.row0);
                x.ulda = x.urank = Lf.b;
                x.ut = Lf.row0;
                tiles.push_back(x);
            }
        }
        add_phase(tiles, S.leaf, tb);
    }
}

// Algorithmic work of one phase: the update's and the panel's multiply-adds, and
// their factors once, x read and written.
static double phase_flops(const SweepPhase &ph, int nrhs) { return 2.0 * (ph.urows + ph.prows) * nrhs; }
static double phase_bytes(const SweepPhase &ph, int nrhs) { return 8.0 * (ph.urows + ph.prows + 2.0 * ph.rows * nrhs); }

template <class K>
static int launch_sweep(K *kern, const SweepPhase &ph, SweepArgs a, int smem_doubles, int nrhs, cudaStream_t st,
                        bool chained)
{
    a.tiles = ph.d;
    a.rmax = ph.rmax;
    a.pmax = ph.pmax;
    if (ph.count == 0) return 0;
    const size_t smem = (size_t)smem_doubles * sizeof(double);
    DG_CUDA(allow_smem((const void *)kern, smem, kSweepSmemMost, 0));
    return launch_chained(kern, dim3((unsigned)ph.count, (unsigned)((nrhs + a.nbt - 1) / a.nbt)), kTT, smem, st, chained,
                          a);
}

static int sweep_tiles(Plan *p, Fact *F, int trans, int lowest, const double *B, int ldb, double *Xo, int ldx,
                       int nrhs, cudaStream_t st, int next)
{
    int rc;
    // short tiles while they are not much more than the SMs, then tall ones, which
    // have fewer barriers and parts (N = 1024, rank 32: 16 columns 162 us short, 165
    // tall; 64: 229, 165; 1000: 1562, 775; N = 2048, rank 64: 32 columns 269, 318;
    // 64: 386, 319); one column in over 2048 rows is faster on tall ones (N = 4096,
    // rank 8: 43, 39)
    const long long ctas = (long long)F->leafT[0].tiles.size() * ((nrhs + kColTile - 1) / kColTile);
    const int set = F->nsets > 1 && (3 * ctas > 4LL * F->sms || (nrhs == 1 && p->m > 2048)) ? 1 : 0;
    SweepOp &S = F->sw[set][trans];
    const Schedule &leafT = F->leafT[set];
    const int na = (int)S.act.size(), m = p->m;
    // Levels follow each other as chained launches where a tile's work is small
    // beside a launch, with one right-hand side (N = 16384, leaf 128, rank 16: 100
    // -> 83 us).  With more, tiles that start early crowd on the SMs that end
    // first (5 right-hand sides, leaf 256: 229 -> 259 us; a factorisation of N =
    // 12288 with ranks 47: 7.9 -> 8.6 ms).
    const bool chained = nrhs == 1;
    int k0 = 0;
    while (k0 < na && S.act[k0] < lowest) ++k0;
    if (trans && k0 == na) return run_expand(leafT, F->leafinv, nullptr, B, ldb, Xo, ldx, nrhs, 1.0, 0.0, st);
    if ((rc = ensure_work(F, p, nrhs))) return rc;
    double *T = F->work, *W = T + (size_t)p->total_rank * nrhs;
    double *parts[2] = {W + (size_t)p->total_rank * nrhs, W + (size_t)(p->total_rank + S.parts) * nrhs};
    SweepArgs a = {};
    a.nrhs = nrhs;
    a.nbt = col_tile(nrhs, kColTile);
    a.trans = trans;
    a.kbase = F->kpool;
    a.sigpool = p->pool;
    a.W = W;
    a.pbase = trans ? F->zpool : p->pool;
    double *X = Xo;
    int ld = ldx, cur = 0;
    if (trans) {
        if ((rc = ensure_buffer(&F->gtr, &F->gtr_doubles, (size_t)m * nrhs))) return rc;
        X = F->gtr;
        ld = m;
    }
    a.x = X;
    a.ldx = ld;
    a.xin = B;
    a.ldin = ldb;
    a.parts = parts[cur];
    {
        const SweepPhase &first = trans ? S.lv[k0].first : S.leaf;
        ProfScope ps("sweep_first", st, phase_flops(first, nrhs), phase_bytes(first, nrhs));
        if (!trans) {
            const int smem = kTileSmem + 64 * (a.nbt | 1) + 64 * (S.leaf.pmax | 1);
            a.ubase = F->leafinv;
            rc = launch_sweep(sweep_leaf_kernel, S.leaf, a, smem, nrhs, st, false);
        } else {
            rc = launch_sweep(sweep_level_kernel<false>, first, a, sweep_smem(first.rmax, first.pmax, a.nbt, 0, 0),
                              nrhs, st, false);
        }
        if (rc) return rc;
    }
    a.xin = X;
    a.ldin = ld;
    a.ubase = trans ? p->pool : F->zpool;
    for (int s = 0; s < na - k0; ++s) {
        const int k = trans ? k0 + s : na - 1 - s, l = S.act[k];
        SweepLevel &V = S.lv[k];
        const Schedule &C = trans ? F->lv[l].t : F->lv[l].n;
        const bool fused = sweep_fused(V.level.count * ((nrhs + a.nbt - 1) / a.nbt), F->sms, V.sum * a.nbt,
                                       V.order * a.nbt, V.rank_order);
        a.parts_in = parts[cur];
        a.parts = parts[cur ^ 1];
        a.caps = C.d_caps;
        a.reds = V.d_pair;
        if (!fused) {
            if ((rc = run_reduce(V.red, trans ? nullptr : p->pool, parts[cur], nrhs, T, st))) return rc;
            if ((rc = run_caps(C, F->kpool, trans ? p->pool : nullptr, trans, T, W, nrhs, st))) return rc;
        }
        const SweepPhase &ph = V.level;
        double fl = phase_flops(ph, nrhs), by = phase_bytes(ph, nrhs);
        if (fused && prof_on())
            for (const CapItem &c : C.caps) {     // W of every node, once
                const double r = c.r1 + c.r2;
                fl += 2.0 * r * r * nrhs;
                by += 8.0 * r * r;
            }
        ProfScope ps("sweep_level", st, fl, by);
        a.kmax = fused ? V.rank_order : 0;
        a.tmax = fused ? V.order * a.nbt : 0;
        const int smem = sweep_smem(ph.rmax, ph.pmax, a.nbt, a.kmax, a.tmax);
        if ((rc = fused ? launch_sweep(sweep_level_kernel<true>, ph, a, smem, nrhs, st, chained)
                        : launch_sweep(sweep_level_kernel<false>, ph, a, smem, nrhs, st, chained)))
            return rc;
        cur ^= 1;
    }
    if (trans) return run_expand(leafT, F->leafinv, nullptr, X, ld, Xo, ldx, nrhs, 1.0, 0.0, st);
    // the parts of the level above (k0 - 1) are in parts[cur]
    if (next >= 0) return run_reduce(S.lv[k0 - 1].red, p->pool, parts[cur], nrhs, T, st);
    return 0;
}

// One sweep over the leaves and the H levels from `lowest` to the deepest
// (all of them for lowest = 0).  op N, bottom-up: Xo = leaf^-1 B, then per
// level from the deepest up: Xo -= Z K^-1 S V~^T Xo.  op T, top-down: a
// copy G of B takes G -= V~ S K^-T Z^T G per level from `lowest` down to
// the deepest, then Xo = leaf^-T G.  B and Xo are m x nrhs (ld ldb / ldx)
// and must not alias.
//
// Levels of ranks up to kSweepRank go by row tiles (sweep.cuh), sweep_cols
// right-hand sides at a time; the others launch panel, reduce, capacitance and
// update per level.  With next (op N; the level above `lowest`, nrhs its width),
// that level's S V^T Xo comes back in T as well.
static int sweep(Plan *p, Fact *F, int trans, int lowest, const double *B, int ldb, double *Xo,
                 int ldx, int nrhs, cudaStream_t st, int next = -1)
{
    if (sweep_by_tiles(F)) {
        const int cols = sweep_cols(F);
        for (int j = 0; j < nrhs; j += cols) {
            const int rc = sweep_tiles(p, F, trans, lowest, B + (long long)j * ldb, ldb, Xo + (long long)j * ldx, ldx,
                                       std::min(cols, nrhs - j), st, next);
            if (rc) return rc;
        }
        return 0;
    }
    int rc = ensure_work(F, p, nrhs);
    if (rc) return rc;
    double *T = F->work;
    double *W = F->work + (size_t)p->total_rank * nrhs;
    double *partials = W + (size_t)p->total_rank * nrhs;
    if (!trans) {
        if ((rc = run_expand(F->leafN, F->leafinv, nullptr, B, ldb, Xo, ldx, nrhs, 1.0, 0.0, st))) return rc;
        for (int l = (int)F->lv.size() - 1; l >= lowest; --l) {
            const LevelOps &L = F->lv[l];
            if (L.width == 0) continue;
            if ((rc = run_panel(L.n, p->pool, Xo, ldx, nrhs, partials, st))) return rc;
            if ((rc = run_reduce(L.n, p->pool, partials, nrhs, T, st))) return rc;
            if ((rc = run_caps(L.n, F->kpool, nullptr, 0, T, W, nrhs, st))) return rc;
            if ((rc = run_expand(L.n, F->zpool, W, nullptr, 0, Xo, ldx, nrhs, -1.0, 1.0, st))) return rc;
        }
        if (next < 0) return 0;
        if ((rc = run_panel(F->lv[next].n, p->pool, Xo, ldx, nrhs, partials, st))) return rc;
        return run_reduce(F->lv[next].n, p->pool, partials, nrhs, T, st);
    }
    const int m = p->m;
    if ((rc = ensure_buffer(&F->gtr, &F->gtr_doubles, (size_t)m * nrhs))) return rc;
    double *G = F->gtr;
    DG_CUDA(cudaMemcpy2DAsync(G, (size_t)m * sizeof(double), B, (size_t)ldb * sizeof(double),
                              (size_t)m * sizeof(double), nrhs, cudaMemcpyDeviceToDevice, st));
    for (int l = lowest; l < (int)F->lv.size(); ++l) {
        const LevelOps &L = F->lv[l];
        if (L.width == 0) continue;
        if ((rc = run_panel(L.t, F->zpool, G, m, nrhs, partials, st))) return rc;       // Z^T G
        if ((rc = run_reduce(L.t, nullptr, partials, nrhs, T, st))) return rc;
        if ((rc = run_caps(L.t, F->kpool, p->pool, 1, T, W, nrhs, st))) return rc;     // S K^-T
        if ((rc = run_expand(L.t, p->pool, W, nullptr, 0, G, m, nrhs, -1.0, 1.0, st))) return rc;   // V~
    }
    return run_expand(F->leafT[0], F->leafinv, nullptr, G, m, Xo, ldx, nrhs, 1.0, 0.0, st);
}

// ------------------------------------------------------------- schedules

// With caps_only (the sweeps go by row tiles) the levels' schedules hold their
// capacitance items alone.
static void build_level_schedules(Plan *p, Fact *F, bool caps_only)
{
    std::vector<int> starts;
    tile_starts(p, starts, sweep_rows(p, 0, caps_only));
    const int m = p->m;
    for (size_t l = 0; l < F->lv.size(); ++l) {
        LevelOps &L = F->lv[l];
        for (int trans = 0; trans < 2; ++trans) {
            Schedule &S = trans ? L.t : L.n;
            long long poff = 0;
            int maxr = 0;
            for (int b : L.blocks) {
                const LRDesc &D = p->lr[b];
                if (D.rank == 0 || caps_only) continue;
                maxr = std::max(maxr, D.rank);
                const int CH = chunk_rows(p, D);
                int nch = (D.n + CH - 1) / CH;
                for (int c = 0; c < nch; ++c) {
                    PanelItem it;
                    if (!trans) {          // V_b^T x[col0 rows]
                        it.f = D.v;
                        it.n = D.n;
                        it.in0 = D.col0;
                    } else {               // Z_l[row0 rows]^T g[row0 rows] (Z_l: ld m, in zpool)
                        it.f = F->zoff[l] + D.row0;
                        it.n = m;
                        it.in0 = D.row0;
                    }
                    it.p = poff;
                    it.rank = D.rank;
                    it.r0 = c * CH;
                    it.len = std::min(CH, D.n - c * CH);
                    it.chunk = c;
                    S.items.push_back(it);
                }
                ReduceItem r;
                r.p = poff;
                r.t = D.toff;
                r.sig = trans ? -1 : D.sig;
                r.rank = D.rank;
                r.nch = nch;
                S.max_nch = std::max(S.max_nch, nch);
                S.reduces.push_back(r);
                poff += (long long)nch * D.rank;
                // update tiles: op N, rows of the block with Z_l (ld m, in
                // zpool); op T, the block's column rows with its V (ld n,
                // in the factor pool)
                const auto rng = tile_range(starts, trans ? D.col0 : D.row0, D.n);
                for (int t = rng.first; t < rng.second; ++t) {
                    const int t0 = starts[t];
                    TileTerm tt;
                    tt.a = trans ? D.v + (t0 - D.col0) : F->zoff[l] + t0;
                    tt.b = D.toff;
                    tt.lda = trans ? D.n : m;
                    tt.K = D.rank;
                    tt.trans_a = 0;
                    tt.src = 0;
                    tt.ldb = D.rank;
                    tt.x_row0 = 0;
                    S.tiles.push_back(make_int2(t0, starts[t + 1] - t0));
                    S.tile_begin.push_back((int)S.terms.size());
                    S.terms.push_back(tt);
                }
            }
            S.tile_begin.push_back((int)S.terms.size());
            S.partial_per_rhs = poff;
            S.t_per_rhs = p->total_rank;
            S.max_rank = maxr;
            S.nb_cap = p->nb_cap;
            for (int nd : L.nodes) {
                const HDesc &H = p->nodes[nd];
                const LRDesc &ne = p->lr[H.ne], &sw = p->lr[H.sw];
                if (ne.rank + sw.rank == 0) continue;
                CapItem c;
                c.k = F->koff[nd];
                c.t1 = ne.toff;
                c.t2 = sw.toff;
                c.s1 = ne.sig;
                c.s2 = sw.sig;
                c.r1 = ne.rank;
                c.r2 = sw.rank;
                S.caps.push_back(c);
            }
        }
    }
    // Leaf step: x[leaf rows] = op(Leaf^-1) b[leaf rows].
    for (int which = 0; which <= F->nsets; ++which) {          // op N, then op T of each set
        const int trans = which > 0;
        Schedule &S = trans ? F->leafT[which - 1] : F->leafN;
        if (trans) tile_starts(p, starts, sweep_rows(p, which - 1, caps_only));
        S.nb_cap = p->nb_cap;
        for (size_t i = 0; i < p->leaves.size(); ++i) {
            const LeafDesc &Lf = p->leaves[i];
            const auto rng = tile_range(starts, Lf.row0, Lf.b);
            for (int t = rng.first; t < rng.second; ++t) {
                const int t0 = starts[t];
                TileTerm tt;
                tt.b = 0;
                tt.lda = Lf.b;
                tt.K = Lf.b;
                tt.src = 1;
                tt.ldb = 0;
                tt.x_row0 = Lf.row0;
                tt.trans_a = trans;
                tt.a = F->leafoff[i] + (trans ? (long long)(t0 - Lf.row0) * Lf.b : (t0 - Lf.row0));
                S.tiles.push_back(make_int2(t0, starts[t + 1] - t0));
                S.tile_begin.push_back((int)S.terms.size());
                S.terms.push_back(tt);
            }
        }
        S.tile_begin.push_back((int)S.terms.size());
    }
}

void factor_free(Plan *p)
{
    Fact *F = (Fact *)p->fact;
    if (!F) return;
    for (LevelOps &L : F->lv) {
        free_schedule(L.n);
        free_schedule(L.t);
    }
    free_schedule(F->leafN);
    for (Schedule &S : F->leafT) free_schedule(S);
    cudaFree(F->zpool);
    cudaFree(F->ztpool);
    cudaFree(F->kpool);
    cudaFree(F->leafinv);
    cudaFree(F->d_tables);
    cudaFree(F->work);
    cudaFree(F->gtr);
    cudaFree(F->rhs);
    cudaFree(F->vec);
    delete F;
    p->fact = nullptr;
}

// Build the level-r right-hand side: factor `which` (0: U, 1: V) of every
// block at level l placed at the block's rows (U: row0, V: col0).
static int level_rhs(Plan *p, Fact *F, int l, int which, cudaStream_t st)
{
    const int width = F->lv[l].width;
    int rc;
    if ((rc = zero_device(F->rhs, (long long)p->m * width, st))) return rc;
    const int cnt = F->scat_count[which][l];
    if (cnt == 0) return 0;
    dim3 g((unsigned)std::min(64, (F->scat_max[which][l] + 255) / 256), (unsigned)cnt);
    scatter_kernel<<<g, 256, 0, st>>>(F->d_scat + F->scat_begin[which][l], p->pool, F->rhs, p->m);
    note_launch();
    DG_CUDA(cudaGetLastError());
    return 0;
}

// Everything of a factorisation that depends on the plan's structure only:
// offsets, device pools, the level schedules, the levels' scatter items and
// capacitance inverse lists.  Built once; refactorisations after a change
// of the values (the adjoint's every step) reuse it.
static int factor_layout(Plan *p, Fact *F, int flags)
{
    F->flags = flags;
    F->transposed = (flags & 1) != 0;
    F->key_chunk = p->chunk_rows;
    F->key_nb = p->nb_cap;
    const int nlev = p->levels;
    F->lv.resize(nlev);
    for (size_t b = 0; b < p->lr.size(); ++b) {
        const LRDesc &D = p->lr[b];
        LevelOps &L = F->lv[D.level];
        L.blocks.push_back((int)b);
        L.width = std::max(L.width, D.rank);
    }
    for (size_t nd = 0; nd < p->nodes.size(); ++nd) F->lv[p->nodes[nd].level].nodes.push_back((int)nd);
    long long z = 0;
    int wmax = 1;
    for (int l = 0; l < nlev; ++l) {
        F->zoff.push_back(z);
        z += align32((long long)p->m * F->lv[l].width);
        wmax = std::max(wmax, F->lv[l].width);
    }
    F->zdoubles = z;
    std::vector<int> ksize(p->nodes.size());
    long long k = 0;
    for (size_t nd = 0; nd < p->nodes.size(); ++nd) {
        int r = p->lr[p->nodes[nd].ne].rank + p->lr[p->nodes[nd].sw].rank;
        F->koff.push_back(k);
        ksize[nd] = r;
        k += align32((long long)r * r);
    }
    F->kdoubles = k;
    std::vector<int> lsize(p->leaves.size());
    std::vector<long long> lsrc(p->leaves.size());
    long long lo = 0;
    for (size_t i = 0; i < p->leaves.size(); ++i) {
        F->leafoff.push_back(lo);
        lsrc[i] = p->leaves[i].d;
        lsize[i] = p->leaves[i].b;
        lo += align32((long long)lsize[i] * lsize[i]);
    }
    F->leafdoubles = lo;
    for (int r : ksize)
        if (r > 1024) return fail(DPLR_GPU_EINVAL, "capacitance order %d exceeds 1024", r);
    for (int b : lsize)
        if (b > 1024) return fail(DPLR_GPU_EINVAL, "leaf size %d exceeds 1024", b);

    int rc;
    auto alloc = [&](double **ptr, long long n) -> int {
        cudaError_t e = dev_malloc((void **)ptr, std::max<long long>(n, 1) * sizeof(double));
        if (e != cudaSuccess)
            return fail(DPLR_GPU_ENOMEM, "factorisation: cannot allocate %lld doubles", n);
        F->bytes += std::max<long long>(n, 1) * 8;
        return 0;
    };
    if ((rc = alloc(&F->zpool, F->zdoubles))) return rc;
    if (F->transposed && (rc = alloc(&F->ztpool, F->zdoubles))) return rc;
    if ((rc = alloc(&F->kpool, F->kdoubles))) return rc;
    if ((rc = alloc(&F->leafinv, F->leafdoubles))) return rc;
    TableBlock tb;
    tb.add(F->leafoff, &F->d_leafoff);
    tb.add(lsrc, &F->d_leafsrc);
    tb.add(lsize, &F->d_leafsize);
    // one info slot per leaf, then one per node (each inverse writes its own)
    std::vector<int> zeros(p->leaves.size() + p->nodes.size() + 1, 0);
    tb.add(zeros, &F->d_info);

    const bool by_tiles = sweep_by_tiles(F);
    if (by_tiles && sweep_rows(p, 0) < 64)
        for (int b : lsize)
            if (b > sweep_rows(p, 0)) F->nsets = 2;
    build_level_schedules(p, F, by_tiles);
    for (LevelOps &L : F->lv) {
        add_schedule(L.n, tb, by_tiles);
        add_schedule(L.t, tb, by_tiles);
    }
    add_schedule(F->leafN, tb, by_tiles);
    // both ops and sets, so that no solve pays for its tables
    for (int v = 0; v < F->nsets; ++v) {
        add_schedule(F->leafT[v], tb);
        for (int trans = 0; trans < 2 && by_tiles; ++trans) build_sweep(p, F, v, trans, tb);
    }

    // scatter items of every level (U, and V for the transposed panels)
    std::vector<ScatterItem> scat;
    for (int which = 0; which < 2; ++which) {
        F->scat_begin[which].assign(nlev, 0);
        F->scat_count[which].assign(nlev, 0);
        F->scat_max[which].assign(nlev, 0);
        for (int l = 0; l < nlev; ++l) {
            F->scat_begin[which][l] = (int)scat.size();
            for (int b : F->lv[l].blocks) {
                const LRDesc &D = p->lr[b];
                if (D.rank == 0) continue;
                ScatterItem it;
                it.src = which == 0 ? D.u : D.v;
                it.row0 = which == 0 ? D.row0 : D.col0;
                it.n = D.n;
                it.rank = D.rank;
                scat.push_back(it);
                F->scat_max[which][l] = std::max(F->scat_max[which][l], D.n * D.rank);
            }
            F->scat_count[which][l] = (int)scat.size() - F->scat_begin[which][l];
        }
    }
    tb.add(scat, &F->d_scat);
    // capacitance inverses of every level
    std::vector<long long> ioff;
    std::vector<int> isize;
    F->inv_begin.assign(nlev, 0);
    F->inv_count.assign(nlev, 0);
    F->inv_max.assign(nlev, 0);
    for (int l = 0; l < nlev; ++l) {
        F->inv_begin[l] = (int)ioff.size();
        for (int nd : F->lv[l].nodes) {
            const HDesc &H = p->nodes[nd];
            int r = p->lr[H.ne].rank + p->lr[H.sw].rank;
            if (r == 0) continue;
            ioff.push_back(F->koff[nd]);
            isize.push_back(r);
            F->inv_ids.push_back(nd);
            F->inv_max[l] = std::max(F->inv_max[l], r);
        }
        F->inv_count[l] = (int)ioff.size() - F->inv_begin[l];
    }
    tb.add(ioff, &F->d_inv_off);
    tb.add(isize, &F->d_inv_size);
    if ((rc = tb.upload(&F->d_tables, &F->bytes))) return rc;
    // scratch for the widest level, so that the numeric pass allocates nothing
    if ((rc = ensure_buffer(&F->rhs, &F->rhs_doubles, (size_t)p->m * wmax))) return rc;
    if (F->transposed && (rc = ensure_buffer(&F->gtr, &F->gtr_doubles, (size_t)p->m * wmax))) return rc;
    return ensure_work(F, p, wmax);
}

// The first nonzero info of the last numeric pass (leaves first, then the
// nodes in factorisation order), reported as DPLR does.
static int factor_check(Plan *p, Fact *F)
{
    const size_t nl = p->leaves.size();
    std::vector<int> info(nl + F->inv_ids.size());
    if (!info.empty())
        DG_CUDA(cudaMemcpy(info.data(), F->d_info, info.size() * sizeof(int), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < nl; ++i)
        if (info[i] != 0) {
            F->sing_kind = 1;
            F->sing_index = (int)i;
            F->sing_info = info[i];
            return fail(DPLR_GPU_ESINGULAR, "leaf %d is singular (zero pivot %d)", (int)i, info[i]);
        }
    for (int l = (int)F->lv.size() - 1; l >= 0; --l)
        for (int q = F->inv_begin[l]; q < F->inv_begin[l] + F->inv_count[l]; ++q)
            if (info[nl + q] != 0) {
                F->sing_kind = 2;
                F->sing_index = F->inv_ids[q];
                F->sing_info = info[nl + q];
                return fail(DPLR_GPU_ESINGULAR, "capacitance %d is singular (zero pivot %d)", q - F->inv_begin[l],
                            info[nl + q]);
            }
    return 0;
}

void factor_invalidate(Plan *p)
{
    if (p->fact) ((Fact *)p->fact)->valid = false;
}

Fact *factor_of(const Plan *p)
{
    Fact *F = (Fact *)p->fact;
    return F && F->valid ? F : nullptr;
}

int factor_build(Plan *p, int flags, cudaStream_t st)
{
    Fact *F = (Fact *)p->fact;
    if (!F || F->flags != flags || F->key_chunk != p->chunk_rows || F->key_nb != p->nb_cap) {
        factor_free(p);
        F = new Fact();
        p->fact = F;
        int rc0 = factor_layout(p, F, flags);
        if (rc0) {
            factor_free(p);
            return rc0;
        }
    }
    F->valid = false;
    int dev = 0;
    DG_CUDA(cudaGetDevice(&dev));
    DG_CUDA(cudaDeviceGetAttribute(&F->sms, cudaDevAttrMultiProcessorCount, dev));
    F->sing_kind = 0;
    F->sing_index = -1;
    F->sing_info = 0;
    int rc;
    const int nlev = (int)F->lv.size();
    int lmax = 0;
    for (const LeafDesc &Lf : p->leaves) lmax = std::max(lmax, Lf.b);

    // Leaf inverses, read straight from the factor pool.
    double lfl = 0.0;
    for (const LeafDesc &Lf : p->leaves) lfl += 2.0 * Lf.b * Lf.b * (double)Lf.b;
    if ((rc = batched_inverse(F->leafinv, F->d_leafoff, F->d_leafsize, p->pool, F->d_leafsrc,
                              (int)p->leaves.size(), lmax, F->d_info, F->sms, st, lfl)))
        return rc;

    // Levels bottom-up: Z_l (and Zt_l) through the already factored
    // deeper levels, then the capacitance matrices of level l.
    for (int l = nlev - 1; l >= 0; --l) {
        LevelOps &L = F->lv[l];
        if (L.width == 0) continue;
        if (F->transposed) {
            if ((rc = level_rhs(p, F, l, 1, st))) return rc;
            if ((rc = sweep(p, F, 1, l + 1, F->rhs, p->m, F->ztpool + F->zoff[l], p->m, L.width, st)))
                return rc;
        }
        // Z_l, and S V^T Z_l of the level's blocks in T; then K per node
        if ((rc = level_rhs(p, F, l, 0, st))) return rc;
        if ((rc = sweep(p, F, 0, l + 1, F->rhs, p->m, F->zpool + F->zoff[l], p->m, L.width, st, l))) return rc;
        double *T = F->work;
        if (!L.n.caps.empty()) {
            assemble_k_kernel<<<(unsigned)L.n.caps.size(), 256, 0, st>>>(L.n.d_caps, T, L.width,
                                                                         F->kpool);
            note_launch();
            DG_CUDA(cudaGetLastError());
            // invert this level's capacitance matrices (info slots after the leaves')
            const int b0 = F->inv_begin[l];
            double kfl = 0.0;
            for (int q = b0; q < b0 + F->inv_count[l]; ++q) {
                const HDesc &H = p->nodes[F->inv_ids[q]];
                const double r = p->lr[H.ne].rank + p->lr[H.sw].rank;
                kfl += 2.0 * r * r * r;
            }
            if ((rc = batched_inverse(F->kpool, F->d_inv_off + b0, F->d_inv_size + b0, nullptr, nullptr,
                                      F->inv_count[l], F->inv_max[l], F->d_info + p->leaves.size() + b0, F->sms, st, kfl)))
                return rc;
        }
    }
    DG_CUDA(cudaStreamSynchronize(st));
    if ((rc = factor_check(p, F))) return rc;
    F->valid = true;
    return 0;
}

int factor_solve(Plan *p, int trans, int nrhs, const double *B, int ldb, double *X, int ldx,
                 cudaStream_t st)
{
    Fact *F = factor_of(p);
    if (!F) return fail(DPLR_GPU_ESTATE, "solve: plan is not factored");
    if (nrhs <= 0 || p->m == 0) return 0;
    return sweep(p, F, trans, 0, B, ldb, X, ldx, nrhs, st);
}

long long factor_bytes(const Plan *p)
{
    const Fact *F = (const Fact *)p->fact;
    if (!F) return 0;
    return F->bytes + (long long)(F->work_doubles + F->rhs_doubles + F->vec_doubles + F->gtr_doubles) * 8;
}

}  // namespace dg
