// sweep.cuh -- the Woodbury sweep by row tiles: what one level does to a row
// tile and what the next level needs from it run in one launch.
//
// A level of the sweep is x -= A W over the rows of its blocks (A = Z, W the
// capacitance product) after T = B^T x (B = V).  As separate launches (panel,
// reduce, capacitance, update) every level reads x twice and writes it once,
// and a solve of one right-hand side is 4 launches per level.  Here a CTA owns a
// row tile (at most 64 rows) and a column tile:
//   first launch  x = leaf^-1 b (or x = b), then the tile's part of the first
//                 level's T;
//   per level     x -= A W, then the tile's part of the next level's T from the
//                 new x in shared memory;
// and W comes either from the reduce and capacitance launches between two
// levels, or, where summing the node's parts and multiplying its few rows of
// K^-1 costs a tile less than a launch (sweep_fused), from the CTA itself.  The
// tiles of A and B are fetched by cp.async before anything else, so their
// latency overlaps the sums; with one right-hand side that is before the level in
// front has ended (a chained launch).
// Measured on a GB300 against four launches per level (with the tiles of
// fp64tile.cuh), us:
//   one solve, N = 16384, leaf 128, rank 16: 1 RHS 191 -> 100 (82 chained), 16 RHS 556 -> 310
//   one solve, N = 65536, leaf 256, rank 48, 16 RHS   2554 -> 2262
//   factorisation and solve, N = 8192, leaf 64, rank 8   1512 -> 927
//   factorisation and solve, N = 32768, leaf 256, rank 64   29424 -> 28321
#pragma once

#include "fp64tile.cuh"

namespace dg {

constexpr int kSweepRank = 64;           // largest rank of a level's blocks
constexpr int kSweepSum = 8192;          // largest fused sum: parts x right-hand sides
constexpr int kSweepT = 1024;            // largest fused node: order x right-hand sides
constexpr int kSweepK = 2048;            // largest fused rows of K^-1: rank x order

// Whether the tiles of a level form W themselves: only where the level is a few
// CTAs per SM, so that launches and their latency are what it costs (with
// thousands of tiles the repeated sums cost more: 64 matrices of N = 1024 to
// 8192, 8 right-hand sides, 638 us unfused, 712 fused; one N = 16384 solve 137
// us unfused and 100 fused by plain launches, 127 and 82 chained), and where the
// repeated sums and rows of K^-1 stay small beside the tile's own products.
inline bool sweep_fused(long long ctas, int sms, long long sum, long long order, long long rank_order)
{
    return ctas <= 4LL * sms && sum <= kSweepSum && order <= kSweepT && rank_order <= kSweepK;
}

// One row tile in one phase of the sweep.
struct SweepTile {
    long long ua;        // update: offset of A's (tile row 0, column 0), ld ulda
    long long pf;        // panel: offset of B's (tile row 0, column 0), ld pld
    long long pp;        // panel: offset of the tile's part / nrhs (ld prank)
    int row0, h;
    int ulda, urank;     // urank 0: no block of this level covers the tile
    int ut, urow;        // offset / nrhs of the block's W; its first row in the node
    int cap;             // the node's item in the level's capacitance list
    int pld, prank;      // prank 0: no panel
    int pad;
};

struct SweepArgs {
    const SweepTile *tiles;
    const double *ubase, *pbase;
    const double *xin;   // x before this phase (the sweep's input in the first)
    double *x;
    double *parts;       // the next level's parts, written
    // W: given, or formed here from this level's parts
    const double *W;
    const CapItem *caps;
    const ReduceItem *reds;      // two per capacitance item, in its order
    const double *parts_in, *kbase, *sigpool;
    int trans;           // op T: W = S K^-T T; op N: W = K^-1 (S T)
    int ldin, ldx, nrhs, nbt, rmax, pmax;
    int kmax, tmax;      // fused: largest rank x order, order x nbt
};

constexpr int kSweepLd = 65;             // row stride of the update's A in shared memory

// Shared memory in doubles: the update's A and W, the new x, the panel's B, the
// reductions, and the fused rows of K^-1 and sums.
__host__ __device__ constexpr int sweep_smem(int rmax, int pmax, int nbt, int kmax, int tmax)
{
    return kSweepLd * rmax + rmax * nbt + 64 * (nbt | 1) + 64 * (pmax | 1) + 4 * kTT + kmax + tmax;
}

// What any level and any first phase may need (bytes; 113 KB).
constexpr size_t kSweepSmemMost = sizeof(double) * sweep_smem(kSweepRank, kSweepRank, kColTile, kSweepK, kSweepT);
static_assert(sizeof(double) * (kTileSmem + 64 * (kColTile | 1) + 64 * (kSweepRank | 1)) <= kSweepSmemMost,
              "first phase of op N");

// Largest power of two p <= 32 with count * p <= kTT: adjacent lanes that share
// one of `count` outputs (their sums meet in log2 p shuffles).
__device__ __forceinline__ int sweep_split(int count)
{
    int lg = 0;
    while (lg < 5 && count << (lg + 1) <= kTT) ++lg;
    return lg;
}

__device__ __forceinline__ double sweep_lanes(double v, int lg)
{
    for (int o = (1 << lg) >> 1; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// This tile's part of the panel: P (rank x nj) = Bs^T Xs over h rows; Bs (h x
// rank, row stride rank | 1) and Xs (row stride nj | 1) in shared memory.
__device__ __forceinline__ void sweep_panel(const double *Bs, const double *Xs, int h, int rank, int nj,
                                            double *__restrict__ P, double *red, int t)
{
    const int cnt = rank * nj, ldb = rank | 1, ldx = nj | 1;
    if (2 * cnt <= kTT) {                         // adjacent lanes share an output
        const int lg = sweep_split(cnt), per = 1 << lg, e = t >> lg, s = t & (per - 1);
        const int k = e % rank, j = e / rank;
        double v = 0.0;
        if (e < cnt)
            for (int r = s; r < h; r += per) v = fma(Bs[r * ldb + k], Xs[r * ldx + j], v);
        v = sweep_lanes(v, lg);
        if (e < cnt && s == 0) P[e] = v;
        return;
    }
    const int JG = kPanelGroups.jg[rank - 1][nj - 1], RG = kTT / (rank * JG);
    const int kk = t % rank, rest = t / rank, jg = rest % JG, rg = rest / JG;
    const int nq = (nj - jg + JG - 1) / JG;
    const bool active = rg < RG;
    const int nqw = __reduce_max_sync(0xffffffffu, active ? nq : 0);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    tile_fma_n(nqw, Bs + kk, ldb, Xs + jg, ldx, JG, rg, RG, h, acc);
    if (RG > 1) {
        if (active && rg > 0)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < nq) red[q * kTT + t] = acc[q];
        __syncthreads();
        if (rg == 0)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < nq)
                    for (int g = 1; g < RG; ++g) acc[q] += red[q * kTT + t + g * rank * JG];
    }
    if (rg == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < nq) P[kk + (long long)(jg + JG * q) * rank] = acc[q];
}

__device__ __forceinline__ void sweep_fetch_panel(const SweepTile &tl, const double *pbase, double *Bs, int t)
{
    const double *src = pbase + tl.pf;
    const int ld = tl.prank | 1, i = t & 63;
    if (i < tl.h)
        for (int k = t >> 6; k < tl.prank; k += kTT / 64) cp_async8(Bs + i * ld + k, src + i + (long long)k * tl.pld);
}

// Sums over the parts of a node's two blocks for one column tile (times sig
// where sig >= 0) into Ts[k + j * (r1 + r2)].  The 256 threads are 2^lg part
// groups x the elements of both blocks (elements contiguous, so that a part is
// read in full lines); groups meet in shared memory, then in shuffles.  The parts
// are written while a chained kernel already lives: ordinary loads.  red: kTT
// doubles.  All threads call it; ends with a barrier.
__device__ __forceinline__ void sweep_sums(const ReduceItem *__restrict__ pair, const double *parts,
                                           const double *sigpool, int nrhs, int j0, int nj, double *Ts, double *red,
                                           int t)
{
    const ReduceItem R0 = pair[0], R1 = pair[1];
    const int c0 = R0.rank * nj, cnt = c0 + R1.rank * nj, ld = R0.rank + R1.rank;
    for (int e0 = 0; e0 < cnt; e0 += kTT) {
        const int live = min(kTT, cnt - e0), lg = sweep_split(live), per = 1 << lg;
        const int s = t / live, ea = e0 + t - s * live;
        const bool second = ea >= c0;
        double v = 0.0;
        if (s < per) {
            const ReduceItem &R = second ? R1 : R0;
            const int e = second ? ea - c0 : ea;
            const double *P = parts + R.p * nrhs + (long long)j0 * R.rank + e;
            const long long step = (long long)R.rank * nrhs;
            double v1 = 0.0, v2 = 0.0, v3 = 0.0;
            int c = s;
            for (; c + 3 * per < R.nch; c += 4 * per) {
                v += P[c * step];
                v1 += P[(c + per) * step];
                v2 += P[(c + 2 * per) * step];
                v3 += P[(c + 3 * per) * step];
            }
            for (; c < R.nch; c += per) v += P[c * step];
            v = (v + v1) + (v2 + v3);
        }
        int eo = ea;
        if (per > 1) {                            // group s of element ea -> adjacent lanes
            red[t] = v;
            __syncthreads();
            const int el = t >> lg, g = t & (per - 1);
            v = sweep_lanes(el < live ? red[g * live + el] : 0.0, lg);
            eo = el < live && g == 0 ? e0 + el : -1;
        } else if (s > 0) {
            eo = -1;
        }
        if (eo >= 0) {
            const bool b = eo >= c0;
            const ReduceItem &R = b ? R1 : R0;
            const int e = b ? eo - c0 : eo, k = e % R.rank, j = e / R.rank;
            if (R.sig >= 0) v *= __ldg(sigpool + R.sig + k);
            Ts[(b ? R0.rank : 0) + k + j * ld] = v;
        }
        __syncthreads();
    }
}

// One level (or, with urank 0 everywhere and xin != x, the first phase of op
// T): grid (tiles, column tiles).
template <bool FUSED>
__global__ void __launch_bounds__(kTT) sweep_level_kernel(const SweepArgs a)
{
    extern __shared__ __align__(16) double sm[];
    const SweepTile tl = a.tiles[blockIdx.x];
    const bool copy = a.xin != a.x;
    if (tl.urank == 0 && tl.prank == 0 && !copy) return;
    const int t = threadIdx.x, j0 = blockIdx.y * a.nbt, nj = min(a.nbt, a.nrhs - j0), h = tl.h, K = tl.urank;
    double *As = sm, *Ws = As + kSweepLd * a.rmax, *Xs = Ws + a.rmax * a.nbt, *Bs = Xs + 64 * (a.nbt | 1);
    double *red = Bs + 64 * (a.pmax | 1), *Ks = red + 4 * kTT, *Ts = Ks + a.kmax;
    const int ldx = nj | 1;
    CapItem c = {};
    if (K > 0) {
        if (FUSED) c = a.caps[tl.cap];
        const double *A = a.ubase + tl.ua;
        const int i = t & 63;
        if (i < h)
            for (int k = t >> 6; k < K; k += kTT / 64) cp_async8(As + k * kSweepLd + i, A + i + (long long)k * tl.ulda);
    }
    const int r = c.r1 + c.r2;
    if (FUSED && K > 0) {
        const double *Kg = a.kbase + c.k;
        // rows urow .. urow + K of K^-1 (op T: columns, as rows)
        for (int e = t; e < K * r; e += kTT) {
            const int k = e % K, q = e / K;
            cp_async8(Ks + e, a.trans ? Kg + q + (long long)(tl.urow + k) * r : Kg + tl.urow + k + (long long)q * r);
        }
    }
    if (tl.prank > 0) sweep_fetch_panel(tl, a.pbase, Bs, t);
    cp_commit();
    // from here on, what the kernels in front wrote: x, the parts, W
    const double *parts_in = chain_wait(a.parts_in);
    {
        const int i = t & 63;
        if (i < h)
            for (int j = t >> 6; j < nj; j += kTT / 64)
                cp_async8(Xs + i * ldx + j, a.xin + tl.row0 + i + (long long)(j0 + j) * a.ldin);
    }
    if (!FUSED && K > 0) {
        const double *W = a.W + (long long)tl.ut * a.nrhs + (long long)j0 * K;
        for (int e = t; e < K * nj; e += kTT) cp_async8(Ws + e, W + e);
    }
    cp_commit();
    if (FUSED && K > 0) {
        sweep_sums(a.reds + 2 * tl.cap, parts_in, a.sigpool, a.nrhs, j0, nj, Ts, red, t);
        cp_wait<1>();
        __syncthreads();
        // W: adjacent lanes share an element where there are few
        const int cnt = K * nj, lg = sweep_split(cnt), per = 1 << lg, s = t & (per - 1);
        for (int e0 = 0; e0 < cnt; e0 += kTT >> lg) {
            const int e = e0 + (t >> lg), k = e % K, j = e / K;
            double w = 0.0, w1 = 0.0;
            if (e < cnt) {
                int q = s;
                for (; q + per < r; q += 2 * per) {
                    w = fma(Ks[k + q * K], Ts[q + j * r], w);
                    w1 = fma(Ks[k + (q + per) * K], Ts[q + per + j * r], w1);
                }
                if (q < r) w = fma(Ks[k + q * K], Ts[q + j * r], w);
            }
            w = sweep_lanes(w + w1, lg);
            if (e < cnt && s == 0) {
                if (a.trans) {
                    const int i = tl.urow + k;
                    w *= __ldg(a.sigpool + (i < c.r1 ? c.s1 + i : c.s2 + i - c.r1));
                }
                Ws[e] = w;
            }
        }
    }
    cp_wait<0>();
    __syncthreads();
    // x -= A W
    double *x = a.x + tl.row0 + (long long)j0 * a.ldx;
    const int cnt = h * nj;
    if (K == 0) {
        if (copy)
            for (int e = t; e < cnt; e += kTT) x[e % h + (long long)(e / h) * a.ldx] = Xs[(e % h) * ldx + e / h];
    } else if (2 * cnt <= kTT) {                  // adjacent lanes share an element
        const int lg = min(sweep_split(cnt), 2), per = 1 << lg;
        const int e = t >> lg, s = t & (per - 1), i = e % h, j = e / h;
        double v = 0.0;
        if (e < cnt)
            for (int k = s; k < K; k += per) v = fma(As[k * kSweepLd + i], Ws[k + j * K], v);
        v = sweep_lanes(v, lg);
        if (e < cnt && s == 0) {
            v = Xs[i * ldx + j] - v;
            Xs[i * ldx + j] = v;
            x[i + (long long)j * a.ldx] = v;
        }
    } else {
        // columns jg, jg + G, ...: at most four (G >= 4, nj <= 16), and only as many
        // multiply-adds as the warp has columns (four under a predicate each: 4
        // right-hand sides, N = 131072, leaf 256, rank 32 1937 us).  A warp of two
        // jg may read G columns past W and drop them: G < 16 then, within Xs, Bs
        // and red.
        const int G = kTT / h, i = t % h, j = t / h, nq = j < G ? (nj - j + G - 1) / G : 0;
        const int nqw = __reduce_max_sync(0xffffffffu, nq);
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        tile_fma_n(nqw, As + i, kSweepLd, Ws + (nq > 0 ? j * K : 0), 1, G * K, 0, 1, K, acc);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < nq) {
                const double v = Xs[i * ldx + j + q * G] - acc[q];
                Xs[i * ldx + j + q * G] = v;
                x[i + (long long)(j + q * G) * a.ldx] = v;
            }
    }
    if (tl.prank > 0) {
        __syncthreads();
        chain_next();
        sweep_panel(Bs, Xs, h, tl.prank, nj, a.parts + tl.pp * a.nrhs + (long long)j0 * tl.prank, red, t);
    }
}

// First phase of op N: x = leaf^-1 b and the deepest level's parts.  ubase:
// the leaf inverses; ua, ulda, urank: the tile's rows of its leaf's (urank = the
// leaf's order); ut: the leaf's first row.
__global__ void __launch_bounds__(kTT) sweep_leaf_kernel(const SweepArgs a)
{
    extern __shared__ __align__(16) double sm[];
    const SweepTile tl = a.tiles[blockIdx.x];
    const int t = threadIdx.x, j0 = blockIdx.y * a.nbt, nj = min(a.nbt, a.nrhs - j0);
    double *Xs = sm + kTileSmem, *Bs = Xs + 64 * (a.nbt | 1);
    if (tl.prank > 0) sweep_fetch_panel(tl, a.pbase, Bs, t);
    cp_commit();
    auto term = [&](int) {
        ExpandTerm e;
        e.a = a.ubase + tl.ua;
        e.b = a.xin + tl.ut + (long long)j0 * a.ldin;
        e.lda = tl.ulda;
        e.ldb = a.ldin;
        e.K = tl.urank;
        e.row_major = e.cg = false;
        return e;
    };
    auto out = [&](int i, int j, double v) {
        a.x[tl.row0 + i + (long long)(j0 + j) * a.ldx] = v;
        Xs[i * (nj | 1) + j] = v;
    };
    expand_tile(tl.h, 1, term, nj, out, sm, blockIdx.x);      // ends with a barrier
    if (tl.prank > 0) {
        cp_wait<0>();
        __syncthreads();
        chain_next();
        sweep_panel(Bs, Xs, tl.h, tl.prank, nj, a.parts + tl.pp * a.nrhs + (long long)j0 * tl.prank, sm, t);
    }
}

}  // namespace dg
