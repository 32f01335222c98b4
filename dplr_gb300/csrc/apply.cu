// apply.cu -- FP64 PLR apply  Y := alpha*op(A)*X + beta*Y  on the GPU.
//
// DPLR recurses over the tree and makes two BLAS-2/3 calls per low-rank
// block plus one per leaf (src/dplrpmv.c:19-180, src/dplrpdmm.c:23-241).
// Here the whole tree is applied in three launches over the block table:
//   1. panel:  for every (block, row chunk) item, the partial product
//              F_in[chunk]^T X[chunk rows]  (F_in = V for op N, U for op T)
//   2. reduce: T_b = sig_b o sum_chunks(partials)           (rank x nrhs)
//   3. expand: for every row tile of Y, the sum over levels of
//              F_out[tile] T_b  plus the leaf term  D[tile] X[leaf rows]
//              (D^T for op T), then Y = alpha*acc + beta*Y (beta == 0 does
//              not read Y).
// Every output element is written by exactly one thread (no atomics), so
// results are deterministic.  FP64 on GB300 runs at ~1.2 TFLOP/s, so for
// more than a few right-hand sides the kernels are FP64-issue bound; the
// smem staging only has to keep HBM traffic low, not feed tensor cores.
#include "internal.cuh"
#include "fp64tile.cuh"

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>

namespace dg {

constexpr int kThreads = kTT;

// ----------------------------------------------------------------- panel
// One CTA per (item, tile of nbt right-hand sides): panel_tile (fp64tile.cuh).
__global__ void __launch_bounds__(kThreads, kTileCtas) panel_kernel(
    const PanelItem *__restrict__ items, const double *__restrict__ fbase, const double *__restrict__ X, int ldx,
    int nrhs, int nbt, double *__restrict__ partials)
{
    __shared__ __align__(16) double sm[kTileSmem];
    const PanelItem it = items[blockIdx.x];
    const int j0 = blockIdx.y * nbt, nj = min(nbt, nrhs - j0);
    panel_tile(fbase + it.f + it.r0, it.n, it.len, it.rank, X + (long long)j0 * ldx + it.in0 + it.r0, ldx, nj,
               partials + it.p * nrhs + (long long)it.chunk * it.rank * nrhs + (long long)j0 * it.rank, sm, blockIdx.x);
    chain_next();
}

// ------------------------------------------------------- one right-hand side
// With a single right-hand side the apply is a pair of matrix-vector products
// that stream every factor once: HBM- (and on GB300 FP64-FMA-) bound.  These
// kernels read the factors straight from global memory with 16-byte loads,
// several columns in flight per warp, and keep only x in shared memory.

constexpr int kPanel1MaxLen = 2048;

// Panel, 1 RHS: P[k] = F[r0:r0+len, k]^T x[in0+r0 : ...]; warp w handles
// columns k = w, w+8, ... four at a time; shuffle reduction per column.
__global__ void __launch_bounds__(kThreads) panel1_kernel(const PanelItem *__restrict__ items,
                                                          const double *__restrict__ fbase,
                                                          const double *__restrict__ X,
                                                          double *__restrict__ partials)
{
    __shared__ __align__(16) double xs[kPanel1MaxLen];
    const PanelItem it = items[blockIdx.x];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int r = t; r < it.len; r += kThreads) xs[r] = X[it.in0 + it.r0 + r];
    __syncthreads();
    const double *F = fbase + it.f + it.r0;
    double *P = partials + it.p + (long long)it.chunk * it.rank;
    const bool vec = ((it.f | it.n | it.r0 | it.len) & 1) == 0;   // 16-byte loads of the factor
    for (int k0 = warp; k0 < it.rank; k0 += 4 * (kThreads / 32)) {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        if (vec) {
            for (int r = 2 * lane; r < it.len; r += 64) {
                const double2 xv = *reinterpret_cast<const double2 *>(xs + r);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int k = k0 + c * (kThreads / 32);
                    if (k < it.rank) {
                        const double2 fv = __ldg(reinterpret_cast<const double2 *>(F + (long long)k * it.n + r));
                        acc[c] = fma(fv.x, xv.x, fma(fv.y, xv.y, acc[c]));
                    }
                }
            }
        } else {
            for (int r = lane; r < it.len; r += 32) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int k = k0 + c * (kThreads / 32);
                    if (k < it.rank) acc[c] = fma(__ldg(F + (long long)k * it.n + r), xs[r], acc[c]);
                }
            }
        }
        // butterfly reduction of the four column sums: two exchange rounds
        // leave lane l with the partial of column (l >> 3) & 3, three more
        // finish it (6 FP64 adds per lane instead of 20)
        {
            const bool hi16 = lane & 16, hi8 = lane & 8;
            const double s0 = hi16 ? acc[0] : acc[2], s1 = hi16 ? acc[1] : acc[3];
            double a0 = (hi16 ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, s0, 16);
            double a1 = (hi16 ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, s1, 16);
            // lanes < 16 now hold columns {0, 1}, lanes >= 16 columns {2, 3}
            const double t = hi8 ? a0 : a1;
            double v = (hi8 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, t, 8);
            // lane l holds column 2*(l >= 16) + (l & 8 ? 1 : 0)
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const int c = (hi16 ? 2 : 0) + (hi8 ? 1 : 0);
            const int k = k0 + c * (kThreads / 32);
            if ((lane & 7) == 0 && k < it.rank) P[k] = v;
        }
    }
    chain_next();
}

// A chained expand starts while the last panels still run: its tiles go where
// room is first, and beyond eight of them per SM the load evens out (N = 131072,
// leaf 256, rank 32, 2048 tiles: 243 -> 231 us, the reduce and the launches
// hidden).  With a wave or two they crowd on a few SMs (N = 3200, leaf 50, 55
// right-hand sides: 125 -> 180 us), so fewer tiles, and the kernel for several
// right-hand sides, are launched plainly.
constexpr int kChainTiles = 8 * 152;

// Expand, 1 RHS: y[tile] = alpha * sum_terms A[tile, 0:K] b + beta y.  Thread
// (i, g) owns row i of the tile and the inner indices k == g (mod G); the G
// partial sums meet in shared memory.  A term may be row-major (the leaves of op T):
//   kDotRows    dot products, four rows per warp at a time, their sums by the
//               panel's butterfly (6 additions for four rows); 64 registers;
//   kShortRows  as a column-major term, its sectors shared in L1, for short tiles
//               and leaves, where the dot products leave half of their rows empty
//               and the registers half of the CTAs out.
enum RowMajor { kNoRows, kDotRows, kShortRows };

template <RowMajor ROWS>
__global__ void __launch_bounds__(kThreads) expand1_kernel(
    const double *__restrict__ abase, const TileTerm *__restrict__ terms, const int2 *__restrict__ tiles,
    const int *__restrict__ tile_begin, const double *__restrict__ T, const double *__restrict__ X,
    double *__restrict__ Y, double alpha, double beta)
{
    __shared__ double red[kThreads], dots[ROWS == kDotRows ? 64 : 1];
    const int tile = blockIdx.x, row0 = tiles[tile].x, R = tiles[tile].y;
    const int t = threadIdx.x, G = kThreads / R, i = t % R, g = t / R;
    double acc = 0.0, acc2 = 0.0;
    bool rows = false;
    for (int q = tile_begin[tile]; q < tile_begin[tile + 1]; ++q) {
        const TileTerm tt = terms[q];
        // (a second wait returns at once.  Ordinary loads of T: the read-only path is
        // for what nobody writes while the kernel lives, and a chained one lives
        // before T is written)
        const double *B = tt.src == 1 ? X + tt.x_row0 : chain_wait(T + tt.b);
        if (ROWS == kDotRows && tt.trans_a) {            // one per tile: its leaf
            rows = true;
            const int lane = t & 31, W = kThreads / 32;
            const bool hi16 = lane & 16, hi8 = lane & 8;
            for (int r0 = t >> 5; r0 < R; r0 += 4 * W) {
                double s[4] = {0.0, 0.0, 0.0, 0.0};
                for (int k = lane; k < tt.K; k += 32) {
                    const double b = B[k];
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (r0 + c * W < R)
                            s[c] = fma(__ldg(abase + tt.a + (long long)(r0 + c * W) * tt.lda + k), b, s[c]);
                }
                const double s0 = hi16 ? s[0] : s[2], s1 = hi16 ? s[1] : s[3];
                const double a0 = (hi16 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, s0, 16);
                const double a1 = (hi16 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, s1, 16);
                double v = (hi8 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, hi8 ? a0 : a1, 8);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                const int r = r0 + ((hi16 ? 2 : 0) + (hi8 ? 1 : 0)) * W;
                if ((lane & 7) == 0 && r < R) dots[r] = v;
            }
            continue;
        }
        if (g >= G) continue;
        const bool row = ROWS == kShortRows && tt.trans_a;
        const double *A = abase + tt.a + (row ? (long long)i * tt.lda : i);
        const long long lda = row ? 1 : tt.lda;
        int k = g;
        for (; k + G < tt.K; k += 2 * G) {
            acc = fma(__ldg(A + k * lda), B[k], acc);
            acc2 = fma(__ldg(A + (k + G) * lda), B[k + G], acc2);
        }
        if (k < tt.K) acc = fma(__ldg(A + k * lda), B[k], acc);
    }
    red[t] = acc + acc2;
    __syncthreads();
    chain_wait();
    if (t < R) {
        double s = ROWS == kDotRows && rows ? dots[t] : 0.0;
        for (int gg = 0; gg < G; ++gg) s += red[gg * R + t];
        double *y = Y + row0 + t;
        *y = beta == 0.0 ? alpha * s : fma(alpha, s, beta * *y);
    }
}

// ---------------------------------------------------------------- reduce
// T[k, j] = sig[k] * sum_c P[c][k, j] (no scaling with a null sigbase); grid:
// (item, elements).  With few right-hand sides, or in items of many chunks, the
// chunk sums of an element are spread over 8 warps (32 elements x 8 chunk groups
// per CTA, four loads in flight each) instead of one thread walking all chunks:
// 54 us for the 512 chunks of a level of N = 32768, 6 us grouped.  More than
// 65535 CTAs of 32 elements (rank 512 and 4096 right-hand sides) are past a
// grid's limit in y and fill the chip with a thread per element.
constexpr int kGroupedChunks = 64, kGridY = 65535;

__global__ void __launch_bounds__(256) reduce_kernel(const ReduceItem *__restrict__ items,
                                                     const double *__restrict__ sigbase,
                                                     const double *__restrict__ partials, int nrhs,
                                                     int grouped_from, double *__restrict__ T)
{
    __shared__ double red[8][33];
    chain_next();
    const ReduceItem R = items[blockIdx.x];
    const double *parts = chain_wait(partials);
    const long long cnt = (long long)R.rank * nrhs;
    double s = 0.0;
    long long e;
    if (R.nch >= grouped_from) {
        const int el = threadIdx.x & 31, grp = threadIdx.x >> 5;
        e = (long long)blockIdx.y * 32 + el;
        if ((long long)blockIdx.y * 32 >= cnt) return;
        if (e < cnt) {
            const double *P = parts + R.p * nrhs + e;
            double s1 = 0.0, s2 = 0.0, s3 = 0.0;
            int c = grp;
            for (; c + 24 < R.nch; c += 32) {
                s += P[(long long)c * cnt];
                s1 += P[(long long)(c + 8) * cnt];
                s2 += P[(long long)(c + 16) * cnt];
                s3 += P[(long long)(c + 24) * cnt];
            }
            for (; c < R.nch; c += 8) s += P[(long long)c * cnt];
            s = (s + s1) + (s2 + s3);
        }
        red[grp][el] = s;
        __syncthreads();
        if (grp != 0 || e >= cnt) return;
        s = 0.0;
#pragma unroll
        for (int g = 0; g < 8; ++g) s += red[g][el];
    } else {
        e = (long long)blockIdx.y * 256 + threadIdx.x;
        if (e >= cnt) return;
        const double *P = parts + R.p * nrhs + e;
        double s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int c = 0;
        for (; c + 3 < R.nch; c += 4) {
            s += P[(long long)c * cnt];
            s1 += P[(long long)(c + 1) * cnt];
            s2 += P[(long long)(c + 2) * cnt];
            s3 += P[(long long)(c + 3) * cnt];
        }
        for (; c < R.nch; ++c) s += P[(long long)c * cnt];
        s = (s + s1) + (s2 + s3);
    }
    T[R.t * nrhs + e] = (R.sig >= 0 && sigbase) ? sigbase[R.sig + (int)(e % R.rank)] * s : s;
}

// ---------------------------------------------------------------- expand
// One CTA per (row tile, tile of nbt right-hand sides): expand_tile.
__global__ void __launch_bounds__(kThreads, kTileCtas) expand_kernel(
    const double *__restrict__ abase, const TileTerm *__restrict__ terms, const int2 *__restrict__ tiles,
    const int *__restrict__ tile_begin, const double *__restrict__ T, const double *__restrict__ X, int ldx,
    double *__restrict__ Y, int ldy, int nrhs, int nbt, double alpha, double beta)
{
    __shared__ __align__(16) double sm[kTileSmem];
    const int2 tile = tiles[blockIdx.x];
    const int q0 = tile_begin[blockIdx.x];
    const int j0 = blockIdx.y * nbt, nj = min(nbt, nrhs - j0);
    auto term = [&](int q) {
        const TileTerm tt = terms[q0 + q];
        ExpandTerm e;
        e.a = abase + tt.a;
        e.lda = tt.lda;
        e.K = tt.K;
        e.row_major = tt.trans_a != 0;
        e.cg = false;
        if (tt.src == 1) {
            e.b = X + tt.x_row0 + (long long)j0 * ldx;
            e.ldb = ldx;
        } else {
            e.b = T + (tt.src == 0 ? tt.b * nrhs : tt.b) + (long long)j0 * tt.ldb;
            e.ldb = tt.ldb;
        }
        return e;
    };
    auto out = [&](int i, int j, double s) {
        double *y = Y + tile.x + i + (long long)(j0 + j) * ldy;
        *y = beta == 0.0 ? alpha * s : fma(alpha, s, beta * *y);
    };
    expand_tile(tile.y, tile_begin[blockIdx.x + 1] - q0, term, nj, out, sm, blockIdx.x);
}

// ----------------------------------------------------------- capacitance
// W = op(Kinv) [T1; T2] of one H node (rows times [sig1; sig2] when scaled) as
// an expand of two terms: the columns of Kinv for T1 and those for T2.  grid:
// (node, right-hand-side tile, row tile); row tiles past the node's are empty.
__global__ void __launch_bounds__(kThreads, kTileCtas) cap_kernel(
    const CapItem *__restrict__ items, const double *__restrict__ kbase,
    const double *__restrict__ sigbase, int trans, int scaled, const double *__restrict__ T,
    double *__restrict__ W, int nrhs, int nbt)
{
    __shared__ __align__(16) double sm[kTileSmem];
    const CapItem c = items[blockIdx.x];
    const int r = c.r1 + c.r2, nt = (r + 63) / 64;
    if ((int)blockIdx.z >= nt) return;
    const int i0 = (int)((long long)blockIdx.z * r / nt), h = (int)((long long)(blockIdx.z + 1) * r / nt) - i0;
    const int j0 = blockIdx.y * nbt, nj = min(nbt, nrhs - j0);
    const double *K = kbase + c.k;
    auto term = [&](int q) {
        const int k0 = q == 0 ? 0 : c.r1;
        ExpandTerm e;
        e.a = trans ? K + (long long)i0 * r + k0 : K + i0 + (long long)k0 * r;
        e.lda = r;
        e.K = q == 0 ? c.r1 : c.r2;
        e.row_major = trans != 0;
        e.cg = false;
        e.b = q == 0 ? T + c.t1 * nrhs + (long long)j0 * c.r1 : T + c.t2 * nrhs + (long long)j0 * c.r2;
        e.ldb = q == 0 ? c.r1 : c.r2;
        return e;
    };
    auto out = [&](int ii, int j, double v) {
        const int i = i0 + ii;
        if (scaled) v *= i < c.r1 ? sigbase[c.s1 + i] : sigbase[c.s2 + i - c.r1];
        if (i < c.r1)
            W[c.t1 * nrhs + i + (long long)(j0 + j) * c.r1] = v;
        else
            W[c.t2 * nrhs + (i - c.r1) + (long long)(j0 + j) * c.r2] = v;
    };
    expand_tile(h, 2, term, nj, out, sm, blockIdx.x);
}

// ------------------------------------------------------------- utilities
__global__ void scale_kernel(double *Y, int rows, int cols, int ldy, double beta)
{
    long long n = (long long)rows * cols;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        int r = (int)(e % rows), c = (int)(e / rows);
        double *y = Y + r + (long long)c * ldy;
        *y = beta == 0.0 ? 0.0 : beta * *y;
    }
}

__global__ void transpose_kernel(const double *__restrict__ src, int rows, int cols, int lds,
                                 double *__restrict__ dst, int ldd)
{
    __shared__ double tile[32][33];
    int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        int r = bx + threadIdx.x, c = by + y;
        if (r < rows && c < cols) tile[y][threadIdx.x] = src[r + (long long)c * lds];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        int r = by + threadIdx.x, c = bx + y;   // dst is cols x rows
        if (r < cols && c < rows) dst[r + (long long)c * ldd] = tile[threadIdx.x][y];
    }
}

int scale_device(double *Y, int rows, int cols, int ldy, double beta, cudaStream_t st)
{
    if (rows <= 0 || cols <= 0 || beta == 1.0) return 0;
    long long n = (long long)rows * cols;
    int grid = (int)std::min<long long>((n + 255) / 256, 152LL * 16);
    scale_kernel<<<grid, 256, 0, st>>>(Y, rows, cols, ldy, beta);
    note_launch();
    DG_CUDA(cudaGetLastError());
    return 0;
}

// dst (cols x rows, ld ldd) := src^T (src rows x cols, ld lds)
int transpose_device(const double *src, int rows, int cols, int lds, double *dst, int ldd,
                     cudaStream_t st)
{
    if (rows <= 0 || cols <= 0) return 0;
    dim3 grid((rows + 31) / 32, (cols + 31) / 32), block(32, 8);
    transpose_kernel<<<grid, block, 0, st>>>(src, rows, cols, lds, dst, ldd);
    note_launch();
    DG_CUDA(cudaGetLastError());
    return 0;
}

// Right-hand sides per CTA: as few equal tiles as kColTile (or the autotuned
// cap) allows, so that 17 right-hand sides are tiles of 9 and 8.
int col_tile(int nrhs, int cap)
{
    const int most = std::min(kColTile, std::max(cap, 1)), nt = (nrhs + most - 1) / most;
    return (nrhs + nt - 1) / nt;
}

int run_panel(const Schedule &S, const double *fbase, const double *X, int ldx, int nrhs,
              double *partials, cudaStream_t st, SchedPart part)
{
    const int i0 = part.begin, count = (part.end < 0 ? (int)S.items.size() : part.end) - i0;
    if (count <= 0 || nrhs <= 0) return 0;
    const int nb = col_tile(nrhs, S.nb_cap);
    dim3 g((unsigned)count, (unsigned)((nrhs + nb - 1) / nb));
    double fl = 0, by = 0;
    for (int i = i0; i < i0 + count && prof_on(); ++i) {
        const PanelItem &it = S.items[i];
        fl += 2.0 * it.len * it.rank * nrhs;
        by += 8.0 * ((double)it.len * it.rank + (double)it.len * nrhs + (double)it.rank * nrhs);
    }
    ProfScope ps("panel", st, fl, by);
    if (nrhs == 1 && S.max_len <= kPanel1MaxLen) {
        panel1_kernel<<<(unsigned)count, kThreads, 0, st>>>(S.d_items + i0, fbase, X, partials);
        note_launch();
        DG_CUDA(cudaGetLastError());
        return 0;
    }
    panel_kernel<<<g, kThreads, 0, st>>>(S.d_items + i0, fbase, X, ldx, nrhs, nb, partials);
    note_launch();
    DG_CUDA(cudaGetLastError());
    return 0;
}

int run_reduce(const Schedule &S, const double *sigbase, const double *partials, int nrhs,
               double *T, cudaStream_t st, SchedPart part)
{
    const int i0 = part.begin, count = (part.end < 0 ? (int)S.reduces.size() : part.end) - i0;
    if (count <= 0 || nrhs <= 0 || S.max_rank <= 0) return 0;
    double fl = 0, by = 0;
    for (int i = i0; i < i0 + count && prof_on(); ++i) {
        const ReduceItem &r = S.reduces[i];
        fl += (double)r.nch * r.rank * nrhs;
        by += 8.0 * (r.nch + 1.0) * r.rank * nrhs;
    }
    ProfScope ps("reduce", st, fl, by);
    const long long cnt = (long long)S.max_rank * nrhs;
    const int from = nrhs < 8 ? 0 : (cnt + 31) / 32 <= kGridY ? kGroupedChunks : INT_MAX;
    const int per = S.max_nch >= from ? 32 : 256;
    const dim3 g((unsigned)count, (unsigned)((cnt + per - 1) / per));
    return launch_chained(reduce_kernel, g, 256, 0, st, true, S.d_reduces + i0, sigbase, partials, nrhs, from, T);
}

int run_expand(const Schedule &S, const double *abase, const double *T, const double *X, int ldx,
               double *Y, int ldy, int nrhs, double alpha, double beta, cudaStream_t st, bool chained)
{
    const int ntiles = (int)S.tiles.size();
    if (ntiles == 0 || nrhs <= 0) return 0;
    const int nb = col_tile(nrhs, S.nb_cap);
    dim3 g(ntiles, (unsigned)((nrhs + nb - 1) / nb));
    double fl = 0, by = 0;
    for (int i = 0; i < ntiles && prof_on(); ++i) {
        const double h = S.tiles[i].y;
        by += 8.0 * h * nrhs * (beta == 0.0 ? 1.0 : 2.0);
        for (int q = S.tile_begin[i]; q < S.tile_begin[i + 1]; ++q) {
            const TileTerm &t = S.terms[q];
            fl += 2.0 * h * t.K * nrhs;
            by += 8.0 * (h * t.K + (double)t.K * nrhs);
        }
    }
    ProfScope ps("expand", st, fl, by);
    if (nrhs == 1)
        return launch_chained(!S.has_row_major ? expand1_kernel<kNoRows>
                              : S.short_rows ? expand1_kernel<kShortRows> : expand1_kernel<kDotRows>, g, kThreads, 0, st,
                              chained && ntiles >= kChainTiles, abase, S.d_terms, S.d_tiles, S.d_tile_begin, T, X, Y,
                              alpha, beta);
    note_launch();
    expand_kernel<<<g, kThreads, 0, st>>>(abase, S.d_terms, S.d_tiles, S.d_tile_begin, T, X, ldx, Y, ldy, nrhs, nb,
                                          alpha, beta);
    DG_CUDA(cudaGetLastError());
    return 0;
}

int run_cap_list(const std::vector<CapItem> &caps, const CapItem *d_caps, const double *kbase, const double *sigbase,
                 int trans, const double *T, double *W, int nrhs, cudaStream_t st)
{
    if (caps.empty() || nrhs <= 0) return 0;
    const int scaled = sigbase != nullptr;
    int rmax = 0;
    double fl = 0, by = 0;
    for (const CapItem &c : caps) {
        const double r = c.r1 + c.r2;
        rmax = std::max(rmax, c.r1 + c.r2);
        fl += 2.0 * r * r * nrhs;
        by += 8.0 * (r * r + 2.0 * r * nrhs);
    }
    const int nb = col_tile(nrhs, kColTile);
    ProfScope ps("capacitance", st, fl, by);
    note_launch();
    dim3 g((unsigned)caps.size(), (unsigned)((nrhs + nb - 1) / nb), (unsigned)((rmax + 63) / 64));
    cap_kernel<<<g, kThreads, 0, st>>>(d_caps, kbase, sigbase, trans, scaled, T, W, nrhs, nb);
    DG_CUDA(cudaGetLastError());
    return 0;
}

int run_caps(const Schedule &S, const double *kbase, const double *sigbase, int trans, const double *T, double *W,
             int nrhs, cudaStream_t st)
{
    return run_cap_list(S.caps, S.d_caps, kbase, sigbase, trans, T, W, nrhs, st);
}

int apply_device(Plan *p, int trans, int nrhs, double alpha, const double *X, int ldx,
                 double beta, double *Y, int ldy, cudaStream_t st, bool alpha0_squares_beta)
{
    if (nrhs <= 0 || p->m == 0) return 0;
    if (alpha == 0.0) {
        // Quick path of DPLR: y := beta*y (beta^2 for the vector apply, whose
        // alpha == 0 branch scales twice, src/dplrpmv.c:140-160).
        int rc = scale_device(Y, p->m, nrhs, ldy, beta, st);
        if (!rc && alpha0_squares_beta && beta != 0.0) rc = scale_device(Y, p->m, nrhs, ldy, beta, st);
        return rc;
    }
    if (pairs_usable(p, trans, nrhs)) return pairs_apply(p, alpha, X, beta, Y, st);
    // Three launches; one persistent launch where the autotuner timed it faster
    // (DPLR_GB300_APPLY=launches or =persistent asks for either).  The persistent
    // launch took, of the three launches' time (N = 32768 to 524288, leaves of 128
    // and 256, ranks 8 to 64, and the 2D Gaussian kernel with N = 2^18, ranks up to
    // 128; panels of 512 rows): one column 0.93 to 1.16 under op N (0.97 on the 2D
    // kernel, 1219 / 1251 us) and 1.2 to 1.56 under op T, 2 to 4 columns 1.03 to
    // 1.38, 16 and more 0.98 to 1.08; on small matrices and batches 1.0 to 3: its
    // tiles wait for the slowest panel.  No line in N or rank separates the few
    // shapes that it wins.
    const char *mode = getenv("DPLR_GB300_APPLY");
    const bool launches = mode ? !strcmp(mode, "launches") : p->apply_launches != 0;
    if (!launches)
        return persist_apply(p, trans, nrhs, alpha, X, ldx, beta, Y, ldy, st);
    const Schedule &S = p->sched[trans ? 1 : 0];
    // columns in passes that the grids' limits in y allow (one, but for products
    // like rank 64 with more than 262140 right-hand sides)
    const int pass = std::min(std::min(kGridY * std::min(kColTile, std::max(S.nb_cap, 1)),
                                       kGridY * 256 / std::max(S.max_rank, 1)), nrhs);
    size_t need = (size_t)(S.t_per_rhs + S.partial_per_rhs) * pass;
    int rc = ensure_buffer(&p->work, &p->work_doubles, need);
    if (rc) return rc;
    for (int j = 0; j < nrhs; j += pass) {
        const int k = std::min(pass, nrhs - j);
        const double *Xj = X + (long long)j * ldx;
        double *T = p->work, *partials = p->work + (size_t)S.t_per_rhs * k;
        if ((rc = run_panel(S, p->pool, Xj, ldx, k, partials, st))) return rc;
        if ((rc = run_reduce(S, p->pool, partials, k, T, st))) return rc;
        if ((rc = run_expand(S, p->pool, T, Xj, ldx, Y + (long long)j * ldy, ldy, k, alpha, beta, st,
                             !S.reduces.empty())))
            return rc;
    }
    return 0;
}

}  // namespace dg
