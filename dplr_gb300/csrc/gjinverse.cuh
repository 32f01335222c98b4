// gjinverse.cuh -- batched explicit inverses of small dense matrices (leaves
// and capacitance matrices), orders 1 to 1024, in place.
//
// DPLR's dplrdinv (src/dplrinv.c:20-84) calls LAPACK dgetrf + dgetri.  Here
// the same inverse is formed by blocked Gauss-Jordan elimination with
// partial pivoting: the pivots are those of dgetrf, the work is the same n^3
// multiply-adds, but every panel of 16 columns is followed by ONE update of
// all the other columns,
//     A_O <- A_O (pivot rows: 0) + P (n x 16) W (16 x w),   W = the pivot rows of A_O,
// where P = [A_PP^-1; -A_RP A_PP^-1] is the panel after its own elimination,
// instead of dgetrf's shrinking updates and dgetri's two triangular passes.
// A numpy mirror on random, graded, exponential- and Gaussian-kernel, row- and
// column-scaled matrices with condition numbers up to 3e11 gave errors of
// 0.1 to 2.2 times LAPACK's (0.25 to 0.5 on kernel leaves); panels of 32 lost
// up to 6x in the right residual, which is why the panel is 16.
//
// One thread-block cluster of C CTAs per matrix.  The matrix stays in global
// memory (L2): FP64 issues 2 multiply-adds per clock and SM, so a rank-16
// update, two accesses per 16 multiply-adds, leaves L2 idle, and shared memory
// need not hold the matrix (it limited the previous kernel to order 160 and one
// CTA per SM).  Column blocks of 16 go round-robin to the CTAs; every CTA
// eliminates the panel itself (n x 16 in registers, one row per thread, one
// barrier per column), which costs 8 n^2 clocks but saves the exchange, so one
// cluster barrier per panel is all that the CTAs share.  The rank-16 update
// runs as independent warp tasks of 32 rows x NC columns.
//
// What bounds it: FP64 issue (1.1 to 1.2 TFLOP/s on a GB300) where there are
// matrices for every SM, the chain of n pivots (search, barrier, division, n x
// 16 multiply-adds on one SM) where there are few.  Measured, us per batch
// (before: LU with dgetri's passes, one CTA per matrix):
//     order x count     now   before        order x count     now   before
//       32 x 512         69      202         160 x 128       1245     2035
//      128 x 1          267     1331         256 x 1         1081    18408
//      128 x 256       1230     2651         256 x 128       4577    19373
//      128 x 512       2219     5305         512 x 32       10153   143149
// 128 x 512 runs at 0.97 TFLOP/s (2 n^3 flops per matrix).
#pragma once

#include "smemlimit.cuh"

#include <algorithm>

namespace dg {

constexpr int kGjPanel = 16;      // columns per panel and per column block
constexpr int kGjMax = 1024;      // largest order

__device__ __forceinline__ void gj_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Position i of the rows after the panel's swaps (j <-> piv[j], j = p ..
// p + nb - 1, in this order) holds the row that was at the returned position.
__device__ __forceinline__ int gj_source(const int *piv, int p, int nb, int i)
{
    for (int k = nb - 1; k >= 0; --k) {
        const int q = piv[p + k];
        if (i == p + k)
            i = q;
        else if (i == q)
            i = p + k;
    }
    return i;
}

// Shared memory of one CTA (doubles): the eliminated panel (16 x n rounded up
// to 32; also the staging of the final column permutation) and the pivot rows
// of the CTA's column blocks.
__host__ __device__ constexpr int gj_smem_doubles(int n, int C)
{
    const int np = (n + 31) & ~31, nblk = (n + kGjPanel - 1) / kGjPanel;
    return kGjPanel * np + kGjPanel * kGjPanel * ((nblk + C - 1) / C);
}

constexpr size_t kGjSmemMost = 200 * 1024;       // bytes: order 1024 on two CTAs takes 192 KB
constexpr size_t kGjSmemHeld = 20 * 1024;        // its static arrays, for 1024 threads

// A = base + off[id], n = size[id]; the values are read from S = sbase +
// soff[id] when soff is given (then A is written only), else from A.  info[id]
// = 0 or the 1-based index of the first zero pivot (A is then unspecified).
// Columns are searched for the largest magnitude, the first of equals; NaN is
// never chosen over a number.
template <int T, int NC>
__global__ void __launch_bounds__(T) gj_inverse_kernel(double *base, const long long *__restrict__ off,
                                                       const int *__restrict__ size, const double *sbase,
                                                       const long long *__restrict__ soff, int *info, int C)
{
    constexpr int NB = kGjPanel, NW = T / 32;
    extern __shared__ __align__(16) double sm[];
    __shared__ __align__(16) double crow[2][NW][NB], jrow[2][NB];
    __shared__ unsigned long long ckey[2][NW];
    __shared__ int cidx[2][NW];
    __shared__ int piv[kGjMax], sig[kGjMax], wsrc[NB], dsrc[NB], ddst[NB];

    const int id = blockIdx.x / C, rank = blockIdx.x % C;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n = size[id], np = (n + 31) & ~31, nblk = (n + NB - 1) / NB, nrb = np / 32;
    double *A = base + off[id];
    const double *S = soff ? sbase + soff[id] : A;
    const bool outofplace = soff != nullptr;
    double *Ps = sm, *Ws = sm + NB * np;
    const int nlb = rank < nblk ? (nblk - rank + C - 1) / C : 0;     // column blocks rank, rank + C, ...
    const int wl = nlb * NB;

    for (int p = 0, pb = 0; p < n; p += NB, ++pb) {
        const int nb = min(NB, n - p);
        const double *src = p == 0 ? S : A;
        // ---- panel elimination, one row per thread, in registers
        double P[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) P[k] = (t < n && k < nb) ? __ldcg(src + t + (long long)(p + k) * n) : 0.0;
        bool singular = false;
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            if (k < nb && !singular) {
                const int j = p + k, buf = k & 1;
                if (warp < nrb) {
                    const double v = fabs(P[k]);
                    const unsigned long long key =
                        (t >= j && t < n && v == v) ? (unsigned long long)__double_as_longlong(v) + 1 : 0ull;
                    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
                    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
                    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
                    const unsigned who = __ballot_sync(0xffffffffu, hi == mh && lo == ml);
                    if (lane == __ffs(who) - 1) {
                        ckey[buf][warp] = key;
                        cidx[buf][warp] = t;
#pragma unroll
                        for (int q = 0; q < NB; ++q) crow[buf][warp][q] = P[q];
                    }
                    if (t == j)
#pragma unroll
                        for (int q = 0; q < NB; ++q) jrow[buf][q] = P[q];
                }
                __syncthreads();
                const unsigned long long key = lane < nrb ? ckey[buf][lane] : 0ull;
                const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
                const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
                const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
                const int w = __ffs(__ballot_sync(0xffffffffu, hi == mh && lo == ml)) - 1;
                const bool none = mh == 0 && ml == 0;            // every candidate is NaN: row j itself
                singular = mh == 0 && ml == 1;                   // the largest magnitude is zero
                const int pi = none ? j : cidx[buf][w];
                const double *row = none ? jrow[buf] : crow[buf][w];
                if (t == 0) piv[j] = pi;
                if (!singular && warp < nrb) {
                    // rows j and pi change places; row j becomes row / pivot, the
                    // others lose their multiple of it (one multiply-add each)
                    const double d = 1.0 / row[k];
                    const bool isj = t == j;
                    if (t == pi && !isj)
#pragma unroll
                        for (int q = 0; q < NB; ++q) P[q] = jrow[buf][q];
                    const double mm = isj ? d : -(P[k] * d);
#pragma unroll
                    for (int q = 0; q < NB; ++q)
                        if (q != k) P[q] = fma(mm, row[q], isj ? 0.0 : P[q]);
                    P[k] = mm;
                }
                if (singular && rank == 0 && t == 0) info[id] = j + 1;
            }
        }
        if (singular) return;                                    // the same decision in every CTA of the cluster
        if (t < np)
#pragma unroll
            for (int k = 0; k < NB; ++k) Ps[k * np + t] = t < n ? P[k] : 0.0;
        __syncthreads();                                         // piv and Ps are complete
        // ---- where the pivot rows come from, and which rows outside the
        // panel receive one of the panel's (always from inside the panel)
        if (t < NB) {
            wsrc[t] = t < nb ? gj_source(piv, p, nb, p + t) : 0;
            int d = t < nb ? piv[p + t] : -1;
            if (d < p + nb) d = -1;
            for (int k = t + 1; k < nb && d >= 0; ++k)
                if (piv[p + k] == d) d = -1;                     // counted once
            ddst[t] = d;
            dsrc[t] = d >= 0 ? gj_source(piv, p, nb, d) : 0;
        }
        __syncthreads();
        for (int e = t; e < wl * NB; e += T) {
            const int kk = e % NB, lc = e / NB, cb = (lc / NB) * C + rank, c = cb * NB + lc % NB;
            Ws[e] = (cb != pb && c < n && kk < nb) ? __ldcg(src + wsrc[kk] + (long long)c * n) : 0.0;
        }
        const bool mapped = p == 0 && outofplace;                // S is not written: read through the swaps
        if (!mapped) {
            __syncthreads();                                     // the pivot rows have been read
            for (int e = t; e < wl * NB; e += T) {
                const int kk = e % NB, lc = e / NB, cb = (lc / NB) * C + rank, c = cb * NB + lc % NB;
                if (ddst[kk] >= 0 && cb != pb && c < n)
                    A[ddst[kk] + (long long)c * n] = __ldcg(A + dsrc[kk] + (long long)c * n);
            }
        }
        __syncthreads();
        // ---- rank-16 update of the CTA's column blocks
        const int ntask = nrb * (wl / NC);
        int have = -1, ri = 0;
        for (int id2 = warp; id2 < ntask; id2 += NW) {
            const int rb = id2 % nrb, lc0 = (id2 / nrb) * NC, cb = (lc0 / NB) * C + rank;
            if (cb == pb) continue;
            const int i = rb * 32 + lane, c0 = cb * NB + lc0 % NB;
            if (rb != have) {
                have = rb;
                ri = mapped ? gj_source(piv, p, nb, i) : i;
#pragma unroll
                for (int k = 0; k < NB; ++k) P[k] = Ps[k * np + i];
            }
            const bool live = i < n && !(i >= p && i < p + nb);
            // the 16 products first, then the element: one rounding at the
            // element's size per panel instead of 16
            double old[NC], acc[NC];
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                old[q] = (live && c0 + q < n) ? __ldcg(src + ri + (long long)(c0 + q) * n) : 0.0;
                acc[q] = P[0] * Ws[(lc0 + q) * NB];
            }
#pragma unroll
            for (int k = 1; k < NB; ++k)
#pragma unroll
                for (int q = 0; q < NC; ++q) acc[q] = fma(P[k], Ws[(lc0 + q) * NB + k], acc[q]);
#pragma unroll
            for (int q = 0; q < NC; ++q)
                if (i < n && c0 + q < n) A[i + (long long)(c0 + q) * n] = old[q] + acc[q];
        }
        // every CTA has read panel p and written its columns; only then may
        // the panel's owner overwrite it (the next steps read these columns in
        // the owner alone)
        if (C > 1)
            gj_cluster_sync();
        else
            __syncthreads();
        if (pb % C == rank)
            for (int e = t; e < n * nb; e += T) A[e % n + (long long)(p + e / n) * n] = Ps[(e / n) * np + e % n];
    }
    // ---- inv(A) = X P: the row swaps become column swaps, last first
    bool moved = false;
    for (int j = t; j < n; j += T) moved = moved || piv[j] != j;
    const int any = __syncthreads_or(moved);                     // also: the last panel is written
    if (any) {
        if (C > 1) gj_cluster_sync();
        for (int c = t; c < n; c += T) {
            int s = c;
            for (int j = 0; j < n; ++j) {
                const int q = piv[j];
                if (s == j)
                    s = q;
                else if (s == q)
                    s = j;
            }
            sig[c] = s;
        }
        for (int r0 = rank * NB; r0 < n; r0 += C * NB) {
            const int nr = min(NB, n - r0);
            __syncthreads();
            for (int e = t; e < n * NB; e += T)
                if (e % NB < nr) Ps[e] = __ldcg(A + r0 + e % NB + (long long)(e / NB) * n);
            __syncthreads();
            for (int e = t; e < n * NB; e += T)
                if (e % NB < nr) A[r0 + e % NB + (long long)(e / NB) * n] = Ps[sig[e / NB] * NB + e % NB];
        }
    }
    if (rank == 0 && t == 0) info[id] = 0;
}

// CTAs per matrix: the cheapest of 1, 2, 4, 8 by clocks of FP64 issue.  A CTA
// issues n^3 / (2 C) clocks of updates and 8 n^2 of panels; an SM that gets
// several CTAs runs them one after the other's issue slots, and a CTA alone
// also waits for its pivots (~300 clocks each) and barriers.
inline int gj_cluster_size(int n, int count, int sms)
{
    const double nn = n;
    const int nblk = (n + kGjPanel - 1) / kGjPanel;
    int best = 1;
    double tbest = 1e300;
    for (int C = 1; C <= 8; C *= 2) {
        if (C > 1 && C > nblk) break;
        if (gj_smem_doubles(n, C) * sizeof(double) > kGjSmemMost) continue;    // order 1024 needs two CTAs
        const double issue = nn * nn * nn / (2 * C) + 8 * nn * nn;
        const double waits = nblk * (16 * 300.0 + (C > 1 ? 2500.0 : 1000.0));
        const double waves = (double)((long long)count * C + sms - 1) / sms;
        const double t = std::max(issue * (double)(long long)waves, issue + waits);
        if (t < 0.97 * tbest) {
            tbest = t;
            best = C;
        }
    }
    return best;
}

template <int T, int NC>
inline cudaError_t gj_launch_t(double *base, const long long *off, const int *size, const double *sbase,
                               const long long *soff, int *info, int count, int nmax, int C, cudaStream_t st)
{
    const size_t smem = (size_t)gj_smem_doubles(nmax, C) * sizeof(double);
    cudaError_t e = allow_smem((const void *)gj_inverse_kernel<T, NC>, smem, kGjSmemMost, kGjSmemHeld);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)count * C);
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = C > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, gj_inverse_kernel<T, NC>, base, off, size, sbase, soff, info, C);
}

// Inverts `count` matrices of orders up to nmax (1 to kGjMax) on st.  The
// block has a thread per row of the largest matrix (at least 128).
inline cudaError_t gj_launch(double *base, const long long *off, const int *size, const double *sbase,
                             const long long *soff, int *info, int count, int nmax, int sms, cudaStream_t st)
{
    const int C = gj_cluster_size(nmax, count, sms);
    if (nmax <= 128) return gj_launch_t<128, 8>(base, off, size, sbase, soff, info, count, nmax, C, st);
    if (nmax <= 256) return gj_launch_t<256, 8>(base, off, size, sbase, soff, info, count, nmax, C, st);
    if (nmax <= 512) return gj_launch_t<512, 8>(base, off, size, sbase, soff, info, count, nmax, C, st);
    return gj_launch_t<1024, 4>(base, off, size, sbase, soff, info, count, nmax, C, st);
}

}  // namespace dg
