// gemm.cuh -- batched FP64 GEMM of the library's structure operations
// (PLR x PLR product, compression): many small and skinny products per
// launch, described by job tables.
//
//   D = alpha op(A) diag(ks) op(B) + beta C
//
// One CTA of 128 threads computes a 32 x 32 output tile (2 x 4 per thread), K
// staged 16 at a time through registers into two shared-memory buffers, the
// next slab's loads under the multiply-adds of this one.  Skinny products (at
// most 16 tiles, K >= 256) are split along K into slices of >= 128 whose raw
// partial sums a second kernel adds in slice order, so results do not depend on
// scheduling.
//
// What bounds it: FP64 issue, 3.6 multiply-adds per ns and SM.  So a tile is
// small (9 us per 32 of K: the last wave of a launch is short, and a few tiles
// already use the chip) and multiplies only the 16-row and 8-column groups that
// it has.  Measured on a GB300 in dplrgeppmm, N = 8192, leaf 256, rank 32: 32
// leaf products of 256^3 1.07 -> 0.95 ms (1.12 TFLOP/s), the rank products and
// the ancestors' terms into the leaves 1.55 -> 0.90 ms, against 64 x 64 tiles,
// single-buffered, padded to 64, and slices of 512.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

namespace dg {
namespace {

// D = alpha op(A) diag(ks) op(B) + beta C  (C not read when beta == 0; C
// may be D).  op(A) is M x K: a[i + k lda] (ta = 0) or a[k + i lda].
struct GemmJob {
    const double *a, *b, *c, *ks;
    double *d;
    int M, N, K, lda, ldb, ldc, ldd, ta, tb;
    double alpha, beta;
};

// Output tile (i0, j0) of a job over k in [k0, k1); p >= 0: raw partial sums
// to part + p (ld M), summed in slice order by gemm_reduce_kernel (split K
// for long, skinny products).
struct GemmTile {
    int job, i0, j0, k0, k1;
    long long p;
};

struct GemmRed {
    long long p;
    int job, slices;
};

constexpr int kGT = 32;       // output tile edge
constexpr int kGK = 16;       // k step staged in shared memory
constexpr int kGThreads = 128;
constexpr int kGSplit = 128;  // shortest slice of a split K

// acc[r][c] += sum_k A[k][ty + 16 r] B[k][tx + 8 c], k < n
template <int RQ, int CQ>
__device__ __forceinline__ void gemm_slab(const double (*A)[kGT + 1], const double (*B)[kGT + 1], int tx, int ty,
                                          int n, double (&acc)[2][4])
{
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
        double a[RQ], b[CQ];
#pragma unroll
        for (int r = 0; r < RQ; ++r) a[r] = A[k][ty + 16 * r];
#pragma unroll
        for (int c = 0; c < CQ; ++c) b[c] = B[k][tx + 8 * c];
#pragma unroll
        for (int r = 0; r < RQ; ++r)
#pragma unroll
            for (int c = 0; c < CQ; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
    }
}

// The slab product for a tile of mi x nj outputs (the same in the whole CTA).
__device__ __forceinline__ void gemm_slab_n(int mi, int nj, const double (*A)[kGT + 1], const double (*B)[kGT + 1],
                                            int tx, int ty, int n, double (&acc)[2][4])
{
    switch ((mi > 16 ? 4 : 0) + ((nj + 7) >> 3)) {
    case 1: gemm_slab<1, 1>(A, B, tx, ty, n, acc); break;
    case 2: gemm_slab<1, 2>(A, B, tx, ty, n, acc); break;
    case 3: gemm_slab<1, 3>(A, B, tx, ty, n, acc); break;
    case 4: gemm_slab<1, 4>(A, B, tx, ty, n, acc); break;
    case 5: gemm_slab<2, 1>(A, B, tx, ty, n, acc); break;
    case 6: gemm_slab<2, 2>(A, B, tx, ty, n, acc); break;
    case 7: gemm_slab<2, 3>(A, B, tx, ty, n, acc); break;
    default: gemm_slab<2, 4>(A, B, tx, ty, n, acc); break;
    }
}

__global__ void __launch_bounds__(kGThreads, 8) gemm_kernel(const GemmJob *__restrict__ jobs,
                                                            const GemmTile *__restrict__ tiles,
                                                            double *__restrict__ part)
{
    constexpr int E = kGT * kGK / kGThreads;       // elements of an operand's slab per thread
    const GemmTile t = tiles[blockIdx.x];
    const GemmJob J = jobs[t.job];
    __shared__ double As[2][kGK][kGT + 1];
    __shared__ double Bs[2][kGK][kGT + 1];
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    const int mi = min(kGT, J.M - t.i0), nj = min(kGT, J.N - t.j0);
    double acc[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
    // alpha == 0: op(A) op(B) is not read (BLAS semantics, NaN-safe)
    const int kend = J.alpha == 0.0 ? t.k0 : t.k1;
    double va[E], vb[E];
    // a slab of both operands into registers (rows, columns and k past the end: zeros)
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < E; ++q) {
            // consecutive threads walk the contiguous index of the operand
            const int e = threadIdx.x + q * kGThreads;
            const int i = J.ta ? e / kGK : e % kGT, ka = k0 + (J.ta ? e % kGK : e / kGT);
            const int j = J.tb ? e % kGT : e / kGK, kb = k0 + (J.tb ? e / kGT : e % kGK);
            va[q] = vb[q] = 0.0;
            if (i < mi && ka < kend) {
                va[q] = J.ta ? J.a[ka + (long long)(t.i0 + i) * J.lda] : J.a[t.i0 + i + (long long)ka * J.lda];
                if (J.ks) va[q] *= J.ks[ka];
            }
            if (j < nj && kb < kend)
                vb[q] = J.tb ? J.b[t.j0 + j + (long long)kb * J.ldb] : J.b[kb + (long long)(t.j0 + j) * J.ldb];
        }
    };
    if (t.k0 < kend) load(t.k0);
    int buf = 0;
    for (int k0 = t.k0; k0 < kend; k0 += kGK, buf ^= 1) {
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int e = threadIdx.x + q * kGThreads;
            As[buf][J.ta ? e % kGK : e / kGT][J.ta ? e / kGK : e % kGT] = va[q];
            Bs[buf][J.tb ? e / kGT : e % kGK][J.tb ? e % kGT : e / kGK] = vb[q];
        }
        // one barrier per slab: a buffer is written again after the next one's,
        // which every thread reaches when it is done with this one
        __syncthreads();
        if (k0 + kGK < kend) load(k0 + kGK);
        gemm_slab_n(mi, nj, As[buf], Bs[buf], tx, ty, min(kGK, kend - k0), acc);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (ty + 16 * r >= mi || tx + 8 * c >= nj) continue;
            const int i = t.i0 + ty + 16 * r, j = t.j0 + tx + 8 * c;
            if (t.p >= 0) {
                part[t.p + i + (long long)j * J.M] = acc[r][c];
            } else {
                double v = J.alpha * acc[r][c];
                if (J.beta != 0.0) v = fma(J.beta, J.c[i + (long long)j * J.ldc], v);
                J.d[i + (long long)j * J.ldd] = v;
            }
        }
}

// D = alpha * (sum of a split job's slices, in order) + beta C.
__global__ void gemm_reduce_kernel(const GemmJob *__restrict__ jobs, const GemmRed *__restrict__ reds,
                                   const double *__restrict__ part)
{
    const GemmRed R = reds[blockIdx.y];
    const GemmJob J = jobs[R.job];
    const long long mn = (long long)J.M * J.N;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < mn; e += (long long)gridDim.x * blockDim.x) {
        double acc = 0.0;
        for (int q = 0; q < R.slices; ++q) acc += part[R.p + q * mn + e];
        const int i = (int)(e % J.M), j = (int)(e / J.M);
        double v = J.alpha * acc;
        if (J.beta != 0.0) v = fma(J.beta, J.c[i + (long long)j * J.ldc], v);
        J.d[i + (long long)j * J.ldd] = v;
    }
}

// Tiles (and split-K reductions) of a job list; ptot = doubles of partial
// sums needed.
inline void plan_gemm_tiles(const std::vector<GemmJob> &jobs, std::vector<GemmTile> &tiles,
                            std::vector<GemmRed> &reds, long long &ptot)
{
    tiles.clear();
    reds.clear();
    ptot = 0;
    for (int j = 0; j < (int)jobs.size(); ++j) {
        const GemmJob &J = jobs[j];
        const int mt = (J.M + kGT - 1) / kGT, nt = (J.N + kGT - 1) / kGT;
        int slices = 1;
        if (mt * nt <= 16 && J.K >= 2 * kGSplit) slices = std::min(128, J.K / kGSplit);
        const int chunk = ((J.K + slices - 1) / slices + kGK - 1) / kGK * kGK;
        slices = J.K > 0 ? (J.K + chunk - 1) / chunk : 1;
        const long long p = slices > 1 ? ptot : -1;
        for (int q = 0; q < slices; ++q)
            for (int i0 = 0; i0 < J.M; i0 += kGT)
                for (int j0 = 0; j0 < J.N; j0 += kGT)
                    tiles.push_back({j, i0, j0, q * chunk, std::min(J.K, (q + 1) * chunk),
                                     p < 0 ? -1 : p + (long long)q * J.M * J.N});
        if (slices > 1) {
            reds.push_back({p, j, slices});
            ptot += (long long)slices * J.M * J.N;
        }
    }
}

// Launch over uploaded tables (tiles in at most 2^30 per grid).
inline void run_gemm_tables(const GemmJob *dj, const GemmTile *dt, size_t ntiles, const GemmRed *dr, size_t nreds,
                            double *part, cudaStream_t st)
{
    for (size_t b0 = 0; b0 < ntiles; b0 += 1u << 30) {
        const unsigned nb = (unsigned)std::min<size_t>(ntiles - b0, 1u << 30);
        gemm_kernel<<<nb, kGThreads, 0, st>>>(dj, dt + b0, part);
    }
    for (size_t b0 = 0; b0 < nreds; b0 += 65535)                   // a grid's limit in y
        gemm_reduce_kernel<<<dim3(16, (unsigned)std::min<size_t>(nreds - b0, 65535)), 256, 0, st>>>(dj, dr + b0, part);
}

}  // namespace
}  // namespace dg
