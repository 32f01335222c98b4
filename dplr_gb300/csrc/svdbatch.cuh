// svdbatch.cuh -- truncated SVDs of many small low-rank blocks in three
// launches, with no library call.
//
// A block U diag(sig) V^T (n x n, rank r <= min(n, kSvdBatchRank)) is
// recompressed as the library path does it (QR of U diag(sig) and of V, SVD
// of the r x r core Ru Rv^T, U' = Qu Uc, V' = Qv Vc), with the dense steps
// written here:
//   1. svd_qr_kernel, one CTA per chunk of at most svd_chunk_rows(r) rows of
//      U diag(sig) or of V: Householder QR in shared memory (the LAPACK dgeqrf
//      / dlarfg convention: beta = -sign(alpha) ||x||, v(0) = 1, tau = (beta -
//      alpha) / beta), the chunk's reflectors and its r x r R kept;
//   2. svd_core_kernel, one CTA per block: QR of the stacked R's (the
//      tall-skinny QR of Demmel, Grigori, Hoemmen and Langou, SIAM J. Sci.
//      Comput. 34 (2012)), the core, its one-sided (Hestenes) Jacobi SVD:
//      columns p, q are rotated until |c_p . c_q| <= tol ||c_p|| ||c_q|| for
//      every pair (round-robin order, rp / 2 disjoint pairs per round, at most
//      kSvdSweeps sweeps); the column norms are the singular values, the
//      normalised columns the left singular vectors of the core and the
//      accumulated rotations its right ones (Demmel and Veselic, "Jacobi's
//      method is more accurate than QR", SIAM J. Matrix Anal. Appl. 13
//      (1992)); then the stack's reflectors applied to [Uc; 0] and [Vc; 0];
//   3. svd_apply_kernel, one CTA per chunk: the chunk's reflectors applied to
//      its part of those, written to the destination.
// Every loop is bounded; a core that has not converged after kSvdSweeps
// sweeps is reported (info 1) and the block is left as it was.  (A numpy mirror
// took at most 28 on 210 random, appended, clustered and kernel cores of rank up
// to 64, singular values over up to 14 decades, and 27 with FP64 angles.)
//
// What bounds it: FP64 issue (2 per clock and SM, so a warp instruction holds
// the pipe for 16 clocks however few lanes matter) and the chain of r
// reflectors and of the Jacobi rounds.  So the rows of tall blocks are split
// over CTAs, the next column's norm is taken by the warp that updates it (one
// barrier per reflector), a Jacobi pair takes 8 lanes (four pairs per warp
// instruction), and a rotation's angle comes from FP32: only its sine and
// cosine have to be exact to rounding, the angle sets the convergence alone.
// Measured on a GB300, 510 blocks of an N = 16384 plan (leaf 64, rank 16 -> 8,
// the tallest 8192 rows): 0.38 ms (step 1), 0.76 ms (2), 0.30 ms (3), against
// 11.9 ms for one CTA per block over all steps; the recompression with its
// plans and copies 25.3 -> 4.0 ms (3.6 with the tables in one allocation).
#pragma once

#include "smemlimit.cuh"

namespace dg {

constexpr int kSvdBatchRank = 64;     // largest rank taking the batched path
constexpr int kSvdThreads = 256;
constexpr int kSvdWarps = kSvdThreads / 32;
constexpr int kSvdSweeps = 60;
constexpr int kSvdChunkMax = 1024;    // rows of a chunk: 32 per lane in svd_apply_kernel

// One block.  u (n x r, ld ldu), v (n x r, ld n; null: the identity) and sig
// (null: ones) are read, du and dv (ld n) and dsig written; all on the device.
struct SvdBatchJob {
    const double *u, *v, *sig;
    double *du, *dv, *dsig;
    long long ldu;
    long long off;                    // scratch offset (doubles), svd_scratch(n, r) of them
    int n, r, nch;
    double eps;                       // singular values below it are dropped
};

struct SvdTask {
    int job, side, chunk;             // side 0: U diag(sig), 1: V
};

// Largest chunk: 8192 doubles of shared memory (three CTAs per SM), at least
// 256 rows, so that the stacked R's of the tallest blocks (n r^2 <= 2^22) fit a
// CTA of step 2; 320 for r > 48, for the same reason.  A block of more rows is
// cut evenly, so a chunk never has fewer than r rows.
__host__ __device__ constexpr int svd_chunk_rows(int r)
{
    return r > 48 ? 320 : 8192 / r > kSvdChunkMax ? kSvdChunkMax : 8192 / r > 256 ? 8192 / r : 256;
}

__host__ __device__ constexpr int svd_chunks(int n, int r)
{
    return (n + svd_chunk_rows(r) - 1) / svd_chunk_rows(r);
}

// Scratch of one side (doubles): reflectors, their factors, the stacked R's
// (then the stack's reflectors), the stack's factors, the coefficients.
__host__ __device__ constexpr long long svd_side_scratch(int n, int r, int nch)
{
    return (long long)n * r + (long long)nch * r + 2LL * nch * r * r + r;
}

__host__ __device__ constexpr long long svd_scratch(int n, int r)
{
    return 2 * svd_side_scratch(n, r, svd_chunks(n, r));
}

// Shared memory of a step-2 CTA, in doubles: the stack (or the core and the
// rotations), Ru and Rv.
__host__ __device__ constexpr int svd_core_ld(int r) { return r | 1; }
__host__ __device__ constexpr int svd_core_smem(int r, int nch)
{
    const int x = 2 * r * svd_core_ld(r), s = nch > 1 ? nch * r * r : 0;
    return (s > x ? s : x) + 2 * r * r;
}

// What any block of rank r <= kSvdBatchRank and n r^2 <= 2^22 may need (bytes):
// a chunk of 320 rows of rank 64, the stack of a rank-64 block of 1024 rows.
constexpr size_t kSvdChunkSmemMost = sizeof(double) * 320 * 64, kSvdCoreSmemMost = sizeof(double) * 24576;
constexpr size_t kSvdSmemHeld = 4 * 1024;         // static arrays

__device__ __forceinline__ double svd_warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the CTA, the same value in every thread; red: a double per warp.
// The leading barrier keeps a previous call's readers ahead of its writers.
__device__ __forceinline__ double svd_block_sum(double v, double *red)
{
    v = svd_warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) s += red[w];
    return s;
}

__device__ __forceinline__ int svd_block_max(int v, int *red)
{
    v = __reduce_max_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    int s = red[0];
    for (int w = 1; w < (int)blockDim.x / 32; ++w) s = max(s, red[w]);
    return s;
}

__device__ __forceinline__ int svd_hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }

// 2^k, |k| <= 1000
__device__ __forceinline__ double svd_pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }

// Exponent that brings numbers whose largest high word (magnitude) is mh to
// about 1; 0 for zeros, infinities and NaN.
__device__ __forceinline__ int svd_scale_exp(int mh)
{
    if (mh == 0 || mh >= 0x7ff00000) return 0;
    return max(-1000, min(1000, (mh >> 20) - 1023));
}

struct SvdQrScratch {
    double tau[kSvdBatchRank], scl[kSvdBatchRank], beta[kSvdBatchRank], red[kSvdWarps];
    int redi[kSvdWarps];
};

// Reflector of column j from its entry alpha and the sum of squares ss below
// it (both in every lane); lane 0 writes it.  A column whose remaining norm is
// below 2^-60 of the matrix's is left as it is (tau = 0): its tail is far
// below rounding, and reflecting it would cascade towards underflow when the
// columns repeat (as appended blocks do).
__device__ __forceinline__ void svd_reflector(double alpha, double ss, double neg2, int j, SvdQrScratch &q)
{
    const double nn = fma(alpha, alpha, ss);
    double tau = 0.0, scl = 0.0, beta = alpha;
    if (ss > 0.0 && nn > neg2) {
        beta = -copysign(sqrt(nn), alpha);
        tau = (beta - alpha) / beta;
        scl = 1.0 / (alpha - beta);
    }
    if ((threadIdx.x & 31) == 0) {
        q.tau[j] = tau;
        q.scl[j] = scl;
        q.beta[j] = beta;
    }
}

// Householder QR of S (rows x r, ld rows, rows >= r) in shared memory, entries
// of order 1.  R is left above the diagonal (its diagonal in q.beta), the
// unscaled reflectors below it (times q.scl).  Starts and ends with a barrier.
__device__ void svd_qr_smem(double *S, int rows, int r, SvdQrScratch &q)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    double f = 0.0, first = 0.0;
    for (int c = warp; c < r; c += nw)
        for (int i = lane; i < rows; i += 32) {
            const double x = S[i + c * rows];
            f = fma(x, x, f);
            if (c == 0 && i > 0) first = fma(x, x, first);
        }
    const double neg2 = 0x1p-120 * svd_block_sum(f, q.red);
    if (warp == 0) svd_reflector(S[0], svd_warp_sum(first), neg2, 0, q);
    __syncthreads();
    for (int j = 0; j < r; ++j) {
        const double *a = S + j * rows;
        const double tau = q.tau[j], scl = q.scl[j];
        for (int c = j + 1 + warp; c < r; c += nw) {
            double *ac = S + c * rows;
            if (tau != 0.0) {
                double w = 0.0;
                for (int i = j + 1 + lane; i < rows; i += 32) w = fma(a[i], ac[i], w);
                const double top = ac[j];
                w = tau * fma(scl, svd_warp_sum(w), top);
                const double ws = -w * scl;
                for (int i = j + 1 + lane; i < rows; i += 32) ac[i] = fma(ws, a[i], ac[i]);
                __syncwarp();
                if (lane == 0) ac[j] = top - w;
                __syncwarp();
            }
            if (c == j + 1) {                     // the next reflector, by the warp that has its column
                double ss = 0.0;
                for (int i = c + 1 + lane; i < rows; i += 32) ss = fma(ac[i], ac[i], ss);
                svd_reflector(ac[c], svd_warp_sum(ss), neg2, c, q);
            }
        }
        __syncthreads();
    }
}

// Step 1.
__global__ void __launch_bounds__(kSvdThreads) svd_qr_kernel(const SvdBatchJob *__restrict__ jobs,
                                                            const SvdTask *__restrict__ tasks,
                                                            double *__restrict__ scratch)
{
    extern __shared__ double sm[];
    __shared__ SvdQrScratch q;
    const SvdTask tk = tasks[blockIdx.x];
    const SvdBatchJob jb = jobs[tk.job];
    const int n = jb.n, r = jb.r, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row0 = (int)((long long)tk.chunk * n / jb.nch);
    const int rows = (int)((long long)(tk.chunk + 1) * n / jb.nch) - row0;
    const double *src = tk.side ? jb.v : jb.u;
    const long long ld = tk.side ? n : jb.ldu;
    double *base = scratch + jb.off + tk.side * svd_side_scratch(n, r, jb.nch);
    double *Vg = base + (long long)row0 * r, *tg = base + (long long)n * r + tk.chunk * r,
           *Rg = base + (long long)n * r + (long long)jb.nch * r;
    int mh = 0;
    for (int c = warp; c < r; c += kSvdWarps) {
        const double s = (tk.side == 0 && jb.sig) ? jb.sig[c] : 1.0;
        for (int i = lane; i < rows; i += 32) {
            double x = src ? __ldg(src + row0 + i + c * ld) : (row0 + i == c ? 1.0 : 0.0);
            x *= s;
            mh = max(mh, svd_hi_abs(x));
            sm[i + c * rows] = x;
        }
    }
    const int e = svd_scale_exp(svd_block_max(mh, q.redi));
    if (e != 0) {
        const double s = svd_pow2(-e);
        for (int c = warp; c < r; c += kSvdWarps)
            for (int i = lane; i < rows; i += 32) sm[i + c * rows] *= s;
    }
    svd_qr_smem(sm, rows, r, q);
    const double back = svd_pow2(e);
    for (int c = warp; c < r; c += kSvdWarps) {
        const double s = q.scl[c];
        for (int i = lane; i < rows; i += 32) Vg[i + c * rows] = i > c ? sm[i + c * rows] * s : i == c ? 1.0 : 0.0;
        for (int i = lane; i < r; i += 32)
            Rg[(long long)c * jb.nch * r + tk.chunk * r + i] =
                i < c ? sm[i + c * rows] * back : i == c ? q.beta[c] * back : 0.0;
        if (lane == 0) tg[c] = q.tau[c];
    }
}

// Pair pi of round k of a round-robin over rp (even) columns: element rp-1
// meets k, and k + i meets k - i (mod rp - 1).  Over rp - 1 rounds every
// pair meets once.
__device__ __forceinline__ void svd_pair(int pi, int k, int rp, int &p, int &q)
{
    const int m = rp - 1;
    if (pi == 0) {
        p = k;
        q = m;
    } else {
        p = (k + pi) % m;
        q = (k - pi + m) % m;
    }
}

// The leading 21 bits of a normal double as a float in [1, 2), signed, and its
// exponent; a normal float as a double.  Bit operations: conversions between
// the two types would share the FP64 pipe.
__device__ __forceinline__ float svd_head(double x, int &e)
{
    const int hi = __double2hiint(x);
    e = ((hi >> 20) & 0x7ff) - 1023;
    return __int_as_float((hi & 0x80000000) | 0x3f800000 | ((hi & 0xfffff) << 3));
}

__device__ __forceinline__ double svd_widen(float x)
{
    const int b = __float_as_int(x);
    return __hiloint2double((b & 0x80000000) | ((((b >> 23) & 0xff) + 896) << 20) | ((b & 0x7fffff) >> 3), b << 29);
}

// Cosine and sine of the rotation that makes columns of squared norms a, b and
// inner product g orthogonal: t = sign(z) / (|z| + sqrt(1 + z^2)), z = (b - a)
// / (2 g), in FP32 (a relative error of 1e-6 in the angle leaves 1e-6 of g, so
// the last sweeps converge linearly at that rate); cos = 1 / sqrt(1 + t^2) by
// two Newton steps from the FP32 value (2^-20, 2^-40, then rounding) and sin =
// t cos for that very t, so the rotation is orthogonal to rounding.
__device__ __forceinline__ void svd_rotation(double a, double b, double g, double &cs, double &sn)
{
    const double d = b - a;
    float t = 1.0f;
    if (d != 0.0) {
        int ed, eg;
        const float md = svd_head(d, ed), mg = svd_head(g, eg);
        const int k = max(-126, min(120, ed - eg - 1));
        const float z = (md / mg) * __int_as_float((127 + k) << 23), az = fabsf(z);
        t = az > 1e6f ? 0.5f / az : 1.0f / (az + sqrtf(fmaf(z, z, 1.0f)));
        t = copysignf(t, z);
    }
    const double td = svd_widen(t), y = fma(td, td, 1.0);
    int ey;
    const float my = svd_head(y, ey);
    const double h = 0.5 * y;
    double x = svd_widen(rsqrtf(ey ? 2.0f * my : my));
    x = fma(x, fma(-h * x, x, 0.5), x);
    x = fma(x, fma(-h * x, x, 0.5), x);
    cs = x;
    sn = x * td;
}

// Step 2.  out[2 job] = the new rank, out[2 job + 1] = info.
__global__ void __launch_bounds__(kSvdThreads) svd_core_kernel(const SvdBatchJob *__restrict__ jobs,
                                                              const int *__restrict__ ids,
                                                              double *__restrict__ scratch, int *__restrict__ out)
{
    extern __shared__ double sm[];
    __shared__ SvdQrScratch q;
    __shared__ double sv[kSvdBatchRank], inv[kSvdBatchRank];
    __shared__ int order[kSvdBatchRank];
    const int job = ids[blockIdx.x];
    const SvdBatchJob jb = jobs[job];
    const int n = jb.n, r = jb.r, nch = jb.nch, M = nch * r, T = blockDim.x, nw = T / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, ld = svd_core_ld(r);
    double *X = sm, *Rt[2];
    Rt[1] = sm + svd_core_smem(r, nch) - r * r;
    Rt[0] = Rt[1] - r * r;
    for (int s = 0; s < 2; ++s) {
        double *base = scratch + jb.off + s * svd_side_scratch(n, r, nch) + (long long)n * r + (long long)M;
        double *R = Rt[s];
        if (nch == 1) {
            for (int e = t; e < r * r; e += T) R[e] = base[e];
            continue;
        }
        int mh = 0;
        for (int e = t; e < M * r; e += T) {
            const double x = base[e];
            mh = max(mh, svd_hi_abs(x));
            X[e] = x;
        }
        const int e2 = svd_scale_exp(svd_block_max(mh, q.redi));
        if (e2 != 0) {
            const double sc = svd_pow2(-e2);
            for (int e = t; e < M * r; e += T) X[e] *= sc;
        }
        svd_qr_smem(X, M, r, q);
        const double back = svd_pow2(e2);
        for (int c = warp; c < r; c += nw) {
            const double sc = q.scl[c];
            for (int i = lane; i < M; i += 32)
                base[i + (long long)c * M] = i > c ? X[i + c * M] * sc : i == c ? 1.0 : 0.0;
            for (int i = lane; i < r; i += 32)
                R[i + c * r] = i < c ? X[i + c * M] * back : i == c ? q.beta[c] * back : 0.0;
            if (lane == 0) base[(long long)M * r + c] = q.tau[c];
        }
        __syncthreads();                          // X and q are used again
    }
    __syncthreads();
    // C = Ru Rv^T (both upper triangular)
    double *C = X, *Jm = X + r * ld;
    int mh = 0;
    for (int e = t; e < r * r; e += T) {
        const int i = e % r, k = e / r;
        double s = 0.0;
        for (int l = max(i, k); l < r; ++l) s = fma(Rt[0][i + l * r], Rt[1][k + l * r], s);
        mh = max(mh, svd_hi_abs(s));
        C[i + k * ld] = s;
        Jm[i + k * ld] = i == k ? 1.0 : 0.0;
    }
    const int ec = svd_scale_exp(svd_block_max(mh, q.redi));

    // one-sided Jacobi: C J -> columns orthogonal to tol.  Columns of norm
    // below r u ||C||_F are negligible (singular values at rounding level)
    // and take no rotation: the product C J stays exact, and rotations of
    // rounding noise would only slow the convergence.  C is brought to order
    // 1 by a power of two first, so that no square under- or overflows.
    constexpr double u = 1.1102230246251565e-16;
    const double tol = 4.0 * r * u, tol2 = tol * tol;
    double z2 = 0.0;
    {
        const double sc = svd_pow2(-ec);
        for (int e = t; e < r * r; e += T) {
            const double x = C[e % r + (e / r) * ld] * sc;
            C[e % r + (e / r) * ld] = x;
            z2 = fma(x, x, z2);
        }
    }
    z2 = svd_block_sum(z2, q.red) * ((double)r * u) * ((double)r * u);
    const int rp = r + (r & 1), l8 = t & 7;
    bool converged = false;
    for (int sweep = 0; sweep < kSvdSweeps && !converged; ++sweep) {
        bool any = false;
        for (int k = 0; k < rp - 1; ++k) {
            for (int first = (t >> 5) * 4; first < rp / 2; first += T / 8) {     // uniform in a warp
                const int pi = first + ((t >> 3) & 3);
                int p = r, o = r;
                if (pi < rp / 2) svd_pair(pi, k, rp, p, o);
                const bool valid = p < r && o < r;
                double *cp = C + p * ld, *cq = C + o * ld;
                double a = 0.0, b = 0.0, g = 0.0;
                if (valid)
                    for (int i = l8; i < r; i += 8) {
                        const double x = cp[i], y = cq[i];
                        a = fma(x, x, a);
                        b = fma(y, y, b);
                        g = fma(x, y, g);
                    }
#pragma unroll
                for (int w = 4; w; w >>= 1) {
                    a += __shfl_xor_sync(0xffffffffu, a, w);
                    b += __shfl_xor_sync(0xffffffffu, b, w);
                    g += __shfl_xor_sync(0xffffffffu, g, w);
                }
                if (valid && a > z2 && b > z2 && g * g > tol2 * a * b) {
                    double cs, sn;
                    svd_rotation(a, b, g, cs, sn);
                    double *jp = Jm + p * ld, *jq = Jm + o * ld;
                    for (int i = l8; i < r; i += 8) {
                        const double x = cp[i], y = cq[i], xj = jp[i], yj = jq[i];
                        cp[i] = fma(cs, x, -sn * y);
                        cq[i] = fma(sn, x, cs * y);
                        jp[i] = fma(cs, xj, -sn * yj);
                        jq[i] = fma(sn, xj, cs * yj);
                    }
                    any = true;
                }
                __syncwarp();
            }
            __syncthreads();
        }
        converged = !__syncthreads_or(any);
    }
    if (!converged) {
        if (t == 0) {
            out[2 * job] = r;
            out[2 * job + 1] = 1;
        }
        return;
    }
    // singular values (column norms), largest first (ties by column)
    for (int c = warp; c < r; c += nw) {
        double s = 0.0;
        for (int i = lane; i < r; i += 32) s = fma(C[i + c * ld], C[i + c * ld], s);
        s = svd_warp_sum(s);
        if (lane == 0) sv[c] = sqrt(s);
    }
    __syncthreads();
    // a total order (NaN last), so that the positions are a permutation
    for (int c = t; c < r; c += T) {
        const double kc = isnan(sv[c]) ? -1.0 : sv[c];
        int pos = 0;
        for (int d = 0; d < r; ++d) {
            const double kd = isnan(sv[d]) ? -1.0 : sv[d];
            pos += kd > kc || (kd == kc && d < c);
        }
        order[pos] = c;
    }
    __syncthreads();
    const double back = svd_pow2(ec);
    int rank = 0;
    while (rank < r && !(sv[order[rank]] * back < jb.eps)) ++rank;
    for (int c = t; c < rank; c += T) {
        inv[c] = sv[order[c]] > 0.0 ? 1.0 / sv[order[c]] : 0.0;
        jb.dsig[c] = sv[order[c]] * back;
    }
    __syncthreads();
    for (int e = t; e < r * rank; e += T) {       // the core's vectors, over Ru and Rv
        const int i = e % r, c = e / r;
        Rt[0][e] = C[i + order[c] * ld] * inv[c];
        Rt[1][e] = Jm[i + order[c] * ld];
    }
    __syncthreads();
    for (int s = 0; s < 2; ++s) {
        double *base = scratch + jb.off + s * svd_side_scratch(n, r, nch) + (long long)n * r + (long long)M;
        const double *tau2 = base + (long long)M * r;
        double *coef = base + (long long)M * r + r;
        const double *top = Rt[s];
        if (nch == 1) {
            for (int e = t; e < r * rank; e += T) coef[e] = top[e];
            continue;
        }
        // the stack's reflectors, last first, on [top; 0]: a warp per column
        for (int c = warp; c < rank; c += nw) {
            double *y = X + c * M;
            for (int i = lane; i < M; i += 32) y[i] = i < r ? top[i + c * r] : 0.0;
            __syncwarp();
            for (int j = r - 1; j >= 0; --j) {
                const double tj = tau2[j];
                if (tj == 0.0) continue;
                const double *a = base + (long long)j * M;
                double w = 0.0;
                for (int i = j + lane; i < M; i += 32) w = fma(a[i], y[i], w);
                w = -tj * svd_warp_sum(w);
                for (int i = j + lane; i < M; i += 32) y[i] = fma(w, a[i], y[i]);
                __syncwarp();
            }
            for (int i = lane; i < M; i += 32) coef[i + (long long)c * M] = y[i];
        }
        __syncthreads();                          // X is used again
    }
    if (t == 0) {
        out[2 * job] = rank;
        out[2 * job + 1] = 0;
    }
}

// Columns of the chunk's [coefficients; 0] under its reflectors, a warp per
// column with its rows in registers (lane + 32 k, k < Q).
template <int Q>
__device__ void svd_apply_cols(const double *S, const double *tau, const double *coef, long long ldc, int rows, int r,
                               int rank, double *dst, long long ldd)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = warp; c < rank; c += kSvdWarps) {
        double y[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) y[k] = lane + 32 * k < r ? coef[lane + 32 * k + c * ldc] : 0.0;
        for (int j = r - 1; j >= 0; --j) {
            const double tj = tau[j];
            if (tj == 0.0) continue;
            const double *a = S + j * rows;
            double w = 0.0;
#pragma unroll
            for (int k = 0; k < Q; ++k)
                if (lane + 32 * k < rows) w = fma(a[lane + 32 * k], y[k], w);
            w = -tj * svd_warp_sum(w);
#pragma unroll
            for (int k = 0; k < Q; ++k)
                if (lane + 32 * k < rows) y[k] = fma(w, a[lane + 32 * k], y[k]);
        }
#pragma unroll
        for (int k = 0; k < Q; ++k)
            if (lane + 32 * k < rows) dst[lane + 32 * k + c * ldd] = y[k];
    }
}

// Step 3.  A block whose core did not converge is copied as it was.
__global__ void __launch_bounds__(kSvdThreads) svd_apply_kernel(const SvdBatchJob *__restrict__ jobs,
                                                               const SvdTask *__restrict__ tasks,
                                                               const double *__restrict__ scratch,
                                                               const int *__restrict__ out)
{
    extern __shared__ double sm[];
    __shared__ double tau[kSvdBatchRank];
    const SvdTask tk = tasks[blockIdx.x];
    const SvdBatchJob jb = jobs[tk.job];
    const int n = jb.n, r = jb.r, t = threadIdx.x;
    const int row0 = (int)((long long)tk.chunk * n / jb.nch);
    const int rows = (int)((long long)(tk.chunk + 1) * n / jb.nch) - row0;
    const int rank = out[2 * tk.job];
    double *dst = (tk.side ? jb.dv : jb.du) + row0;
    if (out[2 * tk.job + 1] != 0) {
        const double *src = tk.side ? jb.v : jb.u;
        const long long ld = tk.side ? n : jb.ldu;
        if (!src || src == dst - row0) return;
        for (int c = 0; c < r; ++c)
            for (int i = t; i < rows; i += kSvdThreads) dst[i + (long long)c * n] = src[row0 + i + c * ld];
        if (tk.side == 0 && tk.chunk == 0 && jb.sig)
            for (int c = t; c < r; c += kSvdThreads) jb.dsig[c] = jb.sig[c];
        return;
    }
    if (rank == 0) return;
    const double *base = scratch + jb.off + tk.side * svd_side_scratch(n, r, jb.nch);
    const double *Vg = base + (long long)row0 * r;
    const long long M = (long long)jb.nch * r;
    const double *coef = base + (long long)n * r + M + M * r + r + tk.chunk * r;
    for (int e = t; e < rows * r; e += kSvdThreads) sm[e] = Vg[e];
    for (int c = t; c < r; c += kSvdThreads) tau[c] = base[(long long)n * r + tk.chunk * r + c];
    __syncthreads();
    if (rows <= 64)
        svd_apply_cols<2>(sm, tau, coef, M, rows, r, rank, dst, n);
    else if (rows <= 128)
        svd_apply_cols<4>(sm, tau, coef, M, rows, r, rank, dst, n);
    else if (rows <= 256)
        svd_apply_cols<8>(sm, tau, coef, M, rows, r, rank, dst, n);
    else if (rows <= 512)
        svd_apply_cols<16>(sm, tau, coef, M, rows, r, rank, dst, n);
    else
        svd_apply_cols<32>(sm, tau, coef, M, rows, r, rank, dst, n);
}

}  // namespace dg
