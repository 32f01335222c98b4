// fp64tile.cuh -- the two FP64 tile products behind the apply, the Woodbury
// sweeps and the persistent apply:
//   panel_tile   P (rank x nj) = F[rows, :]^T X[rows, :]  of one row chunk
//   expand_tile  acc (h x nj) = sum_terms A (h x K) B (K x nj)  of one row tile
// for one column tile of nj <= kColTile right-hand sides.
//
// What bounds them: FP64 issue.  GB300 issues two FP64 multiply-adds per clock
// and SM, so a warp instruction holds its sub-core's pipe for 64 clocks
// whatever its lanes hold; shared-memory reads and index arithmetic are free
// beside it, and what costs is every issued multiply-add that is not needed.
// So the 256 threads are cut by the tile's own sizes, not by powers of two:
//   panel:  rank column x column group x row group, RT = the rank itself (up
//           to 64; larger ranks in equal parts);
//   expand: tile row x column group (x inner group, when there are fewer
//           columns than groups), any height h <= 64;
// a thread takes the columns jg, jg + JG, ... that exist (at most 4), and no
// padding is multiplied.  Sums over row or inner groups meet in shared memory
// in a fixed order.  Slabs are staged with 8-byte cp.async (any alignment) into
// two buffers, one being filled while the other is multiplied, and a slab of the
// expand holds columns of several terms, so terms of small rank cost no barrier
// of their own.
// Measured on a GB300 against power-of-two cuts with single-buffered slabs (the
// two-level sums below included):
//   A^T x, N = 25600, leaf 50, rank 12, 5 RHS      981 -> 125 us
//   A X, N = 65536, leaf 256, rank 32, 64 RHS      5.56 -> 5.44 ms (1.18 TFLOP/s)
//   refactorisation, N = 32768, leaf 256, rank 64  32.7 -> 30.7 ms
//   adjoint step, N = 32768, leaf 128, rank 16     7.78 -> 6.52 ms
//   64 matrices of N = 1024 to 8192, 8 RHS, apply + refined solve  2.75 -> 2.48 ms
#pragma once

namespace dg {

constexpr int kTT = 256;             // threads per CTA
// CTAs per SM of the three launches: what the buffers' shared memory allows (48
// registers, a few bytes spilled outside the loops; 64 registers and 4 CTAs cost
// 6% of the batch's sweeps).  The persistent apply is faster with the 80
// registers it takes and 3 CTAs (125 us against 138 on the 50-row leaves below).
constexpr int kTileCtas = 5;
constexpr int kColTile = 16;         // right-hand sides per CTA
constexpr int kSlabCols = 32;        // inner columns of an expand slab
constexpr int kLdA = 65, kLdB = kColTile + 1;
constexpr int kPanelBuf = 2048;      // doubles of one panel buffer
constexpr int kExpandBuf = kSlabCols * (kLdA + kLdB);
// shared memory of a CTA in doubles: the two buffers, and what a column group
// past the last column may read (and drop) beyond them
constexpr int kTileSmem = 2 * (kPanelBuf > kExpandBuf ? kPanelBuf : kExpandBuf) + 64;

// Column groups of the panel by (rank tile, columns): the number JG for which
// the warps issue the fewest multiply-adds per row (active warps x columns per
// thread / row groups), the largest of equals (fewer row groups to add up).
struct PanelGroups {
    unsigned char jg[64][kColTile];
    constexpr PanelGroups() : jg{}
    {
        for (int rt = 1; rt <= 64; ++rt)
            for (int nj = 1; nj <= kColTile; ++nj) {
                int best = 1, bn = 1 << 20, bd = 1;
                for (int g = 1; g <= nj && rt * g <= kTT; ++g) {
                    const int nq = (nj + g - 1) / g, rg = kTT / (rt * g), w = (rt * g * rg + 31) / 32;
                    if (nq > 4) continue;
                    if (w * nq * bd <= bn * rg) {
                        best = g;
                        bn = w * nq;
                        bd = rg;
                    }
                }
                jg[rt - 1][nj - 1] = (unsigned char)best;
            }
    }
};
static __constant__ PanelGroups kPanelGroups;

__device__ __forceinline__ void cp_async8(double *s, const double *g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g)
                 : "memory");
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N> __device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Chained launches (launch_chained): lets the next kernel start; waits until the
// kernels in front have ended and their writes are visible.  A pointer to what
// they wrote goes through the wait, so that no load through it moves above.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class T> __device__ __forceinline__ T *chain_wait(T *p)
{
    asm volatile("griddepcontrol.wait;" : "+l"(p) : : "memory");
    return p;
}

// acc[q] += sum_c a[c * lda] b[c * ldb + q * jstep], c = c0, c0 + cstep, ... < n;
// q < nq, the same nq in the whole warp (the largest of its threads')
template <int Q>
__device__ __forceinline__ void tile_fma(const double *a, int lda, const double *b, int ldb, int jstep, int c0,
                                         int cstep, int n, double (&acc)[4])
{
#pragma unroll 2
    for (int c = c0; c < n; c += cstep) {
        const double x = a[c * lda];
#pragma unroll
        for (int q = 0; q < Q; ++q) acc[q] = fma(x, b[c * ldb + q * jstep], acc[q]);
    }
}

// Sums of two levels: products go to part, and part to acc once kFlush of them
// have been added, so that a long sum rounds at its own size once per kFlush
// products.  (One level of the same loops gave refined solves a factorisation
// with 1.5 times the error; 64 costs 1.6% more additions, every slab of 16 or
// 32 cost 6% of a 64-column product.)
constexpr int kFlush = 64;

// Row groups of a panel from which several lanes add them up per output: rank 3 and
// 4 columns are 85 groups, which the threads of the first one walked through (256
// trees of 512 rows, leaf 32: 370 us, 183 so; N = 131072, leaf 128, rank 2, 3
// columns 272, 192).  At 16 groups the two are level or the lanes are 3% behind.
constexpr int kManyGroups = 20;

__device__ __forceinline__ void tile_flush(double (&acc)[4], double (&part)[4], bool &first)
{
    if (first) {
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = part[q];
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] += part[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) part[q] = 0.0;
    first = false;
}

__device__ __forceinline__ void tile_fma_n(int nq, const double *a, int lda, const double *b, int ldb, int jstep,
                                           int c0, int cstep, int n, double (&acc)[4])
{
    switch (nq) {
    case 4: tile_fma<4>(a, lda, b, ldb, jstep, c0, cstep, n, acc); break;
    case 3: tile_fma<3>(a, lda, b, ldb, jstep, c0, cstep, n, acc); break;
    case 2: tile_fma<2>(a, lda, b, ldb, jstep, c0, cstep, n, acc); break;
    case 1: tile_fma<1>(a, lda, b, ldb, jstep, c0, cstep, n, acc); break;
    default: break;
    }
}

// P[k + j * rank] = sum_r F[r + k * ldf] X[r + j * ldx], r < len, k < rank,
// j < nj.  sm: kTileSmem doubles; all kTT threads call it, and may use sm again
// when it returns.  rot: any number, different from CTA to CTA: where a shape
// leaves warps idle, it moves them over the SM's four sub-cores.
__device__ __forceinline__ void panel_tile(const double *__restrict__ F, long long ldf, int len, int rank,
                                           const double *__restrict__ X, long long ldx, int nj,
                                           double *__restrict__ P, double *sm, int rot)
{
    const int t = (threadIdx.x + 32 * rot) & (kTT - 1);
    const int parts = (rank + 63) / 64, RT = (rank + parts - 1) / parts;
    const int JG = kPanelGroups.jg[RT - 1][nj - 1];
    const int RG = kTT / (RT * JG);
    const int kk = t % RT, rest = t / RT, jg = rest % JG, rg = rest / JG;
    const int nq = (nj - jg + JG - 1) / JG;
    const int ldF = RT | 1, ldX = nj | 1;
    int lg = 4;                                   // slabs of 16 to 128 rows that fit a buffer
    while (lg < 7 && (ldF + ldX) << (lg + 1) <= kPanelBuf && (1 << lg) < len) ++lg;
    const int S = 1 << lg, ns = (len + S - 1) >> lg;
    for (int kt = 0; kt < rank; kt += RT) {
        const int nk = min(RT, rank - kt);
        auto stage = [&](int s) {
            if (s < ns) {
                double *Fs = sm + (s & 1) * kPanelBuf, *Xs = Fs + S * ldF;
                const int r0 = s << lg, live = min(S, len - r0);
                for (int e = t; e < nk << lg; e += kTT) {
                    const int r = e & (S - 1), c = e >> lg;
                    if (r < live) cp_async8(Fs + r * ldF + c, F + r0 + r + (long long)(kt + c) * ldf);
                }
                for (int e = t; e < nj << lg; e += kTT) {
                    const int r = e & (S - 1), c = e >> lg;
                    if (r < live) cp_async8(Xs + r * ldX + c, X + r0 + r + (long long)c * ldx);
                }
            }
            cp_commit();
        };
        double acc[4] = {0.0, 0.0, 0.0, 0.0}, part[4] = {0.0, 0.0, 0.0, 0.0};
        int held = 0;                             // products in part
        bool first = true;                        // acc is still empty
        const bool active = rg < RG && kk < nk;
        const int nqw = __reduce_max_sync(0xffffffffu, active ? nq : 0);
        stage(0);
        for (int s = 0; s < ns; ++s) {
            stage(s + 1);
            cp_wait<1>();
            __syncthreads();
            const double *Fs = sm + (s & 1) * kPanelBuf, *Xs = Fs + S * ldF;
            tile_fma_n(nqw, Fs + kk, ldF, Xs + jg, ldX, JG, rg, RG, min(S, len - (s << lg)), part);
            if ((held += S) >= kFlush * RG || s == ns - 1) {
                tile_flush(acc, part, first);
                held = 0;
            }
            __syncthreads();
        }
        if (RG == 1) {
            if (active)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < nq) P[kt + kk + (long long)(jg + JG * q) * rank] = acc[q];
        } else {
            if (active)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < nq) sm[q * kTT + t] = acc[q];
            __syncthreads();
            const int cnt = nk * nj;
            if (RG >= kManyGroups && 2 * cnt <= kTT) {
                // few outputs, many groups: adjacent lanes share an output
                int lg = 0;
                while (lg < 5 && cnt << (lg + 1) <= kTT) ++lg;
                const int per = 1 << lg, e = t >> lg, k = e % nk, j = e / nk;
                double v = 0.0;
                if (e < cnt)
                    for (int g = t & (per - 1); g < RG; g += per) v += sm[j / JG * kTT + k + RT * (j % JG + JG * g)];
                for (int o = per >> 1; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (e < cnt && (t & (per - 1)) == 0) P[kt + k + (long long)j * rank] = v;
            } else if (active && rg == 0) {
                // the first row group's threads add up the groups of their outputs
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < nq) {
                        double s = acc[q];
                        for (int g = 1; g < RG; ++g) s += sm[q * kTT + t + g * RT * JG];
                        P[kt + kk + (long long)(jg + JG * q) * rank] = s;
                    }
            }
            __syncthreads();
        }
    }
}

// One term of an expand tile: A (h x K) at a + i + c * lda, or a + i * lda + c
// when row_major; B (K x nj) at b + c + j * ldb.  cg: B was written by other
// CTAs of this launch (read past L1).
struct ExpandTerm {
    const double *a, *b;
    long long lda, ldb;
    int K;
    bool row_major, cg;
};

// out(i, j, sum) for i < h <= 64, j < nj; term(q) gives term q < nterms.
template <class TermF, class OutF>
__device__ __forceinline__ void expand_tile(int h, int nterms, TermF term, int nj, OutF out, double *sm, int rot)
{
    const int t = (threadIdx.x + 32 * rot) & (kTT - 1), G = kTT / h;
    const int i = t % h, rest = t / h;
    const int JG = min(nj, G), KS = G / JG;
    const int jg = rest % JG, ks = rest / JG;
    const int nq = (nj - jg + JG - 1) / JG;
    const int lane = t & 31, warp = t >> 5;
    int q0 = 0, k0 = 0;
    // the next slab's columns into buffer buf; returns how many there are
    auto stage = [&](int buf) {
        double *As = sm + buf * kExpandBuf, *Bs = As + kSlabCols * kLdA;
        int c0 = 0;
        while (q0 < nterms && c0 < kSlabCols) {
            const ExpandTerm tt = term(q0);
            const int nk = min(kSlabCols - c0, tt.K - k0);
            if (!tt.row_major) {
                if (rest < G)
                    for (int c = rest; c < nk; c += G)
                        cp_async8(As + (c0 + c) * kLdA + i, tt.a + i + (long long)(k0 + c) * tt.lda);
            } else if (lane < nk) {
                for (int r = warp; r < h; r += kTT / 32)
                    cp_async8(As + (c0 + lane) * kLdA + r, tt.a + (long long)r * tt.lda + k0 + lane);
            }
            if (lane < nk)
                for (int j = warp; j < nj; j += kTT / 32) {
                    const double *src = tt.b + k0 + lane + j * tt.ldb;
                    double *dst = Bs + (c0 + lane) * kLdB + j;
                    if (tt.cg)
                        *dst = __ldcg(src);
                    else
                        cp_async8(dst, src);
                }
            c0 += nk;
            k0 += nk;
            if (k0 >= tt.K) {
                ++q0;
                k0 = 0;
            }
        }
        cp_commit();
        return c0;
    };
    double acc[4] = {0.0, 0.0, 0.0, 0.0}, part[4] = {0.0, 0.0, 0.0, 0.0};
    int held = 0;
    bool first = true;
    const int nqw = __reduce_max_sync(0xffffffffu, ks < KS ? nq : 0);
    int cols = stage(0);
    for (int buf = 0; cols > 0; buf ^= 1) {
        const int next = stage(buf ^ 1);
        cp_wait<1>();
        __syncthreads();
        const double *As = sm + buf * kExpandBuf, *Bs = As + kSlabCols * kLdA;
        tile_fma_n(nqw, As + i, kLdA, Bs + jg, kLdB, JG, ks, KS, cols, part);
        if ((held += cols) >= kFlush * KS || next == 0) {
            tile_flush(acc, part, first);
            held = 0;
        }
        __syncthreads();
        cols = next;
    }
    if (KS > 1) {
        if (ks > 0 && ks < KS)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < nq) sm[q * kTT + t] = acc[q];
        __syncthreads();
        if (ks == 0)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < nq)
                    for (int s = 1; s < KS; ++s) acc[q] += sm[q * kTT + t + s * JG * h];
    }
    if (ks == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < nq) out(i, jg + JG * q, acc[q]);
    __syncthreads();
}

}  // namespace dg
