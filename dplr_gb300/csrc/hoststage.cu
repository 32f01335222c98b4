// hoststage.cu -- see hoststage.cuh.
#include "hoststage.cuh"
#include "hostthreads.h"

#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>

namespace dg {

namespace {

constexpr long long kMove = 4096;                   // doubles of one move

struct Move {
    double *dst;
    const double *src;
    long long n;                                    // <= kMove
};

// The list itself is in host memory too: it is read once.
__global__ void __launch_bounds__(256) move_kernel(const Move *__restrict__ moves, int count)
{
    for (int b = blockIdx.x; b < count; b += gridDim.x) {
        const Move m = moves[b];
        const int n = (int)m.n;
        int i = threadIdx.x;
        for (; i + 768 < n; i += 1024) {
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = m.src[i + 256 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k) m.dst[i + 256 * k] = v[k];
        }
        for (; i < n; i += 256) m.dst[i] = m.src[i];
    }
}

void add_moves(std::vector<Move> &v, double *dst, const double *src, size_t n)
{
    for (size_t o = 0; o < n; o += kMove) v.push_back({dst + o, src + o, (long long)std::min<size_t>(kMove, n - o)});
}

int run_moves(const std::vector<Move> &moves, cudaStream_t st)
{
    if (!moves.empty()) {
        const int count = (int)moves.size();
        move_kernel<<<std::min(count, 152 * 8), 256, 0, st>>>(moves.data(), count);
        note_launch();
        DG_CUDA(cudaGetLastError());
    }
    DG_CUDA(cudaStreamSynchronize(st));             // the list and the host arrays are the caller's
    return 0;
}

// Whether the current device reads and writes pageable host memory.
bool reads_pageable()
{
    int dev = 0, v = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
           cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev) == cudaSuccess && v != 0;
}

// Results above this many doubles (128 MB) come back in one copy to pinned
// staging, kept until dplr_gpu_release_staging, and host threads spread it: the
// 817 MB of an N = 16384 product's grown blocks took 190 ms to touch page by page
// for the GPU (the whole product 233 ms, 57 through the staging).
constexpr size_t kDirectMax = (size_t)1 << 24;

struct Staging {
    std::mutex mu;
    double *p = nullptr;
    size_t n = 0;
};

Staging &staging()
{
    static Staging s;
    return s;
}

void release(Staging &s)
{
    if (s.p) cudaFreeHost(s.p);
    s.p = nullptr;
    s.n = 0;
}

}  // namespace

int stage_upload(double *dev, const std::vector<UploadPiece> &pieces, cudaStream_t st)
{
    if (!reads_pageable()) {
        for (const UploadPiece &q : pieces)
            if (q.n)
                DG_CUDA(cudaMemcpyAsync(dev + q.off, q.host, q.n * sizeof(double), cudaMemcpyHostToDevice, st));
        DG_CUDA(cudaStreamSynchronize(st));
        return 0;
    }
    std::vector<Move> moves;
    for (const UploadPiece &q : pieces) add_moves(moves, dev + q.off, q.host, q.n);
    return run_moves(moves, st);
}

int ResultSpread::begin(const double *dev, size_t n, size_t total, cudaStream_t st)
{
    dev_ = dev;
    st_ = st;
    direct_ = total <= kDirectMax && reads_pageable();
    if (direct_ || n == 0) return 0;
    Staging &sg = staging();
    lock_ = std::unique_lock<std::mutex>(sg.mu);
    if (sg.n < n) {
        release(sg);
        const size_t want = n + n / 2;
        if (pinned_malloc((void **)&sg.p, want * sizeof(double)) != cudaSuccess) {
            cudaGetLastError();
            return fail(DPLR_GPU_ENOMEM, "cannot allocate %zu bytes of pinned staging", want * sizeof(double));
        }
        sg.n = want;
    }
    staged_ = sg.p;
    DG_CUDA(cudaMemcpyAsync(sg.p, dev, n * sizeof(double), cudaMemcpyDeviceToHost, st));
    DG_CUDA(cudaStreamSynchronize(st));
    return 0;
}

int ResultSpread::finish(const std::vector<SpreadPiece> &pieces)
{
    // NaN fills and the values out of the staging, or a write to every page that
    // the GPU will write: a zero in fresh ones, elsewhere the word's own value by
    // one read-modify-write.  (A load and a store fault an untouched page in twice,
    // the second time away from the zero page: products of N = 8192, leaf 256, rank
    // 32 into new trees 33 ms, 8.1 so, 7.2 on pages used before.)
    struct Bite {
        double *p;
        size_t n;
        size_t src;
        bool fresh;
    };
    constexpr size_t kBite = (size_t)1 << 17, kPage = 512;    // 1 MB; 4 KB, the smallest page
    std::vector<Bite> bites;
    size_t total = 0;
    for (const SpreadPiece &q : pieces) {
        const bool fill = q.src == kFillNaN;
        for (size_t o = 0; o < q.n; o += kBite)
            bites.push_back({q.dst + o, std::min(kBite, q.n - o), fill ? kFillNaN : q.src + o, q.fresh});
        total += q.n;
    }
    std::atomic<size_t> next{0};
    auto work = [&]() {
        for (size_t i = next.fetch_add(1); i < bites.size(); i = next.fetch_add(1)) {
            const Bite &b = bites[i];
            if (b.src == kFillNaN) {
                std::fill(b.p, b.p + b.n, std::nan(""));
                continue;
            }
            if (!direct_) {
                memcpy(b.p, staged_ + b.src, b.n * sizeof(double));
                continue;
            }
            for (size_t o = 0; o < b.n; o += kPage) {
                if (b.fresh)
                    *(volatile double *)(b.p + o) = 0.0;
                else
                    __atomic_fetch_or((unsigned long long *)(b.p + o), 0ull, __ATOMIC_RELAXED);
            }
        }
    };
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    // a thread per 4 MB at most: below that it costs more to start than it saves
    const unsigned nt = (unsigned)std::min<size_t>(std::min(direct_ ? 8u : 16u, hw), 1 + total / (1 << 19));
    run_on_threads(nt, work);
    if (!direct_) {
        staged_ = nullptr;
        if (lock_.owns_lock()) lock_.unlock();
        return 0;
    }
    DG_CUDA(cudaStreamSynchronize(st_));          // what is in front reports its errors here
    std::vector<Move> moves;
    for (const SpreadPiece &q : pieces)
        if (q.src != kFillNaN) add_moves(moves, q.dst, dev_ + q.src, q.n);
    return run_moves(moves, st_);
}

void add_schedule(Schedule &S, TableBlock &tb, bool caps_only)
{
    S.max_len = 0;
    for (const PanelItem &it : S.items) S.max_len = std::max(S.max_len, it.len);
    S.has_row_major = false;
    S.short_rows = true;
    for (const TileTerm &t : S.terms) {
        S.has_row_major = S.has_row_major || t.trans_a;
        S.short_rows = S.short_rows && (!t.trans_a || t.K <= 64);
    }
    for (const int2 &t : S.tiles) S.short_rows = S.short_rows && t.y <= 32;
    tb.add(S.caps, &S.d_caps);
    if (caps_only) return;
    tb.add(S.items, &S.d_items);
    tb.add(S.reduces, &S.d_reduces);
    tb.add(S.tiles, &S.d_tiles);
    tb.add(S.tile_begin, &S.d_tile_begin);
    tb.add(S.terms, &S.d_terms);
}

}  // namespace dg

extern "C" void dplr_gpu_release_staging(void)
{
    dg::Staging &sg = dg::staging();
    std::lock_guard<std::mutex> lk(sg.mu);
    dg::release(sg);
}
