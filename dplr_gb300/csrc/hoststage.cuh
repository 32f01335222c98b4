// hoststage.cuh -- host trees and tables to and from the device.
//
// A host tree is hundreds of arrays of a few KB; a copy call for each cost more
// than the device's work (7 of the 22 ms of an N = 8192 dplrgeinv + product were
// calls that copied 2 MB in all, 14 of the 20 ms of an N = 8192 dplrgeppmm +
// product), and a cudaMalloc and a cudaMemcpy for every table of a plan or a
// factorisation another 4 ms.  GB300's GPU reads and writes the host's pageable
// memory through the host's page tables (NVLink-C2C), so one kernel gathers all
// of a tree's arrays into the factor pool, and one scatters a result into the
// tree's buffers: 190 GB/s in and 155 GB/s out over pieces of 32 KB to 4 MB (64 MB
// in all), where a copy call per 32 KB piece gave 9 GB/s and one host thread
// copying into pinned memory 16.  Pages that nothing has touched are touched by
// host threads first: faulting them in from the GPU ran at 2.7 GB/s.
// Results above 128 MB, and all where the device cannot read pageable memory, go
// through pinned staging and host threads; there each upload is a copy call.
#pragma once

#include "internal.cuh"

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

namespace dg {

// dev[off .. off + n) := host[0 .. n)
struct UploadPiece {
    long long off;
    const double *host;
    size_t n;
};

// Copies the pieces on st and waits for it.
int stage_upload(double *dev, const std::vector<UploadPiece> &pieces, cudaStream_t st);

// dst[0 .. n) := dev[src .. src + n), or NaN for src = kFillNaN.  fresh: newly
// allocated, its old values are nobody's.
constexpr size_t kFillNaN = (size_t)-1;
struct SpreadPiece {
    size_t src;
    double *dst;
    size_t n;
    bool fresh = false;
};

// A result's way from the device into a host tree.  begin() takes the n doubles
// at dev, the work of st, of which the pieces will write `total` doubles (fills
// included): the staging, where there is one, is allocated and filled here, so a
// caller that begins before it reshapes its tree leaves it untouched on an
// error.  finish() waits for st, reports its errors before it writes any value,
// copies the pieces and waits for them.
class ResultSpread {
public:
    int begin(const double *dev, size_t n, size_t total, cudaStream_t st);
    int finish(const std::vector<SpreadPiece> &pieces);

private:
    const double *dev_ = nullptr;
    cudaStream_t st_ = nullptr;
    bool direct_ = false;
    const double *staged_ = nullptr;
    std::unique_lock<std::mutex> lock_;           // of the staging, while its values are read
};

// Arrays of one owner in one device allocation.
class TableBlock {
public:
    template <class T> void add(const std::vector<T> &v, T **dst)
    {
        img_.resize((img_.size() + 255) / 256 * 256);
        fix_.push_back({(void **)dst, img_.size()});
        const char *b = (const char *)v.data();
        if (v.empty())
            img_.resize(img_.size() + sizeof(T));
        else
            img_.insert(img_.end(), b, b + v.size() * sizeof(T));
    }
    // allocates *block, copies the arrays and sets their pointers
    int upload(void **block, long long *bytes)
    {
        const size_t n = std::max<size_t>(img_.size(), 1);
        DG_ALLOC(block, n);
        *bytes += (long long)n;
        if (!img_.empty()) DG_CUDA(cudaMemcpy(*block, img_.data(), img_.size(), cudaMemcpyHostToDevice));
        for (auto &f : fix_) *f.first = (char *)*block + f.second;
        return 0;
    }

private:
    std::vector<char> img_;
    std::vector<std::pair<void **, size_t>> fix_;
};

// A schedule's device arrays (its capacitance items alone with caps_only).
void add_schedule(Schedule &S, TableBlock &tb, bool caps_only = false);

}  // namespace dg
