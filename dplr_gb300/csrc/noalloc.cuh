// noalloc.cuh -- what the allocation-free apply may ask for, and its passes.
#pragma once

#include "internal.cuh"

#include <algorithm>

namespace dg {

constexpr size_t kNoAllocScratchDoubles = (size_t)8 << 20;   // 64 MiB

// Doubles that a call is counted with per right-hand side: T and the partial
// panels of 512 rows, or of the autotuned length.
inline size_t noalloc_per_rhs(const Plan *p, const Schedule &S)
{
    long long parts = S.partial_per_rhs;
    if (!p->chunk_tuned) {
        parts = 0;
        for (const LRDesc &L : p->lr) parts += (long long)((L.n + 511) / 512) * L.rank;
    }
    return (size_t)(S.t_per_rhs + parts);
}

// Blocks whose panels and reduces run together.
struct NoAllocGroup {
    SchedPart items, reduces;
    long long p0;                 // partial offset / nrhs of the first block
};

struct NoAllocPasses {
    int cols = 0;                 // right-hand sides of a pass; 0: a block does not fit
    std::vector<NoAllocGroup> groups;
};

// The passes of n right-hand sides through `cap` doubles: T of `cols` of them
// stays, and the partials of one group of blocks after another share the rest.
// The plan's own panels may be shorter than the 512 rows that a call is counted
// with (64 in trees of up to 1024 rows), so the partials of all blocks together
// can exceed what was counted, for a single right-hand side too: 2800 trees of
// N = 1024, leaf 64, rank 32 are counted with 5.4 M doubles and have 8.4 M.  A
// group is at least one block, and T and one block's partials always fit for
// some number of columns: T is at most half of what was counted.
inline NoAllocPasses noalloc_passes(const std::vector<ReduceItem> &reds, long long t_per_rhs, size_t cap, int n)
{
    NoAllocPasses out;
    long long most = 0, all = t_per_rhs;
    for (const ReduceItem &r : reds) {
        const long long need = (long long)r.nch * r.rank;
        most = std::max(most, need);
        all += need;
    }
    const long long c = (long long)cap;
    if (t_per_rhs + most > c) return out;
    out.cols = all * n <= c ? n : (int)std::min<long long>(n, c / std::max<long long>(t_per_rhs + most, 1));
    const long long room = c / out.cols - t_per_rhs;          // partials per right-hand side
    int item = 0;
    for (int r = 0; r < (int)reds.size();) {
        NoAllocGroup g;
        g.items.begin = item;
        g.reduces.begin = r;
        g.p0 = reds[r].p;
        for (; r < (int)reds.size() && reds[r].p + (long long)reds[r].nch * reds[r].rank - g.p0 <= room; ++r)
            item += reds[r].nch;
        g.items.end = item;
        g.reduces.end = r;
        out.groups.push_back(g);
    }
    return out;
}

}  // namespace dg
