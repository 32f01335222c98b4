"""Passes of the allocation-free apply (dplr_gb300/csrc/noalloc.cuh): whatever
it accepts, every pass's T and partial panels lie inside the static scratch and
every block and column is covered once.  A host-only program over the header is
built with nvcc and run on the CPU (no kernel is launched)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dplr_gb300", "csrc")

PROGRAM = r'''
#include "noalloc.cuh"
#include <cstdio>
using namespace dg;
// count trees of m rows, leaf rows and rank; panels of `chunk` rows
static int check(int count, int m, int leaf, int rank, int chunk, int n, int want_groups)
{
    Plan p;
    Schedule S;
    for (int t = 0; t < count; ++t)
        for (int l = 0, h = m / 2; h >= leaf; ++l, h /= 2)
            for (int b = 0; b < (2 << l); ++b) {
                LRDesc D = {};
                D.n = h;
                D.rank = rank;
                D.level = l;
                p.lr.push_back(D);
                const int nch = (h + chunk - 1) / chunk;
                S.reduces.push_back(ReduceItem{S.partial_per_rhs, S.t_per_rhs, -1, rank, nch});
                for (int c = 0; c < nch; ++c) S.items.push_back(PanelItem{});
                S.partial_per_rhs += (long long)nch * rank;
                S.t_per_rhs += rank;
            }
    const size_t cap = kNoAllocScratchDoubles;
    if (noalloc_per_rhs(&p, S) * n > cap) { printf("not accepted\n"); return 1; }
    const NoAllocPasses P = noalloc_passes(S.reduces, S.t_per_rhs, cap, n);
    if (P.cols < 1 || P.cols > n) { printf("cols %d\n", P.cols); return 1; }
    const long long own = S.t_per_rhs + S.partial_per_rhs;
    if (own * n <= (long long)cap && (P.cols != n || P.groups.size() != 1)) { printf("needless passes\n"); return 1; }
    if (want_groups && (int)P.groups.size() < want_groups) { printf("%zu groups\n", P.groups.size()); return 1; }
    int red = 0, item = 0;
    for (const NoAllocGroup &g : P.groups) {
        if (g.reduces.begin != red || g.items.begin != item || g.reduces.end <= red) { printf("gap\n"); return 1; }
        for (int r = g.reduces.begin; r < g.reduces.end; ++r) {
            const ReduceItem &R = S.reduces[r];
            // first and last double of the block's partials, and of its T
            const long long lo = (S.t_per_rhs - g.p0 + R.p) * P.cols, hi = lo + (long long)R.nch * R.rank * P.cols;
            if (lo < S.t_per_rhs * P.cols || hi > (long long)cap) { printf("out of the scratch: %lld\n", hi); return 1; }
            item += R.nch;
        }
        red = g.reduces.end;
        if (g.items.end != item) { printf("items\n"); return 1; }
    }
    if (red != (int)S.reduces.size() || item != (int)S.items.size()) { printf("not covered\n"); return 1; }
    return 0;
}
int main()
{
    if (check(1, 1024, 64, 32, 64, 1, 0)) return 1;
    if (check(1, 1024, 64, 32, 64, 4300, 2)) return 1;       // one column fits, all do not
    if (check(1, 1024, 512, 512, 64, 4096, 2)) return 1;     // one block's partials take several column passes
    if (check(3000, 1024, 64, 32, 64, 1, 2)) return 1;       // one column does not fit at once
    if (check(4096, 1024, 64, 32, 64, 1, 2)) return 1;
    if (check(32768, 1024, 64, 4, 64, 1, 2)) return 1;
    if (check(900, 4096, 64, 24, 128, 1, 0)) return 1;
    if (check(200, 16384, 256, 30, 256, 2, 0)) return 1;
    if (check(2, 65536, 256, 16, 512, 100, 1)) return 1;
    // a block that does not fit at all is refused
    std::vector<ReduceItem> one(1, ReduceItem{0, 0, -1, 1 << 12, 1 << 12});
    if (noalloc_passes(one, 1 << 12, kNoAllocScratchDoubles, 1).cols != 0) { printf("accepted\n"); return 1; }
    printf("ok\n");
    return 0;
}
'''


def test_every_accepted_call_stays_inside_the_static_scratch(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "passes.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "passes"
    build = subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                            f"-I{CSRC}", str(src), "-o", str(exe)], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.startswith("ok"), run.stdout + run.stderr
