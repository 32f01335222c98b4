"""The shared-memory limits that the kernels are given once and for all cover every
size they are launched with, so that no launch sets one of its own.  A host-only
program over the headers is built with nvcc and run on the CPU (no kernel is
launched)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dplr_gb300", "csrc")

PROGRAM = r"""
#include "internal.cuh"
#include "sweep.cuh"
#include "gjinverse.cuh"
#include "svdbatch.cuh"
#include <cstdio>
using namespace dg;
int main()
{
    const size_t sm = 227 * 1024;                 // a CTA's shared memory, static part included
    for (int r = 0; r <= kSweepRank; ++r)
        for (int p = 0; p <= kSweepRank; ++p)
            for (int nb = 1; nb <= kColTile; ++nb) {
                if (sizeof(double) * sweep_smem(r, p, nb, kSweepK, kSweepT) > kSweepSmemMost) return 1;
                if (sizeof(double) * (kTileSmem + 64 * (nb | 1) + 64 * (p | 1)) > kSweepSmemMost) return 2;
            }
    for (int n = 1; n <= kGjMax; ++n)
        for (int count : {1, 3, 19, 152, 1000, 100000}) {
            const int C = gj_cluster_size(n, count, 152);
            if (sizeof(double) * gj_smem_doubles(n, C) > kGjSmemMost) { printf("gj %d x %d\n", n, count); return 3; }
        }
    for (int r = 1; r <= kSvdBatchRank; ++r)
        for (long long n = r; n * r * r <= 1LL << 22; ++n) {
            const int nch = svd_chunks((int)n, r);
            const size_t rows = (size_t)(n + nch - 1) / nch;
            if (sizeof(double) * rows * r > kSvdChunkSmemMost) { printf("chunk %lld %d\n", n, r); return 4; }
            if (sizeof(double) * svd_core_smem(r, nch) > kSvdCoreSmemMost) { printf("core %lld %d\n", n, r); return 5; }
        }
    if (kSweepSmemMost > sm || kGjSmemMost + kGjSmemHeld > sm || kSvdChunkSmemMost + kSvdSmemHeld > sm ||
        kSvdCoreSmemMost + kSvdSmemHeld > sm)
        return 6;
    printf("ok\n");
    return 0;
}
"""


def test_limits_cover_every_launch(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "limits.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "limits"
    build = subprocess.run([nvcc, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-gencode",
                            "arch=compute_103a,code=sm_103a", f"-I{CSRC}", str(src), "-o", str(exe)],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.startswith("ok"), (run.returncode, run.stdout, run.stderr)
