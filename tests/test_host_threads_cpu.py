"""Host threads behind the C entry points (dplr_gb300/csrc/hostthreads.h): all the
work is done, and no exception leaves, whether the system gives every thread, some
or none.  A host program with a pthread_create of its own is run on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dplr_gb300", "csrc")

PROGRAM = r"""
#include "hostthreads.h"
#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <pthread.h>
static int allowed = 1 << 30;
typedef int (*create_t)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x)
{
    if (allowed-- <= 0) return EAGAIN;
    return ((create_t)dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, x);
}
int main()
{
    for (int give : {100, 7, 3, 1, 0})
        for (unsigned count : {0u, 1u, 2u, 8u, 16u}) {
            allowed = give;
            std::atomic<int> next{0}, done{0};
            auto work = [&]() {
                while (next.fetch_add(1) < 1000) done.fetch_add(1);
            };
            dg::run_on_threads(count, work);
            if (done.load() != 1000) { printf("%d of 1000\n", done.load()); return 1; }
        }
    printf("ok\n");
    return 0;
}
"""


def test_all_work_is_done_with_any_number_of_threads(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src = tmp_path / "threads.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "threads"
    build = subprocess.run([gxx, "-std=c++17", "-O1", "-D_GNU_SOURCE", f"-I{CSRC}", str(src), "-o", str(exe), "-rdynamic",
                            "-lpthread", "-ldl"], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.startswith("ok"), (run.returncode, run.stdout, run.stderr)
