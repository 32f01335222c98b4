"""Two host threads on distinct plans, each with its own stream: every solve and
factorisation succeeds and gives the bits it gives alone.  The plans' ranks differ,
so that the same kernels are launched with different amounts of shared memory."""
import threading

import pytest

from dplr_gb300 import gen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_solves_and_factorisations_of_distinct_plans_side_by_side():
    from dplr_gb300.plan import GpuPlan
    jobs = []
    for seed, (leaf, rank) in enumerate([(256, 64), (128, 40)]):
        p = GpuPlan(gen.random_tree(2048, leaf, rank, seed=seed))
        b = torch.randn(16, p.m, dtype=torch.float64, device="cuda",
                        generator=torch.Generator(device="cuda").manual_seed(seed))
        p.factor()
        jobs.append((p, b, p.solve(b), torch.cuda.Stream()))
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(len(jobs))

    def run(p, b, want, st):
        try:
            start.wait()
            with torch.cuda.stream(st):
                for k in range(150):
                    if k % 10 == 0:
                        p.write_pool(p.read_pool(stream=st), stream=st)     # same values: factored anew
                        p.factor(stream=st)
                    x = p.solve(b, stream=st)
                    st.synchronize()
                    assert torch.equal(x, want), k
        except Exception as e:                    # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=run, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for p, *_ in jobs:
        p.close()
