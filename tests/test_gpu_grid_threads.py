"""Queries of one built grid from several host threads at once: every thread's lists are those
of the same queries made alone, whatever the others ask for in the meantime."""
import threading

import numpy as np
import pytest

import sphx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [2, 8])
def test_concurrent_queries_of_one_grid(built, threads):
    rng = np.random.default_rng(threads)
    pos = rng.random((40_000, 3)).astype(np.float32)
    g = sphx.Grid(len(pos))
    g.build(pos, 0.04)
    # sizes that differ from thread to thread and from call to call, so that the workspace
    # grows in one call while another runs
    jobs = []
    for t in range(threads):
        calls = []
        for k in range(6):
            q = rng.random((int(rng.integers(1, 4000)), 3)).astype(np.float32)
            calls.append((q, float(np.float32(rng.choice([0.01, 0.03, 0.06])) ** 2)))
        jobs.append(calls)
    want = [[g.query(q, r2) for q, r2 in calls] for calls in jobs]
    assert max(len(idx) for calls in want for _, idx in calls) > 50_000
    wrong, errors = [], []
    start = threading.Barrier(threads)

    def work(t):
        try:
            start.wait(timeout=60)
            for _ in range(4):
                for k, (q, r2) in enumerate(jobs[t]):
                    counts, idx = g.query(q, r2)
                    if not (np.array_equal(counts, want[t][k][0])
                            and np.array_equal(idx, want[t][k][1])):
                        wrong.append((t, k))
        except Exception as e:  # reported by the test's own thread
            errors.append((t, e))

    pool = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for p in pool:
        p.start()
    for p in pool:
        p.join()
    g.close()
    assert not errors and not wrong
