"""Small sets in a box of very many cells: the lists are the reference's whatever the lengths of
the runs of empty cells, and the runs are not written one cell after another."""
import time

import numpy as np
import pytest

import sphx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [60, 1023, 20_000])
@pytest.mark.parametrize("axis", [0, 2])
def test_runs_of_every_length_keep_the_lists(built, port, n, axis):
    rng = np.random.default_rng(n + axis)
    # empty cells before the next particle: around the lengths where the writer changes, and
    # every alignment of the runs' ends
    lengths = np.array([0, 0, 0, 1, 2, 3, 6, 7, 8, 9, 10, 11, 12, 31, 33, 127, 130])
    gaps = rng.choice(lengths, n)
    long_at = rng.choice(n - 1, 12, replace=False) + 1
    gaps[long_at] = [65534, 65535, 65536, 65537, 65538, 65539, 66000, 131071, 200001, 300000, 70003,
                     90001]
    z = np.cumsum(gaps) + 0.5  # a cell of size 1 each
    assert z[-1] < 1 << 22  # exact in float, and far fewer cells than the grid holds
    pos = np.full((n, 3), 0.5, np.float32)
    pos[:, axis] = z
    pos[:, 1] += rng.random(n).astype(np.float32) * 3  # columns of a few cells beside it
    pos = pos[rng.permutation(n)]
    q = pos[rng.integers(0, n, 300)]
    q[:, axis] += rng.integers(-40, 40, len(q))  # in the empty cells, too
    g = sphx.Grid(n)
    g.build(pos, 1.0)
    for radius in (0.9, 2.0):
        r2 = np.float32(radius) * np.float32(radius)
        counts, idx = g.query(pos, float(r2))
        want_counts, want_idx = port.query(pos, radius, cell_size=1.0)
        assert np.array_equal(counts, want_counts) and np.array_equal(idx, want_idx)
        counts, idx = g.query(q, float(r2))
        for p, mine in zip(q, np.split(idx, np.cumsum(counts)[:-1])):
            d = p - pos
            near = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2] <= r2
            assert np.array_equal(np.sort(mine), np.flatnonzero(near))
    g.close()


def test_a_long_run_takes_no_long_time(built):
    """Two clumps at the ends of a box of 15 million cells: 0.15 ms where one thread that writes
    the cells between them takes 69."""
    pos = (0.3 * np.random.default_rng(5).random((4000, 3))).astype(np.float32)
    pos[2000:] += np.float32(9.6)
    g = sphx.Grid(len(pos))
    g.build(pos, 0.04)
    times = []
    for _ in range(5):
        t = time.perf_counter()
        g.build(pos, 0.04)
        times.append(time.perf_counter() - t)
    g.close()
    assert min(times) < 0.02
