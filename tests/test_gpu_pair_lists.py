"""The neighbour lists' time on small sets, whose passes take tiles of 8 particles: the lists' own
kernels have a lane per particle and take full tiles."""
import time

import numpy as np
import pytest

import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


def test_lists_of_a_small_set_take_full_tiles(built):
    pos = I.lattice(36, 36, 36, seed=5, origin=(0.1,) * 3)
    sel = np.arange(0, len(pos), 60)
    ctxs = [sphx.Context(len(pos), tile_particles=t) for t in (0, 32)]
    times, lists = ([], []), []
    for ctx in ctxs:
        ctx.set_params(I.params16(gas_constant=2e-3))
        ctx.upload(pos, np.zeros_like(pos), np.full(len(pos), 1e-3, np.float32))
        ctx.eval()  # the passes' choice of tiles
    for _ in range(40):  # in turn
        for ctx, mine in zip(ctxs, times):
            t = time.perf_counter()
            lists.append(ctx.pairs_subset(sel))
            mine.append(time.perf_counter() - t)
    assert all(np.array_equal(a, b) for got in lists for a, b in zip(got, lists[-1]))
    assert min(times[0]) < 1.08 * min(times[1])
    for ctx in ctxs:
        ctx.close()
