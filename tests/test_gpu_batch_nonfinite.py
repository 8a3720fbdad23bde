"""Batched scenes with particles that have no finite position: their fields and their step are
those of their own scene."""
import numpy as np
import pytest

import sph_oracle as O
import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2])
@pytest.mark.parametrize("tile", [0, 9, 32])
def test_scenes_bit_identical(port, kernel, tile):
    rng = np.random.default_rng(tile)
    sets = []
    for k, h in enumerate((0.02, 0.03, 0.025, 0.02)):
        n = 200 + 37 * k
        pos = (0.3 * rng.random((n, 3))).astype(np.float32)
        pos[rng.integers(0, n, 25), rng.integers(0, 3, 25)] = rng.choice(
            np.float32([np.nan, np.inf, -np.inf]), 25)
        prm = I.params16(smoothing_length=h, neighbor_search_radius=2 * h, gas_constant=0.1 * k,
                         gravity=-9.81 + k, damping=0.99 - 0.1 * k)
        sets.append((pos, rng.standard_normal((n, 3)).astype(np.float32),
                     np.full(n, 1e-3 * (k + 1), np.float32), prm))
    start = np.cumsum([0] + [len(s[0]) for s in sets])
    ctx = sphx.Context(int(start[-1]), tile_particles=tile)
    ctx.upload(*(np.concatenate([s[k] for s in sets]) for k in range(3)))
    ctx.set_kernel(kernel)
    ctx.set_scenes(start, [s[3] for s in sets])
    ctx.eval()
    out = ctx.download()
    ctx.step(1e-4)
    after = ctx.download()
    ctx.close()
    for a, e, s in zip(start[:-1], start[1:], sets):
        want = port.fields(*s, kernel=kernel)
        for key, w in zip(("rho", "pressure", "acc"), want):
            assert O.bits_equal(out[key][a:e], w), O.mismatch_report(out[key][a:e], w, key)
        alone = sphx.Context(len(s[0]), tile_particles=tile)
        alone.set_params(s[3])
        alone.set_kernel(kernel)
        alone.upload(*s[:3])
        alone.step(1e-4)
        one = alone.download()
        alone.close()
        for key in ("pos", "vel"):
            assert O.bits_equal(after[key][a:e], one[key]), key
