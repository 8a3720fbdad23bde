"""Search radii far beyond the support: pairs so far apart that their squared distance leaves the
range of the packed square root are neighbours without weight, as in the reference."""
import numpy as np
import pytest

import sph_oracle as O
import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2])
@pytest.mark.parametrize("log2_r", [42, 43, 44, 46, 62])
@pytest.mark.parametrize("tile", [0, 32])
def test_far_pairs_have_no_weight(built, port, kernel, log2_r, tile):
    rng = np.random.default_rng(log2_r)
    r = 2.0 ** log2_r
    # clumps within the support, apart by up to the search radius
    centre = 0.5 * r * rng.integers(0, 3, (12, 1, 3))
    pos = (centre + rng.random((12, 4, 3)) * (centre == 0)).astype(np.float32).reshape(-1, 3)
    vel = rng.standard_normal(pos.shape).astype(np.float32)
    mass = np.full(len(pos), 500.0, np.float32)
    prm = I.params16(smoothing_length=1.0, neighbor_search_radius=r, xmin=-r, ymin=-r, zmin=-r,
                     xmax=2 * r, ymax=2 * r, zmax=2 * r)
    ctx = sphx.Context(len(pos), tile_particles=tile)
    ctx.set_params(prm)
    ctx.set_kernel(kernel)
    ctx.upload(pos, vel, mass)
    ctx.eval()
    out = ctx.download()
    ctx.close()
    for got, want, key in zip((out["rho"], out["pressure"], out["acc"]),
                              port.fields(pos, vel, mass, prm, kernel=kernel), ("rho", "P", "acc")):
        assert O.bits_equal(got, want), O.mismatch_report(got, want, key)
