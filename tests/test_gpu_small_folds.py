"""Grids folded to very few cells per axis: on five cells a stencil covers the whole axis, and is
still walked in the reference's order."""
import numpy as np
import pytest

import sph_oracle as O
import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2])
@pytest.mark.parametrize("cells", [125, 200, 216, 343])
@pytest.mark.parametrize("tile", [0, 32])
@pytest.mark.parametrize("layout", ["faces", "clumps"])
def test_fields_bit_identical(port, layout, tile, cells, kernel):
    rng = np.random.default_rng(cells + tile)
    if layout == "faces":  # many particles within rounding of a cell face: two layers on each side
        k = np.arange(12, dtype=np.float32) * np.float32(0.015625)
        pos = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
        pos = np.concatenate([pos, pos + np.float32(40.0)])
        prm = I.params16(smoothing_length=0.015625, neighbor_search_radius=0.03125)
    else:
        centre = 300 * rng.standard_normal((20, 1, 3))
        pos = (centre + 0.03 * rng.standard_normal((20, 150, 3))).astype(np.float32).reshape(-1, 3)
        prm = I.params16(gas_constant=2e-3, neighbor_search_radius=0.05)
    pos = pos[rng.permutation(len(pos))]
    vel = (0.1 * rng.standard_normal(pos.shape)).astype(np.float32)
    mass = (1e-3 * (0.5 + rng.random(len(pos)))).astype(np.float32)
    ctx = sphx.Context(len(pos), max_grid_cells=cells, tile_particles=tile)
    ctx.set_params(prm)
    ctx.set_kernel(kernel)
    ctx.upload(pos, vel, mass)
    ctx.eval()
    out = ctx.download()
    counts, idx = ctx.pairs()
    ctx.close()
    want_counts, want_idx = port.query(pos, float(prm[15]))
    assert np.array_equal(counts, want_counts) and np.array_equal(idx, want_idx)
    for got, want, key in zip((out["rho"], out["pressure"], out["acc"]),
                              port.fields(pos, vel, mass, prm, kernel=kernel), ("rho", "P", "acc")):
        assert O.bits_equal(got, want), O.mismatch_report(got, want, key)
