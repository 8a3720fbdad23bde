"""The exact passes' forms and limits, bit for bit against the oracle: the packed pair
arithmetic itself (every square root and reciprocal compared with CUDA's), and states that
leave its ranges or stress the candidate ring."""
import subprocess

import numpy as np
import pytest

import sph_oracle as O
import sphx
import sphx_build
import sphx_inputs as I

pytestmark = pytest.mark.gpu


def test_pair_arithmetic_is_correctly_rounded(built, tmp_path):
    src = sphx_build.REPO / "tests" / "cpp" / "pair_math_check.cu"
    exe = tmp_path / "pair_math_check"
    subprocess.run([sphx_build._nvcc(), *sphx_build.NVCC_FLAGS, *sphx_build.ARCH,
                    f"-I{sphx_build.PKG / 'csrc'}", str(src), "-o", str(exe),
                    f"-L{sphx_build.LIB}", "-lsphx", f"-Xlinker=-rpath={sphx_build.LIB}"],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["roots", "0", "reciprocals", "0", "quotients", "0", "products", "0"]


def block(n_side, seed, jitter=5e-4, origin=0.1):
    rng = np.random.default_rng(seed)
    pos = I.lattice(n_side, n_side, n_side, seed=seed, jitter=jitter, origin=(origin,) * 3)
    vel = (0.1 * rng.standard_normal(pos.shape)).astype(np.float32)
    return pos, vel, np.full(len(pos), 1e-3, np.float32), I.params16()


def state(name):
    if name in ("one", "two", "thirty_three"):  # fewer and one more than a warp
        pos, vel, mass, prm = block(4, 3)
        n = {"one": 1, "two": 2, "thirty_three": 33}[name]
        return pos[:n], vel[:n], mass[:n], prm
    if name == "tiny_coordinates":  # the general forms: separations down to the subnormals
        pos, vel, mass, prm = block(12, 4, origin=0.0)
        pos[5] = (1e-20, 0.0, 1e-41)
        pos[6] = (0.0, -1e-30, 0.0)
        pos[7] = (1e-20, 0.0, 1e-41)
        return pos, vel, mass, prm
    if name == "light":  # densities outside the shared reciprocals' range
        pos, vel, mass, prm = block(12, 5)
        return pos, vel, np.full(len(pos), 1e-15, np.float32), prm
    if name == "zero_pressure":  # P_i + P_j = 0 among infinities of neither sign
        pos, vel, mass, prm = block(12, 6)
        return pos, vel, mass, I.params16(gas_constant=0.0)
    if name == "close_pairs":  # |r| around the 1e-6 below which the pressure term is skipped
        pos, vel, mass, prm = block(12, 7)
        pos[1::3] = pos[0::3][: len(pos[1::3])] + np.float32(1e-6) * \
            np.random.default_rng(1).random((len(pos[1::3]), 3)).astype(np.float32)
        return pos, vel, mass, prm
    if name == "wide_radius":  # twice the support: 2,100 neighbours, most of zero weight
        pos, vel, mass, prm = block(24, 8)
        return pos, vel, mass, I.params16(neighbor_search_radius=0.08)
    if name == "ties":  # many pairs at |r| = r_search exactly, on cell faces
        k = np.arange(14, dtype=np.float32) * np.float32(0.0078125)
        pos = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
        vel = (0.1 * np.random.default_rng(2).standard_normal(pos.shape)).astype(np.float32)
        return (pos, vel, np.full(len(pos), 1e-3, np.float32),
                I.params16(smoothing_length=0.015625, neighbor_search_radius=0.03125))
    if name == "sparse_column":  # tiles cut along a column of mostly empty cells
        rng = np.random.default_rng(9)
        pos = np.zeros((700, 3), np.float32)
        pos[:, 2] = np.sort(rng.random(700) * 40).astype(np.float32)
        pos[:, :2] = (0.02 * rng.random((700, 2))).astype(np.float32)
        return pos, np.zeros_like(pos), np.full(700, 1e-3, np.float32), I.params16()
    # a dense clump beside a lattice: lanes of one tile with very different neighbour counts
    pos, vel, mass, prm = block(16, 10)
    pos[:1500] = (0.14 + 0.01 * np.random.default_rng(3).random((1500, 3))).astype(np.float32)
    return pos, vel, mass, prm


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2])
@pytest.mark.parametrize("name", ["one", "two", "thirty_three", "tiny_coordinates", "light",
                                  "zero_pressure", "close_pairs", "wide_radius", "ties",
                                  "sparse_column", "clump"])
def test_fields_bit_identical(port, name, kernel):
    pos, vel, mass, prm = state(name)
    ctx = sphx.Context(len(pos))
    ctx.set_params(prm)
    ctx.set_kernel(kernel)
    ctx.upload(pos, vel, mass)
    ctx.eval()
    out = ctx.download()
    rho, p, acc = port.fields(pos, vel, mass, prm, kernel=kernel)
    for got, want, key in ((out["rho"], rho, "rho"), (out["pressure"], p, "P"),
                           (out["acc"], acc, "acc")):
        assert O.bits_equal(got, want), O.mismatch_report(got, want, key)
    ctx.close()


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_GAUSSIAN])
@pytest.mark.parametrize("name", ["thirty_three", "clump", "crowd"])
@pytest.mark.parametrize("tile", [1, 8, 9, 32])
def test_tile_sizes_bit_identical(built, port, tile, name, kernel):
    """Both forms of the exact passes (four lanes per particle up to tiles of 8, one above), and
    tiles whose neighbours do not fit in what the density pass leaves for the force pass."""
    if name == "crowd":  # everything within reach of everything
        rng = np.random.default_rng(21)
        pos = (0.05 + 0.02 * rng.random((2500, 3))).astype(np.float32)
        vel = (0.1 * rng.standard_normal(pos.shape)).astype(np.float32)
        mass, prm = np.full(len(pos), 1e-3, np.float32), I.params16(gas_constant=2e-3)
    else:
        pos, vel, mass, prm = state(name)
    def fields(t):
        ctx = sphx.Context(len(pos), tile_particles=t)
        ctx.set_params(prm)
        ctx.set_kernel(kernel)
        ctx.upload(pos, vel, mass)
        ctx.eval()
        out = ctx.download()
        ctx.close()
        return out["rho"], out["pressure"], out["acc"]

    # the Gaussian's exp is CUDA's, not the host's: there the two forms are compared
    want = (port.fields(pos, vel, mass, prm, kernel=kernel)
            if kernel != sphx.KERNEL_GAUSSIAN else fields(32))
    for g, w, key in zip(fields(tile), want, ("rho", "P", "acc")):
        assert O.bits_equal(g, w), O.mismatch_report(g, w, key)


@pytest.mark.parametrize("name", ["faces", "wide_stencil", "large_cells", "tiny_radius", "folded"])
def test_grid_query_lists_match_the_reference_walk(port, name):
    """The query's cell culling and ranked writes: every particle's list, in order."""
    rng = np.random.default_rng(11)
    cell, radius = {"faces": (0.03125, 0.03125), "wide_stencil": (0.013, 0.04),
                    "large_cells": (0.1, 0.04), "tiny_radius": (0.04, 1e-6),
                    "folded": (0.04, 0.04)}[name]
    if name == "faces":  # points on cell faces, many pairs at the radius exactly
        k = np.arange(16, dtype=np.float32) * np.float32(0.015625) - np.float32(0.125)
        pos = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
    elif name == "folded":  # clusters far apart: the box has far more cells than the grid
        centre = (2e3 * rng.standard_normal((40, 1, 3))).astype(np.float32)
        pos = (centre + 0.05 * rng.random((40, 60, 3))).astype(np.float32).reshape(-1, 3)
    else:
        pos = I.lattice(16, 16, 16, seed=12)
        pos[7::7] = pos[1::7][: len(pos[7::7])]  # coincident points
    g = sphx.Grid(len(pos))
    g.build(pos, cell)
    r = np.float32(radius)
    counts, idx = g.query(pos, float(r * r))
    want_counts, want_idx = port.query(pos, radius, cell_size=cell)
    assert np.array_equal(counts, want_counts) and np.array_equal(idx, want_idx)
    g.close()


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 16384, 16385, 65536, 65537])
@pytest.mark.parametrize("spread", ["dense", "sparse", "nonfinite"])
def test_grid_build_forms_list_the_reference_neighbours(built, port, n, spread):
    """The one-launch grid build at the edges of its blocks, rounds and range: one to four sort
    passes, cells across block ends, particles without a cell."""
    rng = np.random.default_rng(n)
    side = {"dense": 0.04 * (n / 30) ** (1 / 3), "sparse": 6.0, "nonfinite": 0.5}[spread]
    pos = (side * rng.random((n, 3))).astype(np.float32)
    if spread == "nonfinite":
        pos[::3] = np.nan
    g = sphx.Grid(n)
    g.build(pos, 0.04)
    r = np.float32(0.02)
    counts, idx = g.query(pos, float(r * r))
    want_counts, want_idx = port.query(pos, 0.02, cell_size=0.04)
    assert np.array_equal(counts, want_counts) and np.array_equal(idx, want_idx)
    g.close()
    if spread == "dense":
        mass = np.full(n, 1e-3, np.float32)
        ctx = sphx.Context(n)
        ctx.set_params(I.params16())
        ctx.upload(pos, np.zeros_like(pos), mass)
        ctx.eval()
        rho = ctx.download()["rho"]
        want, _, _ = port.fields(pos, np.zeros_like(pos), mass, I.params16())
        assert O.bits_equal(rho, want), O.mismatch_report(rho, want, "rho")
        ctx.close()


@pytest.mark.parametrize("size", [1e-5, 1e-3, 0.02, 0.4, 6.0])
@pytest.mark.parametrize("image", [(333, 217), (64, 1000)])
def test_render_quad_sizes_match_the_oracle(built, port, size, image):
    """Quads from a fraction of a pixel to several images wide: pixels tried within a slack of
    the quad's box and, where that is not provably enough, all around it."""
    rng = np.random.default_rng(31)
    pos = rng.random((400, 3)).astype(np.float32)
    vel = rng.standard_normal(pos.shape).astype(np.float32)
    ctx = sphx.Context(len(pos))
    ctx.set_params(I.params16())
    ctx.upload(pos, vel, np.full(len(pos), 1e-3, np.float32))
    for view, proj in (sphx.camera_matrices((0.5, 0.4, 2.0), -90.0, 0.0, 45.0, 16 / 9),
                       sphx.camera_matrices((1.8, 1.2, 1.6), -135.0, -25.0, 35.0, 4 / 3)):
        # the second projection is also squeezed: quads a few hundredths as wide as high
        for squeeze in (1.0, 0.03):
            p = np.array(proj, np.float32)
            p.reshape(-1)[0] *= np.float32(squeeze)
            rp = sphx.render_params(view, p, particle_size=size, color_mode=0, width=image[0],
                                    height=image[1])
            got, want = ctx.render_image(rp), port.render_image(rp, pos, vel, None)
            assert np.array_equal(got, want)
    ctx.close()


@pytest.mark.parametrize("n", [1, 127, 32768, 32769])
@pytest.mark.parametrize("fields", ["all", "pos", "rho", "acc"])
def test_download_into_pinned_memory(built, n, fields):
    """Fields stored into pinned memory by one kernel (small sets) equal the staged copies."""
    import torch

    rng = np.random.default_rng(n)
    pos = (0.4 * rng.random((n, 3))).astype(np.float32)
    ctx = sphx.Context(n)
    ctx.set_params(I.params16(gas_constant=2e-3))
    ctx.upload(pos, np.zeros_like(pos), np.full(n, 1e-3, np.float32))
    ctx.step(1e-4)
    names = ("pos", "vel", "rho", "pressure", "acc")
    want = ctx.download()
    out = {k: torch.full((3 * n if k in ("pos", "vel", "acc") else n,), 7.0).pin_memory()
           for k in names}
    ctx.download_ptr(*[out[k].data_ptr() if fields in ("all", k) else 0 for k in names])
    for k in names:
        w = want[k].reshape(-1) if fields in ("all", k) else np.full(out[k].shape[0], 7, np.float32)
        assert O.bits_equal(out[k].numpy(), w), k
    ctx.close()
