"""The exact passes with a lane per particle (tiles of more than 8, every set above 65,536
particles), bit for bit against the oracle: states that leave the ranges of the pair forms as a
whole or in a few particles, smoothing lengths of other scales, batches that mix them, and tiles
whose candidates do not fit in what the density pass leaves for the force pass."""
import numpy as np
import pytest

import sph_oracle as O
import sphx
import sphx_inputs as I
from test_gpu_pass_forms import block, state

pytestmark = pytest.mark.gpu

KERNELS = [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2]


def check(port, pos, vel, mass, prm, kernel, capacity=0, tile=32):
    ctx = sphx.Context(max(capacity, len(pos)), tile_particles=tile)
    ctx.set_params(prm)
    ctx.set_kernel(kernel)
    ctx.upload(pos, vel, mass)
    ctx.eval()
    out = ctx.download()
    ctx.close()
    for got, want, key in zip((out["rho"], out["pressure"], out["acc"]),
                              port.fields(pos, vel, mass, prm, kernel=kernel), ("rho", "P", "acc")):
        assert O.bits_equal(got, want), O.mismatch_report(got, want, key)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("name", ["one", "thirty_three", "tiny_coordinates", "light",
                                  "zero_pressure", "close_pairs", "wide_radius", "ties",
                                  "sparse_column", "clump"])
def test_edge_states(port, name, kernel):
    check(port, *state(name), kernel)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("scale", [1e-5, 5e-4, 0.05, 0.1, 1.0, 30.0, 3000.0])
@pytest.mark.parametrize("tile", [0, 32])
def test_smoothing_lengths(port, scale, kernel, tile):
    """The same block at smoothing lengths of 10 um to 3 km, with coincident particles and pairs
    at the edge of the support."""
    pos, vel, _, _ = block(12, 31)
    s = np.float32(scale / 0.02)
    pos[20:40] = pos[60:80]
    pos[100] = pos[101] + np.float32([0.04, 0.0, 0.0])
    pos[102] = pos[103] + np.float32([0.0, 0.0399999, 1e-9])
    prm = I.params16(smoothing_length=scale, neighbor_search_radius=2 * scale)
    check(port, pos * s, vel, np.full(len(pos), 1e-3 * float(s) ** 3, np.float32), prm, kernel,
          tile=tile)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("scale", [5.9e-8, 6.1e-8, 1e-7, 1.04e6, 1.06e6])
@pytest.mark.parametrize("tile", [0, 32])
def test_edges_of_the_smoothing_lengths(port, scale, kernel, tile):
    """Lengths on both sides of the ends of the range of the pair forms."""
    pos, vel, _, _ = block(12, 34)
    s = scale / 0.02
    pos[20:40] = pos[60:80]
    prm = I.params16(smoothing_length=scale, neighbor_search_radius=2 * scale)
    check(port, (pos * s).astype(np.float32), vel, np.full(len(pos), 1e-3 * s ** 3, np.float32), prm,
          kernel, tile=tile)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("h", [0.02, 0.1])
@pytest.mark.parametrize("odd", ["light", "massless", "heavy", "tiny", "far_tiny", "fast", "negative"])
def test_a_few_particles_out_of_range(port, odd, h, kernel):
    """Out-of-range particles among ordinary ones: pairs of each kind in one tile and lane."""
    pos, vel, mass, _ = block(14, 32)
    rng = np.random.default_rng(33)
    pick = rng.permutation(len(pos))[:40]
    prm = I.params16(smoothing_length=h, neighbor_search_radius=2 * h)
    s = np.float32(h / 0.02)
    pos, mass = pos * s, mass * s ** 3
    if odd in ("light", "massless", "heavy", "negative"):
        # alone (their own density) or among others (the others'), by half
        pos[pick[:20]] += np.float32(100 * h) * np.arange(1, 21, dtype=np.float32)[:, None]
        mass[pick] = {"light": 1e-25, "massless": 0.0, "heavy": 1e20, "negative": -0.5}[odd]
    elif odd == "tiny":
        pos[pick, 1] = np.float32(1e-20) * rng.standard_normal(40).astype(np.float32)
    elif odd == "far_tiny":  # pairs of tiny separations, subnormal squares among them
        pos[pick] = (10.0 ** rng.uniform(-44, -12, (40, 3))).astype(np.float32)
    else:
        with np.errstate(over="ignore"):  # infinities among them
            vel[pick] = np.float32(3e38) * rng.standard_normal((40, 3)).astype(np.float32)
    check(port, pos, vel, mass, prm, kernel)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("tile", [0, 32])
def test_scenes_of_different_ranges(port, kernel, tile):
    """A batch whose scenes' smoothing lengths admit different forms, and one out-of-range
    particle in it."""
    lengths = [0.02, 0.1, 5e-4, 2.0]
    sets = []
    for k, h in enumerate(lengths):
        pos, vel, mass, _ = block(9, 40 + k)
        s = np.float32(h / 0.02)
        sets.append((pos * s, vel, mass * s ** 3,
                     I.params16(smoothing_length=h, neighbor_search_radius=2 * h, xmin=-50 * h,
                                xmax=50 * h, ymin=-50 * h, ymax=50 * h, zmin=-50 * h, zmax=50 * h)))
    sets[1][0][3, 2] = np.float32(1e-30)
    for scenes in (sets[:1] * 2, sets[:2], sets[2:], sets):
        n = sum(len(p) for p, _, _, _ in scenes)
        start = np.cumsum([0] + [len(p) for p, _, _, _ in scenes])
        ctx = sphx.Context(n, tile_particles=tile)
        ctx.upload(*(np.concatenate([s[k] for s in scenes]) for k in range(3)))
        ctx.set_kernel(kernel)
        ctx.set_scenes(start, [s[3] for s in scenes])
        ctx.eval()
        out = ctx.download()
        ctx.close()
        for a, e, s in zip(start[:-1], start[1:], scenes):
            want = port.fields(*s, kernel=kernel)
            for got, w, key in zip((out["rho"], out["pressure"], out["acc"]), want, ("rho", "P", "acc")):
                assert O.bits_equal(got[a:e], w), O.mismatch_report(got[a:e], w, key)


@pytest.mark.parametrize("kernel,h", [(sphx.KERNEL_CUBIC_SPLINE, 0.02), (sphx.KERNEL_CUBIC_SPLINE, 0.1),
                                      (sphx.KERNEL_WENDLAND_C2, 0.02)])
def test_tiles_without_room_for_their_candidates(port, kernel, h):
    """Twelve clumps of 8,000 particles within reach of each other: 3,000 tiles that need 500
    records each, of a pool (four records a particle of capacity) that has 400 for each."""
    rng = np.random.default_rng(51)
    centre = 10 * h * np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    pos = (centre[:12] + 0.7 * h * rng.random((12, 8000, 3))).astype(np.float32).reshape(-1, 3)
    vel = (0.1 * rng.standard_normal(pos.shape)).astype(np.float32)
    mass = np.full(len(pos), 1e-3 * (h / 0.02) ** 3, np.float32)
    prm = I.params16(gas_constant=2e-3, smoothing_length=h, neighbor_search_radius=2 * h)
    check(port, pos, vel, mass, prm, kernel, capacity=300_000, tile=0)


@pytest.mark.parametrize("state_of", ["length", "half_millimetre", "tiny"])
def test_out_of_range_states_take_no_multiple_of_the_time(built, state_of):
    """The force pass of 103,823 particles at another smoothing length, or with one coordinate of
    1e-20, against the ordinary set: 1.1 and 1.5 times as long, 3 in the general form."""
    def force_time(h, tiny):
        pos, vel, mass, _ = block(47, 61)
        s = np.float32(h / 0.02)
        if tiny:
            pos[5, 0] = np.float32(1e-20)
        ctx = sphx.Context(len(pos), profile=True)
        ctx.set_params(I.params16(gas_constant=2e-3, smoothing_length=h, neighbor_search_radius=2 * h))
        ctx.upload(pos * s, vel, mass * s ** 3)
        times = []
        for _ in range(9):
            ctx.reset_stats()
            ctx.eval()
            times.append(ctx.stats()["force_computation_time"])
        ctx.close()
        return np.median(times[2:])

    plain = force_time(0.02, False)
    h = {"length": 0.1, "half_millimetre": 5e-4, "tiny": 0.02}[state_of]
    other = force_time(h, state_of == "tiny")
    assert 0 < other < 2 * plain


@pytest.mark.parametrize("kernel", KERNELS + [sphx.KERNEL_GAUSSIAN])
@pytest.mark.parametrize("count", [70_000, 300_000])
def test_lone_particles(port, kernel, count):
    """Particles without a neighbour, and a few pairs among them: no forces but in the pairs, and
    a force pass that takes no longer than the density pass."""
    rng = np.random.default_rng(71)
    k = np.arange(count)
    pos = np.stack([k % 100, k // 100 % 100, k // 10_000], -1) * 0.1 + 0.02 * rng.random((count, 3))
    pos = pos.astype(np.float32)
    pos[1:2000:100] = pos[0:2000:100] + np.float32([0.01, 0.0, 0.0])
    vel = rng.standard_normal(pos.shape).astype(np.float32)
    mass = np.full(count, 1e-3, np.float32)
    prm = I.params16(gas_constant=2e-3)
    ctx = sphx.Context(count, profile=True)
    ctx.set_params(prm)
    ctx.set_kernel(kernel)
    ctx.upload(pos, vel, mass)
    times = []
    for _ in range(7):
        ctx.reset_stats()
        ctx.eval()
        st = ctx.stats()
        times.append(st["force_computation_time"] / st["density_computation_time"])
    out = ctx.download()
    ctx.close()
    paired = np.any(out["acc"] != np.float32([0.0, prm[6], 0.0]), axis=1)
    assert np.array_equal(np.flatnonzero(paired), np.flatnonzero((k < 2000) & (k % 100 < 2)))
    if kernel != sphx.KERNEL_GAUSSIAN:
        for got, want in zip((out["rho"], out["acc"]), port.fields(pos, vel, mass, prm, kernel=kernel)[::2]):
            assert O.bits_equal(got, want)
    assert np.median(times) < 1.1
