"""The precision mode's force sweep over the density sweep's candidate lists."""
import numpy as np
import pytest

import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


def evaluate(pos, vel, mass, prm, capacity=0, kernel=0, mode=sphx.MODE_PRECISE):
    ctx = sphx.Context(max(capacity, len(pos)), mode=mode)
    ctx.set_params(prm)
    ctx.set_kernel(kernel)
    ctx.upload(pos, vel, mass)
    ctx.eval()
    out = ctx.download()
    ctx.close()
    return out


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2])
def test_an_overflowing_viscosity_factor_reaches_neighbours_only(built, kernel):
    """A particle whose viscosity factor overflows beside a clump whose factors do not: the
    clump's particles out of its reach feel nothing of it.  The velocities are zero, so that
    they get what they get without viscosity."""
    rng = np.random.default_rng(1)
    u = rng.standard_normal((200, 3))
    clump = 0.5 + 0.004 * u / np.linalg.norm(u, axis=1)[:, None]
    pos = np.concatenate([clump, [[0.54, 0.5, 0.5]]]).astype(np.float32)
    vel, mass = np.zeros_like(pos), np.full(len(pos), 1e-3, np.float32)
    # (m / rho) mu kl: 1.5 mu / h^2 and 5 mu / h^2 on its own, 1/200 of that in the clump
    want = evaluate(pos, vel, mass, I.params16(gas_constant=2e-3, viscosity=0.0), kernel=kernel)
    got = evaluate(pos, vel, mass, I.params16(gas_constant=2e-3, viscosity=2e35), kernel=kernel)
    away = np.linalg.norm(pos.astype(np.float64) - pos[-1], axis=1) > 0.0401
    assert 20 < away.sum() < 180
    assert got["acc"][away].tobytes() == want["acc"][away].tobytes()
    assert got["rho"].tobytes() == want["rho"].tobytes()


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2,
                                    sphx.KERNEL_GAUSSIAN])
@pytest.mark.parametrize("h", [7e11, 1e12])
def test_lengths_whose_kernel_gradient_underflows(built, kernel, h):
    """Kernel gradients below the smallest float give no force: gravity is what remains."""
    rng = np.random.default_rng(2)
    pos = (4 * h * rng.random((300, 3))).astype(np.float32)
    vel = rng.standard_normal(pos.shape).astype(np.float32)
    prm = I.params16(smoothing_length=h, neighbor_search_radius=2 * h)
    acc = evaluate(pos, vel, np.full(len(pos), 2.0 ** 120, np.float32), prm, kernel=kernel)["acc"]
    assert np.array_equal(acc, np.tile(np.float32([0.0, prm[6], 0.0]), (300, 1)))


@pytest.mark.parametrize("kernel", [sphx.KERNEL_CUBIC_SPLINE, sphx.KERNEL_WENDLAND_C2])
def test_tiles_without_room_for_their_list(built, kernel):
    """Six clumps of 16,000 particles within reach of each other: 3,000 tiles that need 500
    records each.  A pool of four records a particle of a capacity of 300,000 has 400 for each,
    the one of a larger context enough; the two passes sum the same terms in other chunks."""
    rng = np.random.default_rng(3)
    centre = 0.3 * np.arange(6)[:, None, None] * np.ones(3)
    pos = (centre + 0.014 * rng.random((6, 16_000, 3))).astype(np.float32).reshape(-1, 3)
    vel = (0.1 * rng.standard_normal(pos.shape)).astype(np.float32)
    mass = np.full(len(pos), 1e-3, np.float32)
    prm = I.params16(gas_constant=2e-3, xmax=3, ymax=3, zmax=3)
    a, b = (evaluate(pos, vel, mass, prm, capacity=c, kernel=kernel) for c in (300_000, 3_000_000))
    assert a["rho"].tobytes() == b["rho"].tobytes()
    # 16,000 terms of a few ulp (2^-23) each, of at most the largest acceleration's size in sum
    scale = np.abs(b["acc"]).max()
    assert np.abs(a["acc"].astype(np.float64) - b["acc"]).max() < 16 * 2.0 ** -23 * scale
