"""Pinned arrays that are not aligned to their elements (views into a packed block) take the
staged path: the same state and the same bytes as from and into ordinary arrays."""
import numpy as np
import pytest

import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


def pinned_block(nbytes):
    import torch

    return torch.zeros(nbytes + 64, dtype=torch.uint8, pin_memory=True).numpy()


def put(block, at, a):
    block[at:at + a.nbytes] = np.frombuffer(a.tobytes(), np.uint8)
    return block.ctypes.data + at


def particles(n):
    rng = np.random.default_rng(n)
    pos = 0.5 + (n * 1e-6) ** (1 / 3) * rng.random((n, 3))
    return pos, rng.standard_normal((n, 3)).astype(np.float32), np.full(n, 1e-3, np.float32)


def context(n, mode):
    ctx = sphx.Context(n, mode=mode)
    ctx.set_params(I.params16())
    return ctx


def state_after_step(ctx):
    ctx.step(1e-4)
    out = ctx.download()
    out["pos64"] = ctx.positions_f64()
    return out


def same(a, b):
    for k in b:
        assert a[k].tobytes() == b[k].tobytes(), k


@pytest.mark.parametrize("mode", [sphx.MODE_EXACT, sphx.MODE_PRECISE])
@pytest.mark.parametrize("n", [1, 1001, 70_001])  # odd: 3 n floats end on a 4-byte boundary
def test_fp64_positions_behind_floats(built, n, mode):
    pos, vel, mass = particles(n)
    ctx = context(n, mode)
    ctx.upload_f64(pos.copy(), vel.copy(), mass.copy())
    want = state_after_step(ctx)
    block = pinned_block(vel.nbytes + pos.nbytes + mass.nbytes)
    base = -block.ctypes.data % 16
    at = [base, base + vel.nbytes, base + vel.nbytes + pos.nbytes]
    p = [put(block, o, a) for o, a in zip(at, (vel, pos, mass))]
    assert p[1] % 8 == 4
    for with_vel in (True, False):
        # (without velocities the exact mode has no reason to wait for the positions)
        ctx.set_time(0.0)
        if with_vel:
            ctx._check(ctx._lib.sphx_upload_f64(ctx._h, n, p[1], p[0], p[2]), "sphx_upload_f64")
            same(state_after_step(ctx), want)
        else:
            ctx._check(ctx._lib.sphx_upload_f64(ctx._h, n, p[1], None, p[2]), "sphx_upload_f64")
            got = ctx.positions_f64()
            ctx.upload_f64(pos.copy(), None, mass.copy())
            assert got.tobytes() == ctx.positions_f64().tobytes()
    ctx.close()


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("n", [127, 4099])
def test_floats_at_odd_addresses(built, n, shift):
    pos, vel, mass = particles(n)
    pos = pos.astype(np.float32)
    ctx = context(n, sphx.MODE_EXACT)
    ctx.upload(pos, vel, mass)
    want = state_after_step(ctx)
    blocks = [pinned_block(a.nbytes) for a in (pos, vel, mass)]
    ctx.set_time(0.0)
    ctx.upload_ptr(n, *[put(b, shift, a) for b, a in zip(blocks, (pos, vel, mass))])
    same(state_after_step(ctx), want)
    names = ("pos", "vel", "rho", "pressure", "acc")
    for fields in (names, ("rho",), ("acc",)):
        out = {k: pinned_block(want[k].nbytes) for k in names}
        ctx.download_ptr(*[out[k].ctypes.data + shift if k in fields else 0 for k in names])
        for k in names:
            w = want[k].tobytes() if k in fields else b"\0" * want[k].nbytes
            got = out[k].tobytes()
            assert got[shift:shift + len(w)] == w, k
            assert not any(got[:shift]) and not any(got[shift + len(w):]), k
    ctx.close()


def register(cudart, a, first, bytes_):
    assert int(cudart.cudaHostRegister(a.ctypes.data + first, bytes_, 0)) == 0


@pytest.mark.parametrize("gap", [False, True])
def test_arrays_across_two_registrations(built, gap):
    """Two registered ranges that follow one another are pinned memory throughout; with pageable
    memory between them an array is neither one nor the other, which the copies refuse."""
    import torch

    n, page = 60_000, 65536
    pos, vel, mass = particles(n)
    ctx = context(n, sphx.MODE_EXACT)
    ctx.upload_f64(pos, vel, mass)
    want = state_after_step(ctx)
    raw = np.zeros(25 * page, np.uint8)
    block = raw[-raw.ctypes.data % page:][:24 * page]  # whole pages
    cudart = torch.cuda.cudart()
    first = 4 * page
    register(cudart, block, 0, first)
    second = first + (page if gap else 0)
    register(cudart, block, second, 24 * page - second)
    try:
        put(block, 0, pos)
        assert first < pos.nbytes < 24 * page and second < 3 * 4 * n
        f = ctx._lib.sphx_upload_f64
        rc = f(ctx._h, n, block.ctypes.data, vel.ctypes.data, mass.ctypes.data)
        assert (rc != sphx.OK) == gap
        if not gap:
            ctx.set_time(0.0)
            same(state_after_step(ctx), want)
        block[:] = 0
        ctx.upload_f64(pos, vel, mass)
        ctx.set_time(0.0)
        ctx.step(1e-4)
        rc = ctx._lib.sphx_download(ctx._h, block.ctypes.data, None, None, None, None)
        assert (rc != sphx.OK) == gap
        got = block[:want["pos"].nbytes].tobytes()
        assert got == (b"\0" * len(got) if gap else want["pos"].tobytes())
        same(ctx.download(), {k: v for k, v in want.items() if k != "pos64"})
    finally:
        ctx.close()
        for at in (0, second):
            cudart.cudaHostUnregister(block.ctypes.data + at)
