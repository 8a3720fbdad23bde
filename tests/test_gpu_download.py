"""Downloads into pinned memory (stored there by one kernel) against downloads into pageable
memory (device staging and copies): the same bytes, whatever the count, the alignment of the
caller's arrays, the order of the particles, the fields asked for and the mode."""
import numpy as np
import pytest
import torch

import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu

FIELDS = (("pos", 3), ("vel", 3), ("rho", 1), ("pressure", 1), ("acc", 3))


@pytest.mark.parametrize("mode", [sphx.MODE_EXACT, sphx.MODE_PRECISE, sphx.MODE_PRECISE_FP16])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 4099, 70001])
@pytest.mark.parametrize("offset", [0, 1])  # floats past a 16-byte boundary
def test_pinned_and_pageable_downloads_agree(built, n, mode, offset):
    rng = np.random.default_rng(n)
    side = (n * 1e-6) ** (1 / 3)
    pos = (0.5 + side * rng.random((n, 3))).astype(np.float32)  # no order
    vel = rng.standard_normal((n, 3)).astype(np.float32)
    ctx = sphx.Context(n, mode=mode)
    ctx.set_params(I.params16())
    ctx.upload(pos, vel, np.full(n, 1e-3, np.float32))
    ctx.step(1e-4)
    want = ctx.download()  # pageable
    for fields in (("pos", "vel", "rho", "pressure", "acc"), ("acc",), ("vel", "pressure"), ("pos",)):
        out = {k: torch.full((w * n + 8,), 7.0, dtype=torch.float32, pin_memory=True)
               for k, w in FIELDS}
        ctx.download_ptr(*[out[k].data_ptr() + 4 * offset if k in fields else 0 for k, _ in FIELDS])
        for k, w in FIELDS:
            got = out[k].numpy()
            if k in fields:
                assert got[offset:offset + w * n].tobytes() == want[k].tobytes(), k
                got = np.concatenate([got[:offset], got[offset + w * n:]])
            assert (got == 7.0).all(), k  # nothing else written
    ctx.close()


@pytest.mark.parametrize("mode", [sphx.MODE_EXACT, sphx.MODE_PRECISE, sphx.MODE_PRECISE_FP16])
@pytest.mark.parametrize("pinned", [("pos",), ("vel", "mass"), ("pos", "vel", "mass")])
@pytest.mark.parametrize("with_vel", [True, False])
def test_fp64_uploads_from_pinned_memory_agree(built, mode, pinned, with_vel):
    """Positions in FP64 from pinned memory (read in place), pageable memory (staged) and mixtures
    of both: the same state."""
    n = 5001
    rng = np.random.default_rng(n)
    src = {"pos": 1000.0 + 0.2 * rng.random((n, 3)),
           "vel": rng.standard_normal((n, 3)).astype(np.float32),
           "mass": np.full(n, 1e-3, np.float32) * (1 + np.arange(n, dtype=np.float32) % 3)}
    held = {k: torch.from_numpy(v).pin_memory() for k, v in src.items() if k in pinned}

    def state(arrays):
        ctx = sphx.Context(n, mode=mode)
        ctx.set_params(I.params16(xmin=0.0, xmax=2e3, ymin=0.0, ymax=2e3, zmin=0.0, zmax=2e3))
        ctx.upload_f64(arrays["pos"], arrays["vel"] if with_vel else None, arrays["mass"])
        ctx.step(1e-4)
        out = ctx.download()
        ctx.close()
        return out

    want = state(src)
    got = state({k: held[k].numpy() if k in held else v for k, v in src.items()})
    for k in want:
        assert got[k].tobytes() == want[k].tobytes(), k
