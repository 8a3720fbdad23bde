"""Contexts that nearly fill the GPU's memory."""
import numpy as np
import pytest

import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [sphx.MODE_PRECISE, sphx.MODE_PRECISE_FP16])
def test_a_precision_context_leaves_room_for_a_snapshot(built, mode):
    import torch

    n = 8_000_000
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    sphx.Context(1000, mode=mode).close()  # (what the library allocates once)
    before = free()
    ctx = sphx.Context(n, mode=mode)
    takes = before - free()
    ctx.close()
    snapshot = 48 * n
    assert takes > 8 * snapshot
    # what is left holds the context as it is made when memory is plentiful, and half a snapshot
    filler = torch.empty(free() - takes - snapshot // 2, dtype=torch.uint8, device="cuda")
    ctx = sphx.Context(n, mode=mode)
    try:
        ctx.set_params(I.params16())
        pos = I.lattice(20, 20, 20)
        ctx.upload(pos, None, np.full(len(pos), 1e-3, np.float32))
        ctx.snapshot()
        ctx.step(1e-4)
        ctx.restore()
        assert ctx.download(rho=False, pressure=False, acc=False)["pos"].shape == pos.shape
    finally:
        ctx.close()
        del filler
        torch.cuda.empty_cache()
