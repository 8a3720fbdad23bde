"""A failed call reports its error itself; the calls after it do not report it again."""
import numpy as np
import pytest

import sphx
import sphx_inputs as I

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_is_reported_once(built):
    rng = np.random.default_rng(3)
    pos = (0.2 * rng.random((3000, 3))).astype(np.float32)
    ctx = sphx.Context(len(pos))
    ctx.set_params(I.params16())
    ctx.upload(pos, np.zeros_like(pos), np.full(len(pos), 1e-3, np.float32))
    grid = sphx.Grid(len(pos))
    grid.build(pos, 0.04)
    want = grid.query(pos[:50], 1e-4)
    for call in (lambda: ctx.step(1e-4), lambda: grid.build(pos, 0.04),
                 lambda: grid.query(pos[:50], 1e-4), ctx.download):
        with pytest.raises(sphx.SphxError) as e:  # some 500 GB
            sphx.Context((1 << 31) - 100)
        assert e.value.code == -2
        call()
    got = grid.query(pos[:50], 1e-4)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    grid.close()
    ctx.close()
