"""An unstable time step: once the fields overflow, the on-chip loop records the
infinities and NaN of the per-step kernels, cell by cell (the run ends before
they reach the grid's edge)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the source in the first strip (sponge rows and others), one between the rims, the last one
@pytest.mark.parametrize("row", [60, 170, 270])
def test_overflowed_fields_keep_the_bits(row):
    from seis2d_b200 import Context, Shot, Wave
    nx, nz, nb, h, dt = 260, 320, 20, 8.0, 0.01
    vp = np.full((nx, nz), 3000.0, np.float32)
    x = nx // 2
    rec = np.concatenate([np.stack([np.full(nz, (x + k) * h), np.arange(nz) * h], 1) for k in (-5, 0, 2, 7)])
    out = []
    for on in (1, 0):
        with Context(0) as c:
            c.set_option("on_chip", on)
            m = c.model(vp, vp, h, h, nb)
            out.append(c.forward([Shot(m, (x * h, row * h), rec.astype(np.float32))], Wave(29.5 * dt, dt, dt * 1.000001, 5.0))[0])
    assert np.isinf(out[1]).any() and np.isnan(out[1]).any()
    edge = np.concatenate([out[1].reshape(4, nz, -1)[:, :8], out[1].reshape(4, nz, -1)[:, -8:]])
    assert np.isfinite(edge).all()
    np.testing.assert_array_equal(out[0], out[1])
