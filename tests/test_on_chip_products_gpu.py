"""The gradient's forward steps in the on-chip loop (every block shape, sweep and
recomputes) against one launch per step: the same bits for one shot."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0


def _gradient(nx, nz, nb, segment, surface=False, every=1, steps=45, **options):
    from seis2d_b200 import Context, Shot, Wave
    from seis2d_b200.api import derive_steps
    rng = np.random.default_rng(nx + nz)
    vp = (1700.0 + 1200.0 * rng.random((nx, nz))).astype(np.float32)
    rho = (1000.0 + 900.0 * rng.random((nx, nz))).astype(np.float32)
    rec = np.concatenate([np.stack([np.arange(nx) * H, np.full(nx, 2 * H)], 1),
                          np.stack([np.full(nz, (nx // 3) * H), np.arange(nz) * H], 1)]).astype(np.float32)
    wave = Wave((steps - 0.5) * 0.001, 0.001, every * 0.001 * 1.000001, 25.0)
    data = rng.standard_normal((rec.shape[0], derive_steps(wave)["real_nt"])).astype(np.float32)
    with Context(0) as c:
        c.set_option("grad_segment", segment)
        for k, v in options.items():
            c.set_option(k, v)
        m = c.model(vp, rho, H, H, nb, free_surface=surface)
        g = c.gradient([Shot(m, (nx // 2 * H, 3 * H), rec)], wave, data)
        return np.asarray(g.grad_vp), np.asarray(g.grad_rho), np.asarray(g.grad_wavelet)


@pytest.mark.parametrize("shape", [403, 404, 803, 804, 805, 806, 807, 808, 809, 810])
def test_shapes(shape):
    a = _gradient(60, 110, 12, 20, on_chip_shape=shape)
    b = _gradient(60, 110, 12, 20, on_chip=0)
    assert np.abs(b[0]).max() > 0
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


# one and several blocks along x and z, segments that leave one step over
@pytest.mark.parametrize("nx,nz,nb,segment,surface,every", [(30, 96, 12, 44, False, 1), (150, 97, 12, 11, True, 3),
                                                            (301, 241, 20, 0, False, 2), (90, 400, 16, 8, True, 1)])
def test_grids(nx, nz, nb, segment, surface, every):
    a = _gradient(nx, nz, nb, segment, surface, every)
    b = _gradient(nx, nz, nb, segment, surface, every, on_chip=0)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
