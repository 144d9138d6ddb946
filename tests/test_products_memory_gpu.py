"""s2d_gradient does not clear its step products: a call whose buffers hold
another call's NaN everywhere returns the bits of a fresh context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0


# grids whose last rows fill a part of a lane, a whole one, and whose last strip
# is nearly empty; on chip or one launch per step; the order-8 forms
@pytest.mark.parametrize("nx,nz,order,options", [(90, 101, 4, {}), (90, 101, 4, {"on_chip": 0}), (131, 213, 4, {"on_chip": 0}),
                                                 (90, 104, 8, {}), (131, 213, 8, {}), (90, 101, 8, {"adjoint8_form": 1})])
def test_products_of_another_call(nx, nz, order, options):
    from seis2d_b200 import Context, Shot, Wave, derive_steps
    rng = np.random.default_rng(nx * nz)
    vp = (1700.0 + 1200.0 * rng.random((nx, nz))).astype(np.float32)
    rho = (1000.0 + 900.0 * rng.random((nx, nz))).astype(np.float32)
    # a surface line and a borehole through every strip and the source's row
    rec = np.concatenate([np.stack([np.arange(nx) * H, np.full(nx, 2 * H)], 1),
                          np.stack([np.full(nz, (nx // 2 + 3) * H), np.arange(nz) * H], 1)]).astype(np.float32)
    wave = Wave(0.0395, 0.001, 0.002, 25.0)
    adj = rng.standard_normal((1, nx + nz, derive_steps(wave)["real_nt"])).astype(np.float32)

    def gradient(c, wavelet=None):
        m = c.model(vp, rho, H, H, 16, fd_order=order)
        g = c.gradient([Shot(m, (nx // 2 * H, nz // 2 * H), rec)], wave, adj, wavelet=wavelet)
        m.release()
        return [np.array(a) for a in (g.grad_vp, g.grad_rho, g.grad_wavelet)]

    def context():
        c = Context(0)
        for k, v in {"grad_segment": 13, **options}.items():
            c.set_option(k, v)
        return c

    with context() as c:
        ref = gradient(c)
    with context() as c:
        nan = gradient(c, np.full(40, np.nan))
        got = gradient(c)
    assert np.isnan(nan[0]).any() and np.abs(ref[0]).max() > 0
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)
