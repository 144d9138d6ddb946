"""The 4th-order gradient against the FP64 discrete adjoint, at the accuracy of
its arithmetic: 80 steps of some 30 roundings to 2^-24, forward and back, whose
random walk is sqrt(4800) * 2^-24 = 4e-6 of the fields; the bar is five times that."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 2e-5
H = 8.0


# receivers and source at strip seams (120 rows), in the sponge's rows and columns and on top of one another
@pytest.mark.parametrize("nx,nz,surface,every,on_chip", [(70, 230, False, 1, 1), (70, 230, False, 1, 0), (133, 101, True, 2, 1),
                                                         (133, 101, True, 2, 0), (45, 341, False, 3, 0)])
def test_gradient(nx, nz, surface, every, on_chip):
    from seis2d_b200 import Context, Shot, Wave
    nb, steps, dt = 16, 80, 0.001
    rng = np.random.default_rng(nx)
    x, z = np.linspace(0, 1, nx)[:, None], np.linspace(0, 1, nz)[None, :]
    vp = (1800 + 900 * z + 120 * np.sin(6 * x) * np.cos(5 * z) + 0 * x).astype(np.float32)
    rho = (1300 + 600 * z + 80 * np.cos(4 * x + 3 * z)).astype(np.float32)
    rec = np.concatenate([np.stack([np.arange(nx), np.full(nx, 3)], 1), np.stack([np.full(nz, nx // 3), np.arange(nz)], 1),
                          np.full((3, 2), 5), np.stack([np.arange(-nb + 2, nx + nb - 3), np.full(nx + 2 * nb - 5, 104)], 1)])
    rec = ((rec[rec[:, 1] < nz + nb - 3] + 0.25) * H).astype(np.float32)
    src = (float((nx // 2 + 0.25) * H), float((min(87, nz // 2) + 0.25) * H))
    T = (steps - 0.5) * dt
    p = O.Params(nx, nz, nb, H, H, T, dt, every * dt * 1.000001, 25.0, 1 if surface else 0)
    nt = O.derive(p)["real_nt"]
    # a smooth adjoint source, as residuals are
    t = np.arange(nt) / nt
    adj = sum(rng.standard_normal((len(rec), 1)) * np.sin((k + 1) * np.pi * t)[None, :] for k in range(4)).astype(np.float32)
    with Context(0) as c:
        c.set_option("on_chip", on_chip)
        c.set_option("grad_segment", 23)
        m = c.model(vp, rho, H, H, nb, free_surface=surface)
        g = c.gradient([Shot(m, src, rec)], Wave(T, dt, every * dt * 1.000001, 25.0), adj)
    ref = O.gradient(p, vp, rho, src, rec[:, 0], rec[:, 1], adj.astype(np.float64))
    assert O.rel_l2(np.asarray(g.grad_vp), ref["grad_vp"]) <= TOL
    assert O.rel_l2(np.asarray(g.grad_rho), ref["grad_rho"]) <= TOL
