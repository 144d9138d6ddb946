"""The two-step kernel's tasks at their edges (rim and interior cuts, strips,
segments, receivers) against the plain-load kernel: the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(variant, nx, nz, nb, shots, steps, rec, seg=0, order=1, fast=1, surface=False, every=1, h=8.0):
    from seis2d_b200 import Context, Shot, Wave
    rng = np.random.default_rng(nx + nz)
    vp = (1700.0 + 1200.0 * rng.random((nx, nz))).astype(np.float32)
    rho = (1000.0 + 900.0 * rng.random((nx, nz))).astype(np.float32)
    with Context(0) as c:
        c.set_option("variant", variant)
        c.set_option("seg_len", seg)
        c.set_option("task_order", order)
        c.set_option("fast_rows", fast)
        m = c.model(vp, rho, h, h, nb, free_surface=surface)
        sh = [Shot(m, ((k + 0.5) * nx / shots * h, (0.25 + (k * 131) % nz) * h), rec) for k in range(shots)]
        return np.concatenate([o.ravel() for o in c.forward(sh, Wave((steps - 0.5) * 0.001, 0.001,
                                                                     every * 0.001 * 1.000001, 25.0))])


def _surface(nx, h=8.0):
    return np.stack([(np.arange(nx) + 0.25) * h, np.full(nx, 2.25 * h)], 1).astype(np.float32)


# padded rows at the strips' edges (112 rows, reading 128), padded columns
# with no, the narrowest and several interior segments
@pytest.mark.parametrize("nnx,nnz", [(40, 112), (41, 113), (60, 335), (61, 336), (62, 337), (63, 448), (197, 449),
                                     (300, 700)])
def test_grids_at_the_cuts(nnx, nnz):
    nb = 16
    nx, nz = nnx - 2 * nb, nnz - 2 * nb
    a = _run(5, nx, nz, nb, 3, 41, _surface(nx))
    b = _run(1, nx, nz, nb, 3, 41, _surface(nx))
    assert np.abs(b).max() > 0
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("seg,order,fast,surface,every", [(4, 0, 1, False, 1), (7, 1, 1, True, 2), (33, 0, 0, False, 3),
                                                          (255, 1, 1, False, 1)])
def test_options(seg, order, fast, surface, every):
    nx, nz, nb = 150, 420, 12
    # a surface line, a borehole through every strip, several receivers on one cell
    rec = np.concatenate([_surface(nx), np.stack([np.full(80, 600.0), np.linspace(0, nz - 1, 80) * 8.0], 1),
                          np.full((5, 2), 402.0)]).astype(np.float32)
    kw = dict(surface=surface, every=every, fast=fast)
    a = _run(5, nx, nz, nb, 4, 60, rec, seg=seg, order=order, **kw)
    b = _run(1, nx, nz, nb, 4, 60, rec, **kw)
    np.testing.assert_array_equal(a, b)
