"""The 8th-order adjoint step's tasks at their edges (rim and interior cuts,
strips, segments, receivers): against the FP64 discrete adjoint and the
cell-parallel form, and the same bits for one shot however its tasks are cut."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRAD_TOL = 1e-4  # rel-L2 of the FP32 gradient against the FP64 adjoint, as the order's other tests
FORM_TOL = 1e-6  # rel-L2 of the two forms: sums of the same products, in FP32
H = 8.0


def _case(nx, nz, nb, surface, sources):
    rng = np.random.default_rng(nx + nz)
    vp = (1700.0 + 1200.0 * rng.random((nx, nz))).astype(np.float32)
    rho = (1000.0 + 900.0 * rng.random((nx, nz))).astype(np.float32)
    # a surface line, a borehole through every strip, several receivers on one cell
    rec = np.concatenate([np.stack([np.arange(nx) * H, np.full(nx, 2 * H)], 1),
                          np.stack([np.full(nz, (nx // 3) * H), np.arange(nz) * H], 1),
                          np.full((3, 2), 5 * H)]).astype(np.float32)
    src = [((k + 1) * nx // (sources + 1) * H, (3 + (k * 131) % (nz - 3)) * H) for k in range(sources)]
    p = O.Params(nx, nz, nb, H, H, 0.06, 0.001, 0.002, 25.0, 1 if surface else 0, 8)
    adj = rng.standard_normal((sources, rec.shape[0], O.derive(p)["real_nt"])).astype(np.float32)
    return vp, rho, rec, src, p, adj


def _gradient(case, nb, surface, **options):
    from seis2d_b200 import Context, Shot, Wave
    vp, rho, rec, src, p, adj = case
    with Context(0) as c:
        for k, v in options.items():
            c.set_option(k, v)
        m = c.model(vp, rho, H, H, nb, free_surface=surface, fd_order=8)
        g = c.gradient([Shot(m, s, rec) for s in src], Wave(0.06, 0.001, 0.002, 25.0), adj)
        return np.asarray(g.grad_vp), np.asarray(g.grad_rho), np.asarray(g.grad_wavelet)


# padded rows at the strips' edges (112 rows, reading 128; 461: a strip with
# sponge rows and no edge rows), padded columns with no, the narrowest and
# several interior segments; one and several shots
@pytest.mark.parametrize("nnx,nnz,shots,surface", [(40, 112, 1, False), (53, 113, 2, True), (54, 335, 1, False),
                                                   (55, 336, 3, False), (61, 361, 1, True), (170, 461, 2, False)])
def test_grids_at_the_cuts(nnx, nnz, shots, surface):
    nb = 16
    case = _case(nnx - 2 * nb, nnz - 2 * nb, nb, surface, shots)
    gv, gr, gw = _gradient(case, nb, surface)
    vp, rho, rec, src, p, adj = case
    rv, rr = 0, 0
    for s, a in zip(src, adj):
        ref = O.gradient(p, vp, rho, s, rec[:, 0], rec[:, 1], a.astype(np.float64))
        rv, rr = rv + ref["grad_vp"], rr + ref["grad_rho"]
    assert O.rel_l2(gv, rv) <= GRAD_TOL and O.rel_l2(gr, rr) <= GRAD_TOL
    ov, orho, ow = _gradient(case, nb, surface, adjoint8_form=1)
    assert O.rel_l2(gv, ov) <= FORM_TOL and O.rel_l2(gr, orho) <= FORM_TOL
    assert O.rel_l2(gw, ow) <= FORM_TOL


@pytest.mark.parametrize("options", [dict(seg_len=4, task_order=0), dict(seg_len=7), dict(seg_len=33, fast_rows=0),
                                     dict(seg_len=255, task_order=0, fast_rows=0), dict(graph_chunk=7)])
def test_one_shot_keeps_its_bits(options):
    nb = 12
    case = _case(150, 420, nb, False, 1)
    a = _gradient(case, nb, False)
    b = _gradient(case, nb, False, **options)
    for x, y in zip(a, b):
        assert np.abs(x).max() > 0
        np.testing.assert_array_equal(x, y)
