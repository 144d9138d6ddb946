"""The adjoint step's tasks at their edges (rim and interior cuts, strips,
segments, receivers): against the FP64 discrete adjoint, and the same bits for
one shot however its tasks are cut."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRAD_TOL = 1e-4  # rel-L2 of the FP32 gradient against the FP64 adjoint
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
    p = O.Params(nx, nz, nb, H, H, 0.06, 0.001, 0.002, 25.0, 1 if surface else 0)
    adj = rng.standard_normal((sources, rec.shape[0], O.derive(p)["real_nt"])).astype(np.float32)
    return vp, rho, rec, src, p, adj


def _gradient(case, nb, surface, seg=0, order=1, fast=1):
    from seis2d_b200 import Context, Shot, Wave
    vp, rho, rec, src, p, adj = case
    with Context(0) as c:
        c.set_option("seg_len", seg)
        c.set_option("task_order", order)
        c.set_option("fast_rows", fast)
        m = c.model(vp, rho, H, H, nb, free_surface=surface)
        g = c.gradient([Shot(m, s, rec) for s in src], Wave(0.06, 0.001, 0.002, 25.0), adj)
        return np.asarray(g.grad_vp), np.asarray(g.grad_rho)


# padded rows at the strips' edges (120 rows, reading 128), padded columns with
# no, the narrowest and several interior segments; one and several shots
@pytest.mark.parametrize("nnx,nnz,shots,surface", [(40, 120, 1, False), (41, 121, 2, True), (49, 359, 1, False),
                                                   (50, 360, 3, False), (51, 361, 1, True), (150, 485, 2, False)])
def test_grids_at_the_cuts(nnx, nnz, shots, surface):
    nb = 16
    case = _case(nnx - 2 * nb, nnz - 2 * nb, nb, surface, shots)
    gv, gr = _gradient(case, nb, surface)
    vp, rho, rec, src, p, adj = case
    rv, rr = 0, 0
    for s, a in zip(src, adj):
        ref = O.gradient(p, vp, rho, s, rec[:, 0], rec[:, 1], a.astype(np.float64))
        rv, rr = rv + ref["grad_vp"], rr + ref["grad_rho"]
    assert O.rel_l2(gv, rv) <= GRAD_TOL and O.rel_l2(gr, rr) <= GRAD_TOL


@pytest.mark.parametrize("seg,order,fast", [(4, 0, 1), (7, 1, 1), (33, 0, 0), (255, 1, 0)])
def test_one_shot_keeps_its_bits(seg, order, fast):
    nb = 12
    case = _case(150, 420, nb, False, 1)
    a = _gradient(case, nb, False)
    b = _gradient(case, nb, False, seg=seg, order=order, fast=fast)
    assert np.abs(a[0]).max() > 0
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])
