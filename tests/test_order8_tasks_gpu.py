"""The 8th-order step's tasks at their edges (rim and interior cuts, strips,
segments, receivers): against the FP64 oracle, and the same bits however its
tasks are cut."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5  # rel-L2 of the FP32 traces against the FP64 oracle, as the order's other tests
H = 8.0


def _case(nx, nz, shots):
    rng = np.random.default_rng(nx + nz)
    vp = (1700.0 + 1200.0 * rng.random((nx, nz))).astype(np.float32)
    rho = (1000.0 + 900.0 * rng.random((nx, nz))).astype(np.float32)
    # a surface line, a borehole through every strip, several receivers on one cell
    rec = np.concatenate([np.stack([np.arange(nx) * H, np.full(nx, 2 * H)], 1),
                          np.stack([np.full(nz, (nx // 3) * H), np.arange(nz) * H], 1),
                          np.full((3, 2), 5 * H)]).astype(np.float32)
    src = [((k + 1) * nx // (shots + 1) * H, (3 + (k * 131) % (nz - 3)) * H) for k in range(shots)]
    return vp, rho, rec, src


def _forward(case, nb, surface, **options):
    from seis2d_b200 import Context, Shot, Wave
    vp, rho, rec, src = case
    with Context(0) as c:
        for k, v in options.items():
            c.set_option(k, v)
        m = c.model(vp, rho, H, H, nb, free_surface=surface, fd_order=8)
        return [np.array(t) for t in c.forward([Shot(m, s, rec) for s in src], Wave(0.06, 0.001, 0.002, 25.0))]


# padded rows at the strips' edges (112 rows, reading 128), padded columns with
# no, the narrowest and several interior segments
@pytest.mark.parametrize("nnx,nnz,shots,surface", [(40, 112, 1, False), (47, 113, 2, True), (48, 335, 1, False),
                                                   (54, 336, 3, False), (61, 337, 1, True), (170, 461, 2, False)])
def test_grids_at_the_cuts(nnx, nnz, shots, surface):
    nb = 16
    case = _case(nnx - 2 * nb, nnz - 2 * nb, shots)
    vp, rho, rec, src = case
    p = O.Params(nnx - 2 * nb, nnz - 2 * nb, nb, H, H, 0.06, 0.001, 0.002, 25.0, 1 if surface else 0, 8)
    for s, t in zip(src, _forward(case, nb, surface)):
        assert O.rel_l2(t, O.forward(p, vp, rho, s, rec[:, 0], rec[:, 1], O.F64)) <= TOL


@pytest.mark.parametrize("options", [dict(seg_len=4, task_order=0), dict(seg_len=7, fast_rows=0),
                                     dict(seg_len=33, task_order=0, fast_rows=0), dict(seg_len=255), dict(variant=9)])
def test_cuts_keep_the_bits(options):
    case = _case(150, 420, 3)
    a, b = _forward(case, 12, False), _forward(case, 12, False, **options)
    for x, y in zip(a, b):
        assert np.abs(x).max() > 0
        np.testing.assert_array_equal(x, y)
