"""How a single grid is cut into tasks: where a few tasks more than the GPU holds
warps would cost some warps a second one, the cut stays within one round, and
the traces are those of any other cut."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0


# padded 2000 x 300, order 8: 1298 tasks of 7 columns take 20.4 us per step, 1154 of 15 take 15.6;
# padded 932 x 676: 14.3 us at 7 columns, 9.8 at 11 (148 SMs hold 1184 warps)
@pytest.mark.parametrize("nnx,nnz,order,least", [(2000, 300, 8, 15), (932, 676, 4, 11)])
def test_one_round(nnx, nnz, order, least):
    from seis2d_b200 import Context, Shot, Wave
    nb = 50
    nx, nz = nnx - 2 * nb, nnz - 2 * nb
    vp = np.linspace(1600.0, 3000.0, nx * nz, dtype=np.float32).reshape(nx, nz)
    rec = np.stack([np.arange(0, nx, 5) * H, np.full(-(-nx // 5), 16.0)], 1).astype(np.float32)
    got = []
    for seg in (0, 7):
        with Context(0) as c:
            c.set_option("on_chip", 0)
            c.set_option("variant", 7 if order == 8 else 5)
            c.set_option("seg_len", seg)
            m = c.model(vp, 0.5 * vp, H, H, nb, fd_order=order)
            got.append(c.forward([Shot(m, (nx // 2 * H, 16.0), rec)], Wave(0.0395, 0.001, 0.001001, 25.0))[0])
            assert c.last_stats.seg_len == 7 if seg else c.last_stats.seg_len >= least
    assert np.abs(got[0]).max() > 0
    np.testing.assert_array_equal(*got)
