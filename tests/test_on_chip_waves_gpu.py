"""Batches that the on-chip loop takes in several waves of shots, the last one
shorter: forward, continued and with a gradient's products, against one launch
per step; and shots without receivers among others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0
NX, NZ, NB = 661, 361, 20  # 701 x 401 padded: two shots at a time on 148 SMs, 68 blocks each


def _inputs(n):
    rng = np.random.default_rng(n)
    vp = (1700.0 + 1200.0 * rng.random((NX, NZ))).astype(np.float32)
    rho = (1000.0 + 900.0 * rng.random((NX, NZ))).astype(np.float32)
    rec = np.concatenate([np.stack([np.arange(0, NX, 3) * H, np.full(-(-NX // 3), 2 * H)], 1),
                          np.stack([np.full(NZ, 100 * H), np.arange(NZ) * H], 1)]).astype(np.float32)
    src = [((k + 0.5) * NX / n * H, (3 + 61 * k % NZ) * H) for k in range(n)]
    return vp, rho, src, rec


@pytest.mark.parametrize("n,shape,conc", [(5, 806, 2), (7, 809, 3), (3, 806, 2)])
@pytest.mark.parametrize("cuts", [(), (11, 40)])
def test_forward(n, shape, conc, cuts):
    from seis2d_b200 import Context, Shot, Wave
    vp, rho, src, rec = _inputs(n)
    steps, out = 70, []
    for on in (1, 0):
        with Context(0) as c:
            c.set_option("on_chip", on)
            c.set_option("on_chip_shape", shape)
            m = c.model(vp, rho, H, H, NB)
            buf = np.full(n * len(rec) * steps, np.nan, np.float32)
            k = 0
            for count in (*cuts, 0):
                c.forward([Shot(m, s, rec) for s in src], Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0), kt_begin=k,
                          kt_count=count, out=buf)
                if on:
                    assert c.last_stats.kernel_launches == -(-n // conc)
                k += count
            out.append(buf)
    assert np.abs(out[1]).max() > 0
    np.testing.assert_array_equal(*out)


def test_products():
    """Five shots in three waves: traces and the wavelet's gradient (per shot, in
    a fixed order) keep their bits; the shots' sums differ by their order."""
    from seis2d_b200 import Context, Shot, Wave
    n, steps = 5, 60
    vp, rho, src, rec = _inputs(n)
    adj = np.random.default_rng(9).standard_normal((n, len(rec), steps)).astype(np.float32)
    got = []
    for on in (1, 0):
        with Context(0) as c:
            c.set_option("on_chip", on)
            c.set_option("on_chip_shape", 806)
            c.set_option("grad_segment", 16)
            m = c.model(vp, rho, H, H, NB)
            g = c.gradient([Shot(m, s, rec) for s in src], Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0), adj,
                           want_seis=True)
            got.append([np.asarray(v) for v in (g.seis, g.grad_wavelet, g.grad_vp, g.grad_rho)])
    for a, b in zip(got[0][:2], got[1][:2]):
        assert np.abs(b).max() > 0
        np.testing.assert_array_equal(a, b)
    for a, b in zip(got[0][2:], got[1][2:]):
        assert np.linalg.norm(a.astype(np.float64) - b) <= n * steps * 2.0 ** -24 * np.linalg.norm(b)


def test_a_shot_without_receivers():
    from seis2d_b200 import Context, Shot, Wave
    vp, rho, src, rec = _inputs(3)
    wave = Wave(0.0695, 0.001, 0.001001, 25.0)
    with Context(0) as c:
        m = c.model(vp, rho, H, H, NB)
        ref = c.forward([Shot(m, src[1], rec)], wave)[0]
        got = c.forward([Shot(m, src[0], rec[:0]), Shot(m, src[1], rec), Shot(m, src[2], rec[:0])], wave)
        assert c.last_stats.kernel_launches == 1  # all three on chip at once
    assert got[0].size == 0 and got[2].size == 0 and np.abs(ref).max() > 0
    np.testing.assert_array_equal(got[1], ref)
