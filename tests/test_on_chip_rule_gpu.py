"""Which loop a batch takes: grids that fit the chip run there while that is the
faster way, and go back to launches per step where their number fills the GPU;
the bits are the same on both sides of the line, and where a gradient's sweep
and its recomputes take different ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0


def _setup(c, nnx, nnz, n, nb=50):
    from seis2d_b200 import Shot
    nx, nz = nnx - 2 * nb, nnz - 2 * nb
    vp = np.linspace(1600.0, 3000.0, nx * nz, dtype=np.float32).reshape(nx, nz)
    m = c.model(vp, 0.5 * vp, H, H, nb)
    rec = np.stack([np.arange(0, nx, 7) * H, np.full(-(-nx // 7), 16.0)], 1).astype(np.float32)
    return [Shot(m, ((k + 0.5) * nx / n * H, 16.0), rec) for k in range(n)]


# us per step on chip and launched: 44, 52; 348, 266; 113, 133; 13, 18
@pytest.mark.parametrize("nnx,nnz,n,chip", [(1080, 1080, 8, True), (1080, 1080, 64, False), (1301, 501, 32, True),
                                            (701, 401, 8, True)])
def test_forward(nnx, nnz, n, chip):
    import torch
    from seis2d_b200 import Context, Wave
    steps, out, launches = 24, [], []
    for on in (1, 0):
        with Context(0) as c:
            c.set_option("on_chip", on)
            shots = _setup(c, nnx, nnz, n)
            buf = torch.zeros(n * shots[0].rec.shape[0] * steps, device="cuda")
            out.append(c.forward(shots, Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0), out=buf))
            launches.append(c.last_stats.kernel_launches)
    assert out[1].abs().max() > 0 and torch.equal(*out)
    # launches: one per wave of shots on chip, about one per two steps otherwise
    assert (launches[0] != launches[1]) == chip


def test_a_sweep_by_launches_and_products_on_chip():
    from seis2d_b200 import Context, Wave
    n, steps, got = 40, 24, []
    rng = np.random.default_rng(1)
    for on in (1, 0):
        with Context(0) as c:
            c.set_option("on_chip", on)
            c.set_option("grad_segment", 8)
            shots = _setup(c, 1080, 1080, n)
            if not got:
                adj = rng.standard_normal((n, shots[0].rec.shape[0], steps)).astype(np.float32)
            g = c.gradient(shots, Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0), adj, want_seis=True)
            got.append((np.asarray(g.seis), np.asarray(g.grad_vp, np.float64), np.asarray(g.grad_rho, np.float64),
                        c.last_stats.kernel_launches))
    # sweep: two segments of 4 launches and their arguments; products: 40 launches of one shot, three times
    assert got[0][3] - got[1][3] == 3 * n - 3 * (8 + 1)
    assert np.abs(got[1][0]).max() > 0
    np.testing.assert_array_equal(got[0][0], got[1][0])
    # shots add to the gradient in any order: n * steps terms, each sum rounded to 2^-24
    for a, b in zip(got[0][1:3], got[1][1:3]):
        assert np.linalg.norm(a - b) <= n * steps * 2.0 ** -24 * np.linalg.norm(b)


def test_trials_beside_groups_on_chip():
    """Two grids on chip and one launched: the call that runs the trials, one
    that finds them, and one cut into pieces record the same bits."""
    import torch
    from seis2d_b200 import Context, Wave
    steps, out = 130, []
    wave = Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0)
    for on in (1, 0):
        with Context(0) as c:
            c.set_option("on_chip", on)
            shots = [s for g in ((200, 180), (2304, 800), (330, 390)) for s in _setup(c, *g, 2)]
            size = sum(s.rec.shape[0] for s in shots) * steps
            for cuts in ((), (), (85,), (3, 90), (9, 8)):
                buf = torch.zeros(size, device="cuda")
                k = 0
                for n in (*cuts, 0):
                    c.forward(shots, wave, kt_begin=k, kt_count=n, out=buf)
                    k += n
                out.append(buf)
            assert c.last_stats.autotuned == 0
    assert out[0].abs().max() > 0
    assert all(torch.equal(out[0], o) for o in out[1:])
