"""A context's device memory (pieces of shared chunks, reused as they come back)
and the source terms computed on the device: the same bits as a fresh context
whatever ran before, and the reference's wavelet given as samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0


def _model(nx, nz, seed):
    rng = np.random.default_rng(seed)
    return ((1700.0 + 1200.0 * rng.random((nx, nz))).astype(np.float32),
            (1000.0 + 900.0 * rng.random((nx, nz))).astype(np.float32))


def _geometry(nx, shots):
    rec = np.stack([np.arange(nx) * H, np.full(nx, 2 * H)], 1).astype(np.float32)
    return [((k + 1) * nx // (shots + 1) * H, 3 * H) for k in range(shots)], rec


# grids below a chunk, of pieces above the largest one, several in one call;
# shot counts that change from call to call
JOBS = [([(60, 40)], 1), ([(700, 900), (60, 40)], 2), ([(60, 40)], 5), ([(1500, 1600)], 1), ([(130, 70), (300, 200)], 3),
        ([(60, 40)], 1)]


def _run(ctx, job, wave, sync):
    import torch
    from seis2d_b200 import Shot, derive_steps
    grids, n = job
    models, shots = [], []
    for i, (nx, nz) in enumerate(grids):
        m = ctx.model(*_model(nx, nz, i), H, H, 16)
        src, rec = _geometry(nx, n)
        models.append(m)
        shots += [Shot(m, s, rec) for s in src]
    size = sum(s.rec.shape[0] for s in shots) * derive_steps(wave)["real_nt"]
    out = torch.full((size,), 7.0, device="cuda")
    ctx.forward(shots, wave, out=out, sync=sync)
    for m in models:
        m.release()
    return out


@pytest.mark.parametrize("sync", [True, False])
def test_reused_memory_changes_nothing(sync):
    import torch
    from seis2d_b200 import Context, Wave
    wave = Wave(0.0395, 0.001, 0.001, 25.0)
    with Context(0) as c:
        got = [_run(c, j, wave, sync) for j in JOBS for _ in range(2)]
        torch.cuda.synchronize()
    for i, j in enumerate(JOBS):
        with Context(0) as c:
            ref = _run(c, j, wave, True)
        assert ref.abs().max() > 0
        assert torch.equal(got[2 * i], ref) and torch.equal(got[2 * i + 1], ref)


@pytest.mark.parametrize("n", [0, 1, 17, 40, 55])
def test_wavelet_samples(n):
    """The first n samples given (fewer and more than the 40 steps): the traces
    up to the first missing one are those of the whole wavelet; none: silence."""
    from seis2d_b200 import Context, Shot, Wave
    wave = Wave(0.0395, 0.001, 0.001, 25.0)
    vp, rho = _model(60, 40, 3)
    (src,), rec = _geometry(60, 1)
    w = np.random.default_rng(5).standard_normal(55)
    with Context(0) as c:
        m = c.model(vp, rho, H, H, 16)
        whole = np.array(c.forward([Shot(m, src, rec)], wave, wavelet=w)[0])
        part = np.array(c.forward([Shot(m, src, rec)], wave, wavelet=w[:n])[0])
    assert np.abs(whole).max() > 0
    if n == 0:
        assert np.all(part == 0)
    else:
        np.testing.assert_array_equal(part[:, :n], whole[:, :n])
        assert n >= 40 or not np.array_equal(part, whole)


def test_surface_source_is_silent():
    from seis2d_b200 import Context, Shot, Wave
    vp, rho = _model(60, 40, 3)
    _, rec = _geometry(60, 1)
    with Context(0) as c:
        m = c.model(vp, rho, H, H, 16, free_surface=True)
        a, b = c.forward([Shot(m, (30 * H, 0.0), rec), Shot(m, (30 * H, 2 * H), rec)], Wave(0.0395, 0.001, 0.001, 25.0))
        assert np.all(a == 0) and np.abs(b).max() > 0
