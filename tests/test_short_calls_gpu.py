"""Calls of a few steps on grids above the two-step kernel's line: a call of
one step runs a one-step kernel, tuned shape or not, and runs cut into short
calls record the bits of one call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0
TWO_STEP = (5, 6)  # the two-step kernel and its remainder launch


@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("plain", [False, True])
def test_one_step_calls(tuned, plain):
    import torch
    from seis2d_b200 import Context, Shot, Wave, derive_steps
    nx, nz, nb, steps = 1290, 1210, 16, 130  # 1.64 M padded cells: too large for the on-chip loop
    vp = np.linspace(1600.0, 3000.0, nx * nz, dtype=np.float32).reshape(nx, nz)
    rec = np.stack([np.arange(0, nx, 3) * H, np.full(-(-nx // 3), 24.0)], 1).astype(np.float32)
    wave = Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0)
    with Context(0) as c:
        m = c.model(vp, 0.5 * vp, H, H, nb)
        shots = [Shot(m, (nx // 2 * H, 24.0), rec)]
        whole = c.forward(shots, wave, plain=plain)[0]
        out = torch.zeros(whole.size, device="cuda")
        assert derive_steps(wave)["fd_nt"] == steps
        k = 0
        if tuned:
            c.forward(shots, wave, kt_count=100, out=out, plain=plain)
            k = 100
        for n in (1, 1, 3, 2, 1, 5):
            c.forward(shots, wave, kt_begin=k, kt_count=n, out=out, plain=plain)
            assert (c.last_stats.variant in TWO_STEP) == (n > 1)
            k += n
        c.forward(shots, wave, kt_begin=k, out=out, plain=plain)
    np.testing.assert_array_equal(out.cpu().numpy().reshape(whole.shape), whole)
