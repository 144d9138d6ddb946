"""More shots in one call than a grid's y and z dimensions count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("on_chip", [0, 1])
def test_more_than_65535_shots(on_chip):
    import torch
    from seis2d_b200 import Context, Shot, Wave
    vp = np.full((6, 6), 2000.0, np.float32)
    rec = np.array([[20.0, 20.0]], np.float32)
    n, steps = 65537, 12
    src = [(8.0 * (1 + k % 4), 8.0 * (1 + k // 4)) for k in range(16)]
    wave = Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0)
    with Context(0) as c:
        c.set_option("on_chip", on_chip)
        m = c.model(vp, vp, 8.0, 8.0, 2)
        few = np.concatenate(c.forward([Shot(m, s, rec) for s in src], wave))
        assert np.abs(few).max() > 0
        out = torch.zeros(n * steps, device="cuda")
        c.forward([Shot(m, src[k % 16], rec) for k in range(n)], wave, out=out)
    got = out.cpu().numpy().reshape(n, steps)
    np.testing.assert_array_equal(got, few.reshape(16, steps)[np.arange(n) % 16])
