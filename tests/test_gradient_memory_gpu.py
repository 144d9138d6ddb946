"""The gradient's choice of its checkpoint interval when device memory is short
and much of what the context holds cannot go back to the driver (pooled buffers
in chunks that models use); and calls after one that found no memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0
NX = NZ = 361
NB = 20


def _job(c, n, steps, seed=0):
    from seis2d_b200 import Shot, Wave
    vp = np.linspace(1600.0, 3000.0, NX * NZ, dtype=np.float32).reshape(NX, NZ)
    m = c.model(vp, 0.5 * vp, H, H, NB)
    rec = np.stack([np.arange(0, NX, 5) * H, np.full(-(-NX // 5), 16.0)], 1).astype(np.float32)
    return [Shot(m, ((k + 0.5) * NX / n * H, 16.0), rec) for k in range(n)], Wave((steps - 0.5) * 0.001, 0.001, 0.001001, 25.0)


def test_short_memory():
    import torch
    from seis2d_b200 import Context
    from seis2d_b200._lib import S2D_ERR_NOMEM, Seis2dError
    rng = np.random.default_rng(2)
    n, steps = 4, 300
    with Context(0) as c:
        shots, wave = _job(c, n, steps)
        adj = rng.standard_normal((n, shots[0].rec.shape[0], steps)).astype(np.float32)
        ref = [np.asarray(v) for v in (lambda g: (g.grad_vp, g.grad_rho))(c.gradient(shots, wave, adj))]
        whole = c.last_stats.grad_segment
    assert whole == steps
    with Context(0) as c:
        # 300 shots' states, four of 6.8 MB to a chunk of 32 MB, then a model in every chunk's gap:
        # 2 GB that count as free and stay with the context
        shots, wave = _job(c, 300, steps)
        out = torch.zeros(300 * shots[0].rec.shape[0] * steps, device="cuda")
        c.forward(shots, wave, kt_count=2, out=out)
        keep = [_job(c, 1, steps)[0] for _ in range(80)]
        del out
        # 1 GB left: products of all 300 steps would take 4.1 GB
        shots, wave = _job(c, n, steps)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        left = 1 << 30
        hog = torch.empty(free - left, dtype=torch.uint8, device="cuda")
        try:
            g = c.gradient(shots, wave, adj)
            seg = c.last_stats.grad_segment
            got = [np.asarray(g.grad_vp), np.asarray(g.grad_rho)]
            # a call that cannot fit is refused, and the next one is right
            many, _ = _job(c, 300, steps)
            with pytest.raises(Seis2dError) as e:
                c.gradient(many, wave, rng.standard_normal((300, many[0].rec.shape[0], steps)).astype(np.float32))
            assert e.value.code == S2D_ERR_NOMEM
            again = c.gradient(shots, wave, adj)
        finally:
            del hog
            torch.cuda.empty_cache()
        assert keep
    assert seg < steps
    # shots add to the gradient in any order: n * steps terms, each sum rounded to 2^-24
    for a, b, r in zip(got, (again.grad_vp, again.grad_rho), ref):
        for v in (a, np.asarray(b)):
            assert np.linalg.norm(v.astype(np.float64) - r) <= n * steps * 2.0 ** -24 * np.linalg.norm(r)


def test_pooled_memory_goes_back():
    """The states of a batch of many shots, between models that stay, make room
    for a batch of another size."""
    import torch
    from seis2d_b200 import Context, Shot, Wave
    with Context(0) as c:
        shots, wave = _job(c, 300, 20)
        c.forward(shots, wave, kt_count=2)
        keep = [_job(c, 1, 20)[0] for _ in range(80)]
        vp = np.full((2400, 2400), 2000.0, np.float32)
        m = c.model(vp, vp, H, H, NB)
        big = [Shot(m, ((k + 1) * 300 * H, 100 * H), np.array([[(k + 1) * 300 * H, 110 * H]], np.float32)) for k in range(7)]
        ref = c.forward(big[:1], wave)[0]
        c.forward(shots, wave, kt_count=2)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (256 << 20), dtype=torch.uint8, device="cuda")
        try:
            got = c.forward(big, wave)  # 7 states of 200 MB; 2 GB in the pool
        finally:
            del hog
            torch.cuda.empty_cache()
        assert keep and np.abs(ref).max() > 0
    np.testing.assert_array_equal(got[0], ref)
