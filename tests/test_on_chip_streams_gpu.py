"""The on-chip loop beside other work on the GPU: kernels of another stream that
hold SMs only delay it, and contexts of two threads run it side by side."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 8.0
NX, NZ, NB, STEPS = 700, 500, 24, 160
WAVE = ((STEPS - 0.5) * 0.001, 0.001, 0.001001, 25.0)


def _inputs():
    vp = np.linspace(1600.0, 3000.0, NX * NZ, dtype=np.float32).reshape(NX, NZ)
    rec = np.stack([np.arange(0, NX, 3) * H, np.full(-(-NX // 3), 24.0)], 1).astype(np.float32)
    return vp, (0.5 * vp).astype(np.float32), (NX // 2 * H, 24.0), rec


class _Busy:
    """Matrix products of whole-SM blocks queued on a stream of their own."""

    def __init__(self):
        import torch
        self.stream = torch.cuda.Stream()
        self.a = torch.randn(4096, 4096, device="cuda").bfloat16()
        self.out = torch.empty_like(self.a)
        with torch.cuda.stream(self.stream):
            torch.mm(self.a, self.a, out=self.out)
        torch.cuda.synchronize()

    def queue(self, n):
        import torch
        with torch.cuda.stream(self.stream):
            for _ in range(n):
                torch.mm(self.a, self.a, out=self.out)
        assert not self.stream.query()  # still running when the loop is launched


def test_other_work_delays_a_continuation():
    import torch
    from seis2d_b200 import Context, Shot, Wave
    vp, rho, src, rec = _inputs()
    busy = _Busy()
    with Context(0) as c:
        m = c.model(vp, rho, H, H, NB)
        shot = [Shot(m, src, rec)]
        good = c.forward(shot, Wave(*WAVE))[0]
        assert c.last_stats.kernel_launches == 1  # on chip
        c.set_option("spin_limit", 1 << 12)  # a few ms: a small part of the other stream's work
        for _ in range(3):
            out = torch.zeros(good.size, device="cuda")
            c.forward(shot, Wave(*WAVE), kt_count=10, out=out)
            busy.queue(600)
            c.forward(shot, Wave(*WAVE), kt_begin=10, out=out)
            np.testing.assert_array_equal(out.cpu().numpy().reshape(good.shape), good)
            torch.cuda.synchronize()


def test_other_work_delays_the_static_entry():
    import torch
    from seis2d_b200 import Context, Shot, Wave
    from seis2d_b200 import _lib as L
    nz = 300  # what the static scratch holds
    vp, rho, src, rec = _inputs()
    vp, rho = np.ascontiguousarray(vp[:, :nz]), np.ascontiguousarray(rho[:, :nz])
    with Context(0) as c:
        m = c.model(vp, rho, H, H, NB)
        good = c.forward([Shot(m, src, rec)], Wave(*WAVE))[0]
    shot = L.Shot(0, L.Coord(*src), rec.shape[0], rec.ctypes.data_as(C.POINTER(L.Coord)))
    wave, err, busy = L.Wave(*WAVE), C.create_string_buffer(256), _Busy()
    mine = torch.cuda.Stream()
    for _ in range(3):
        out = np.full(good.size, np.nan, np.float32)
        busy.queue(600)
        rc = L.lib().s2d_forward_static(0, NX, nz, H, H, NB, vp.ctypes.data, rho.ctypes.data, C.byref(wave), C.byref(shot),
                                        out.ctypes.data, 0, mine.cuda_stream, err, 256)
        assert rc == 0, err.value
        np.testing.assert_array_equal(out.reshape(good.shape), good)
        torch.cuda.synchronize()


def test_two_threads():
    import torch
    from seis2d_b200 import Context, Shot, Wave
    vp, rho, src, rec = _inputs()
    good, wrong = [], []
    with Context(0) as c:
        good.append(c.forward([Shot(c.model(vp, rho, H, H, NB), src, rec)], Wave(*WAVE))[0])

    def work():
        try:
            with Context(0) as c:
                shot = [Shot(c.model(vp, rho, H, H, NB), src, rec)]
                out = torch.zeros(good[0].size, device="cuda")
                for _ in range(15):
                    out.zero_()
                    torch.cuda.current_stream().synchronize()
                    for k, n in ((0, 20), (20, 40), (60, 30), (90, 0)):
                        c.forward(shot, Wave(*WAVE), kt_begin=k, kt_count=n, out=out)
                    np.testing.assert_array_equal(out.cpu().numpy().reshape(good[0].shape), good[0])
        except BaseException as e:  # noqa: BLE001 - reported by the test
            wrong.append(e)

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
