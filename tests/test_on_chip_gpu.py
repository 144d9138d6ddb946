"""The on-chip time loop (whole runs in one cooperative launch, state in
registers and shared memory) against the per-step kernels: the same bits, at
the edges of its tiles, for every block shape it is built for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (warps, columns per warp): a tile owns warps * columns - 6 columns and 120 rows
SHAPES = [(4, 3), (4, 4), (8, 3), (8, 4), (8, 5), (8, 6), (8, 7), (8, 8), (8, 9), (8, 10)]


def _run(nx, nz, nb, shots, steps, on_chip, shape=0, every=1, surface=False, plain=False, rec=None, pieces=(), h=8.0):
    from seis2d_b200 import Context, Shot, Wave
    rng = np.random.default_rng(nx * 1000 + nz)
    vp = (1700.0 + 1200.0 * rng.random((nx, nz))).astype(np.float32)
    rho = (1000.0 + 900.0 * rng.random((nx, nz))).astype(np.float32)
    if rec is None:
        rec = np.stack([(np.arange(nx) + 0.25) * h, np.full(nx, (min(3, nz - 1) + 0.25) * h)], 1).astype(np.float32)
    with Context(0) as c:
        c.set_option("on_chip", int(on_chip))
        c.set_option("on_chip_shape", shape)
        m = c.model(vp, rho, h, h, nb, free_surface=surface)
        src = [((k + 0.5) * nx / shots * h, (0.25 + (k * 7) % nz) * h) for k in range(shots)]
        sh = [Shot(m, s, rec) for s in src]
        wave = Wave((steps - 0.5) * 0.001, 0.001, every * 0.001 * 1.000001, 25.0)
        if pieces:
            out = np.full(shots * len(rec) * -(-steps // every), np.nan, np.float32)
            k = 0
            for n in (*pieces, 0):
                c.forward(sh, wave, kt_begin=k, kt_count=n, out=out, plain=plain)
                k += n
        else:
            out = np.concatenate([o.ravel() for o in c.forward(sh, wave, plain=plain)])
        return out, c.last_stats


def _same(*args, **kw):
    a, sa = _run(*args, on_chip=True, **kw)
    kw.pop("shape", None)
    b, sb = _run(*args, on_chip=False, **kw)
    assert np.abs(b).max() > 0
    np.testing.assert_array_equal(a, b)
    return sa, sb


@pytest.mark.parametrize("nw,c", SHAPES)
def test_every_block_shape_at_its_tile_edges(nw, c):
    """Two tiles of columns (one column short of, at and past the edge) and two
    strips (one row past the first): sources and receivers beside the seams."""
    own = nw * c - 6
    for nnx, nnz in ((2 * own, 121), (2 * own + 1, 120), (2 * own - 1, 243)):
        nb = 4
        sa, _ = _same(nnx - 2 * nb, nnz - 2 * nb, nb, 2, 60, shape=nw * 100 + c)
        assert sa.kernel_launches <= 2  # the whole run in one launch (one per wave of shots)


@pytest.mark.parametrize("case", [
    dict(nx=1, nz=1, nb=2, shots=1, steps=40),                       # smaller than the halo
    dict(nx=37, nz=29, nb=32, shots=1, steps=130),                   # sponge wider than the model
    dict(nx=201, nz=101, nb=32, shots=1, steps=161, every=4),
    dict(nx=300, nz=260, nb=20, shots=5, steps=120, surface=True),   # several waves of shots
    dict(nx=140, nz=380, nb=40, shots=3, steps=120, plain=True),
    dict(nx=90, nz=70, nb=12, shots=13, steps=125, every=2, pieces=(7, 9, 8, 1, 40)),
])
def test_options_and_sizes_keep_the_bits(case):
    case = dict(case)
    args = [case.pop(k) for k in ("nx", "nz", "nb", "shots", "steps")]
    _same(*args, **case)


@pytest.mark.parametrize("kind", ["none", "scattered", "stacked", "sponge"])
def test_receiver_layouts(kind):
    rng = np.random.default_rng(3)
    nx, nz, nb, h = 150, 260, 16, 8.0
    if kind == "none":
        # a run without receivers leaves the state alone: continue it with some
        rec = np.zeros((0, 2), np.float32)
        a, _ = _run(nx, nz, nb, 1, 40, on_chip=True, rec=rec)
        assert a.size == 0
        return
    if kind == "scattered":
        rec = np.stack([rng.random(500) * (nx - 1) * h, rng.random(500) * (nz - 1) * h], 1)
    elif kind == "stacked":  # several per column and per cell, on two rows
        rec = np.stack([np.repeat(np.arange(40) * 3.5 * h, 3), np.tile([40.2, 40.3, 900.0], 40)], 1)
    else:
        rec = np.stack([(rng.random(200) * (nx + 2 * nb - 2) - nb) * h, (rng.random(200) * (nz + 2 * nb - 2) - nb) * h], 1)
    _same(nx, nz, nb, 2, 120, rec=rec.astype(np.float32), every=2)


def test_a_wait_that_runs_out_is_an_error_and_the_context_survives():
    """Block 0 does not publish step 5: its neighbours' waits run out of their
    bound, the call reports a timeout and the next one is right."""
    from seis2d_b200 import Context, Shot, Wave
    from seis2d_b200._lib import Seis2dError, S2D_ERR_TIMEOUT
    vp = np.full((120, 90), 2000.0, np.float32)
    rec = np.stack([np.arange(120) * 8.0, np.full(120, 24.0)], 1).astype(np.float32)
    wave = Wave(0.0595, 0.001, 0.001001, 25.0)
    with Context(0) as c:
        m = c.model(vp, vp, 8.0, 8.0, 20)
        shot = [Shot(m, (400.0, 24.0), rec)]
        good = c.forward(shot, wave)[0]
        c.set_option("inject_wait_fault", 5)
        c.set_option("spin_limit", 256)
        with pytest.raises(Seis2dError) as e:
            c.forward(shot, wave)
        assert e.value.code == S2D_ERR_TIMEOUT
        c.set_option("inject_wait_fault", -1)
        c.set_option("spin_limit", 1 << 20)
        np.testing.assert_array_equal(c.forward(shot, wave)[0], good)


def test_uneven_batch_mixes_both_loops():
    """Small models on chip, a large one by the per-step kernels, in one call
    and in continuations."""
    from seis2d_b200 import Context, Shot, Wave
    outs = []
    for on in (1, 0):
        with Context(0) as c:
            c.set_option("on_chip", on)
            shots = []
            for nx, nz in ((150, 100), (2300, 700), (260, 330)):
                vp = np.linspace(1600.0, 3000.0, nx * nz, dtype=np.float32).reshape(nx, nz)
                m = c.model(vp, 0.5 * vp, 8.0, 8.0, 24)
                rec = np.stack([np.arange(0, nx, 2) * 8.0, np.full(len(range(0, nx, 2)), 16.0)], 1).astype(np.float32)
                shots += [Shot(m, ((k + 0.5) * nx / 2 * 8.0, 16.0), rec) for k in range(2)]
            wave = Wave(0.1695, 0.001, 0.001001, 25.0)
            whole = np.concatenate([o.ravel() for o in c.forward(shots, wave)])
            out = np.full(whole.size, np.nan, np.float32)
            k = 0
            for n in (9, 33, 0):
                c.forward(shots, wave, kt_begin=k, kt_count=n, out=out)
                k += n
            np.testing.assert_array_equal(out, whole)
            outs.append(whole)
    np.testing.assert_array_equal(outs[0], outs[1])
