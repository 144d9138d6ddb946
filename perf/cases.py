"""The work that programs have this framework do, as cases to be timed.

A case is one call (or one training step) through the public entry points: a
forward survey (``Context.forward``, batched or shot after shot, one grid or
several), the one-call host seam (``modelling_module``), the allocation-free
entry (``s2d_forward_static``), an FWI gradient (``Context.gradient``) and an
inversion step through ``torch.autograd`` (``modelled_seismograms``).

``listed()`` gives fixed sizes, ``draw(rng)`` more of the same ranges.
``exact`` restates the scheme in plain 64-bit torch: the FP64 wavefields of
src/src_cpu/cpumodelling.cpp:115-156, the 8th-order operator and the free
surface of include/seis2d.h, and gradients by torch's own differentiation.
"""
import ctypes as C
import math

import numpy as np
import torch

from seis2d_b200 import Context, Shot, Wave, derive_steps, modelling_module
from seis2d_b200 import _lib as L
from seis2d_b200.autograd import modelled_seismograms


# ------------------------------------------------------------------- the cases

def _case(name, kind, grids, nb, h, dt, f, steps, shots, **more):
    """kind: forward | module | static | gradient | autograd.  grids: "NXxNZ"
    model sizes, several separated by commas; shots: per grid.  order: FD
    order; surface: free surface; every: FD steps per recorded sample; plain:
    shot after shot."""
    c = dict(kind=kind, grids=grids, nb=nb, h=h, dt=dt, f=f, steps=steps, shots=shots, order=4, surface=False,
             every=1, plain=False)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a quick look at a small model: one shot, a few hundred short steps
        _case("small shot 201x101", "forward", "201x101", 32, 10.0, 0.001, 20.0, 500, 1),
        # the same kind of call from a program that may not allocate device memory
        _case("static shot 301x241", "static", "301x241", 32, 10.0, 0.001, 20.0, 400, 1, every=2),
        # the reference's seam in one call on host arrays (context, model, shots, traces), odd sizes, free surface
        _case("module host 487x263", "module", "487x263", 32, 8.0, 0.0008, 25.0, 300, 3, surface=True, every=2),
        # the shipped two-layer card's scale: one shot on 1000 x 1000
        _case("single shot 1000x1000", "forward", "1000x1000", 40, 10.0, 0.001, 15.0, 1000, 1),
        # the salt card's grid: one shot on 3201 x 1201
        _case("salt shot 3201x1201", "forward", "3201x1201", 50, 7.62, 0.0006, 20.0, 800, 1),
        # a survey over models of uneven size in one batch
        _case("uneven batch", "forward", "601x301,1201x601,2401x801", 50, 10.0, 0.0008, 15.0, 250, 6),
        # a large survey: shots of one 5000 x 5000 model in one batch
        _case("large batch 5000x5000", "forward", "5000x5000", 60, 5.0, 0.0005, 20.0, 300, 8),
        # the reference's order, shot after shot
        _case("shot after shot 1201x401", "forward", "1201x401", 50, 10.0, 0.001, 10.0, 400, 8, plain=True),
        # the 8th-order operator on the large model
        _case("order 8 batch 5000x5000", "forward", "5000x5000", 60, 5.0, 0.0005, 20.0, 200, 4, order=8),
        # FWI gradient with a checkpoint every 100 steps, L2 misfit
        _case("gradient 1201x401", "gradient", "1201x401", 50, 10.0, 0.001, 10.0, 600, 8, segment=100, misfit=True),
        # the same of the 8th-order scheme, from an adjoint source
        _case("gradient order 8 1201x401", "gradient", "1201x401", 50, 10.0, 0.001, 10.0, 300, 4, order=8,
              segment=100, misfit=False),
        # one inversion step through torch.autograd: traces, loss, gradients of vp and rho
        _case("autograd step 601x301", "autograd", "601x301", 50, 10.0, 0.001, 10.0, 400, 4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """FLOPs of a case, gradients weighted as the several passes they are."""
    return work(c)["flops"]


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "forward", "module", "static", "gradient", "autograd"])
    order = 8 if kind in ("forward", "gradient", "module") and rng.random() < 0.25 else 4
    nb = rng.choice([20, 32, 40, 50, 60])
    h = rng.choice([4.0, 5.0, 7.62, 10.0])
    dt = round(h * rng.uniform(0.6, 1.0) * 1e-4, 7)
    f = round(rng.uniform(0.8, 1.6) * 150.0 / h, 1)
    every = rng.choice([1, 1, 2, 4])
    more = dict(order=order, every=every, surface=kind in ("forward", "module", "gradient") and rng.random() < 0.2)
    top = _cost(listed()[6])
    while True:
        if kind == "static":
            grids, shots = "%dx%d" % (_log(rng, 100, 560), _log(rng, 80, 560)), 1
            steps = _log(rng, 150, 600)
        elif kind in ("gradient", "autograd"):
            grids, shots = "%dx%d" % (_log(rng, 150, 1400), _log(rng, 100, 700)), rng.randint(1, 8)
            steps = _log(rng, 150, 600)
            if kind == "gradient":
                more.update(segment=rng.choice([50, 100, 128]), misfit=rng.random() < 0.5)
        elif kind == "module":
            grids, shots = "%dx%d" % (_log(rng, 120, 1200), _log(rng, 80, 700)), rng.randint(1, 6)
            steps = _log(rng, 150, 600)
        else:
            n = 1 if rng.random() < 0.75 else rng.randint(2, 3)
            grids = ",".join("%dx%d" % (_log(rng, 120, 5000), _log(rng, 80, 5000)) for _ in range(n))
            shots = _log(rng, 1, 16)
            steps = _log(rng, 150, 1200)
            more.update(plain=rng.random() < 0.15)
        c = _case(None, kind, grids, nb, h, dt, f, steps, shots, **more)
        limit = top / 8 if kind in ("gradient", "autograd") else top
        cells = sum((nx + 2 * nb) * (nz + 2 * nb) for nx, nz in _grids(c)) * shots
        if _cost(c) <= limit and cells <= 2.2e8:
            return c


def _grids(c):
    return [tuple(int(v) for v in g.split("x")) for g in c["grids"].split(",")]


def _wave(c):
    # half a step short of the last step, so that no rounding of the quotient adds one
    return Wave((c["steps"] - 0.5) * c["dt"], c["dt"], c["every"] * c["dt"] * (1 + 1e-6), c["f"])


def _times(c):
    """fd_nt, real_nt, dt_factor, nts as the reference derives them
    (src/src_cpu/cpumodelling.cpp:168-188), in its float arithmetic."""
    w, q = _wave(c), np.float32
    T, dt, rdt, f = q(w.rec_len), q(w.fd_dt), q(w.real_dt), q(w.dom_freq)
    fd_nt, real_nt, every = int(np.ceil(T / dt)), int(np.ceil(T / rdt)), int(rdt / dt)
    td = float(np.sqrt(q(6.0))) / (3.141592654 * float(f))
    return fd_nt, real_nt, every, min(int(5.0 * td / float(dt)) + 1, fd_nt)


def work(c):
    """Models read and traces (or gradients) written once; the arithmetic of
    the scheme per padded cell and step: four derivatives (5 operations each, 11
    at order 8), 15 for the updates; the adjoint's transposes cost as much
    again and the imaging 12."""
    fd_nt, real_nt, _, _ = _times(c)
    per = 15 + 4 * (5 if c["order"] == 4 else 11)
    grad = c["kind"] in ("gradient", "autograd")
    nbytes = flops = 0.0
    for nx, nz in _grids(c):
        cells = (nx + 2 * c["nb"]) * (nz + 2 * c["nb"])
        traces = 4.0 * c["shots"] * nx * real_nt
        nbytes += (8.0 if not grad else 16.0) * nx * nz + traces * (2 if grad else 1)
        flops += float(cells) * fd_nt * c["shots"] * (2 * per + 12 if grad else per)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------- inputs of a case

def _model(nx, nz, gen, dev):
    """vp, rho [nx][nz]: a water layer, a gradient with layers and smooth
    lateral variation, densities after Gardner."""
    z = torch.linspace(0, 1, nz, device=dev)
    x = torch.linspace(0, 1, nx, device=dev)[:, None]
    r = torch.rand(16, generator=gen, device=dev)
    vp = 1600.0 + 1500.0 * z + 200.0 * torch.sin(6.3 * (x * (1 + 2 * r[0]) + r[1])) * z
    for k in range(4):
        dip = 0.1 * (r[2 + k] - 0.5) * (x - 0.5)
        vp = vp + torch.where(z > 0.15 + 0.2 * k + 0.1 * r[6 + k] + dip, 350.0 * r[10 + k], 0.0)
    vp = torch.where(z < 0.05, torch.full_like(vp, 1500.0), vp).clamp(max=4500.0)
    rho = 310.0 * vp.double().pow(0.25)
    return vp.float().contiguous(), rho.float().contiguous()


def _geometry(nx, nz, c, gen, dev):
    """Sources along the surface with some jitter, a receiver at every surface cell."""
    h = np.float32(c["h"])
    jit = torch.rand(c["shots"], generator=gen, device=dev).cpu().numpy()
    iz = 3 if c["surface"] else 2
    rec = np.stack([(np.arange(nx, dtype=np.float32) + np.float32(0.25)) * h,
                    np.full(nx, (iz + 0.25) * h, np.float32)], 1).astype(np.float32)
    src = []
    for s in range(c["shots"]):
        ix = min(nx - 1, int((s + 0.25 + 0.5 * float(jit[s])) * nx / c["shots"]))
        src.append((float(np.float32(ix + 0.25) * h), float(np.float32(iz + 0.25) * h)))
    return src, rec


def _inputs(c, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    got = []
    for nx, nz in _grids(c):
        vp, rho = _model(nx, nz, gen, dev)
        got.append((vp, rho, *_geometry(nx, nz, c, gen, dev)))
    return got


def _data(c, seed, inputs):
    """Observed traces (or an adjoint source) of each shot, [shots][nrec][real_nt]:
    Ricker arrivals along hyperbolas, in the amplitudes of modelled pressure."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed) + 7919)
    _, real_nt, every, _ = _times(c)
    t = torch.arange(real_nt, device=dev) * (every * c["dt"])
    out = []
    for _, _, src, rec in inputs:
        x = torch.from_numpy(rec[:, 0].copy()).to(dev)
        for sx, _ in src:
            r = torch.rand(9, generator=gen, device=dev)
            d = torch.zeros(rec.shape[0], real_nt, device=dev)
            for k in range(3):
                t0 = t[-1] * (0.15 + 0.25 * k + 0.2 * r[k])
                arr = torch.sqrt(t0 * t0 + ((x - sx) / (1600.0 + 900.0 * r[3 + k])) ** 2)
                a = (math.pi * c["f"] * (t[None, :] - arr[:, None])) ** 2
                d += 2e4 * (0.3 + r[6 + k]) * (1 - 2 * a) * torch.exp(-a)
            out.append(d)
    return torch.cat([d.reshape(-1) for d in out])


# --------------------------------------------------------------- what is timed

def prepare(case, seed):
    c = dict(case)
    ins = _inputs(c, seed)
    wave = _wave(c)
    state = {"kind": c["kind"], "wave": wave, "case": c}
    if c["kind"] == "module":
        vp, rho, src, rec = ins[0]
        state.update(vp=vp.cpu().numpy(), rho=rho.cpu().numpy(), geometry=[(s, rec) for s in src])
        return state
    _, real_nt, _, _ = _times(c)
    if c["kind"] == "static":
        vp, rho, src, rec = ins[0]
        crec = np.ascontiguousarray(rec)
        shot = L.Shot(0, L.Coord(*src[0]), crec.shape[0], crec.ctypes.data_as(C.POINTER(L.Coord)))
        state.update(vp=vp, rho=rho, rec=crec, shot=shot, cwave=wave.c(), err=C.create_string_buffer(256),
                     out=torch.zeros(crec.shape[0], real_nt, device="cuda"))
        return state
    if c["kind"] == "autograd":
        vp, rho, src, rec = ins[0]
        state.update(vp=vp.requires_grad_(), rho=rho.requires_grad_(), geometry=[(s, rec) for s in src],
                     data=_data(c, seed, ins))
        return state
    ctx = Context(torch.cuda.current_device())
    shots, samples = [], 0
    for vp, rho, src, rec in ins:
        m = ctx.model(vp, rho, c["h"], c["h"], c["nb"], free_surface=c["surface"], fd_order=c["order"])
        shots += [Shot(m, s, rec) for s in src]
        samples += len(src) * rec.shape[0] * real_nt
    state.update(ctx=ctx, shots=shots)
    if c["kind"] == "gradient":
        ctx.set_option("grad_segment", c["segment"])
        state.update(data=_data(c, seed, ins), grad_vp=torch.zeros_like(ins[0][0]),
                     grad_rho=torch.zeros_like(ins[0][1]))
    else:
        state["out"] = torch.zeros(samples, device="cuda")
    return state


def run(state):
    c, wave, kind = state["case"], state["wave"], state["kind"]
    if kind == "forward":
        return state["ctx"].forward(state["shots"], wave, out=state["out"], plain=c["plain"])
    if kind == "module":
        return modelling_module(state["vp"], state["rho"], c["h"], c["h"], wave, state["geometry"], c["nb"],
                                free_surface=c["surface"], fd_order=c["order"])
    if kind == "static":
        nx, nz = state["vp"].shape
        rc = L.lib().s2d_forward_static(
            torch.cuda.current_device(), nx, nz, c["h"], c["h"], c["nb"], state["vp"].data_ptr(),
            state["rho"].data_ptr(), C.byref(state["cwave"]), C.byref(state["shot"]), state["out"].data_ptr(),
            L.S2D_STATIC_MODEL_DEVICE | L.S2D_STATIC_SEIS_DEVICE, torch.cuda.current_stream().cuda_stream,
            state["err"], 256)
        if rc:
            raise RuntimeError(state["err"].value.decode())
        return state["out"]
    if kind == "gradient":
        g = state["ctx"].gradient(state["shots"], wave, state["data"], misfit=c["misfit"],
                                  grad_vp=state["grad_vp"], grad_rho=state["grad_rho"])
        out = {"vp": g.grad_vp, "rho": g.grad_rho, "wavelet": g.grad_wavelet}
        if c["misfit"]:
            out["misfit"] = float(g.misfit)
        return out
    vp, rho = state["vp"], state["rho"]
    vp.grad = rho.grad = None
    seis = modelled_seismograms(vp, rho, state["geometry"], wave, c["h"], c["h"], c["nb"])
    loss = 0.5 * ((seis - state["data"]) ** 2).sum()
    loss.backward()
    return {"seis": seis.detach(), "vp": vp.grad, "rho": rho.grad}


# ------------------------------------------------------------ the 64-bit answer

_C4 = (1.125, float(np.float32(-1.0) / np.float32(24.0)))
_C8 = tuple(float(np.float32(a / b)) for a, b in ((1225, 1024), (-245, 3072), (49, 5120), (-5, 7168)))


def _taps(fl, n, dim, lo, hi, coefs):
    """sum_k c_k (f[i+k-1] - f[i-k]) for k = 1..len(coefs), rows i of [lo, hi) (fl: f.narrow)."""
    out = None
    for k, ck in enumerate(coefs):
        d = fl(lo + k, hi + k) - fl(lo - 1 - k, hi - 1 - k)
        out = d * ck if out is None else out.add_(d, alpha=ck) if not d.requires_grad else out + ck * d
    return out


def _dminus(f, dim, order):
    """D- along `dim`: rows [2, n-2] by the 4-tap pair ([4, n-4] by the 8 taps
    at order 8), rows 1 and n-1 the plain difference, row 0 zero."""
    n = f.shape[dim]
    fl = lambda a, b: f.narrow(dim, a, b - a)  # noqa: E731
    zero = torch.zeros_like(fl(0, 1))
    one = fl(1, 2) - fl(0, 1)
    last = fl(n - 1, n) - fl(n - 2, n - 1)
    if order == 4 or n < 9:
        mid = [_taps(fl, n, dim, 2, n - 1, _C4)]
    else:
        mid = [_taps(fl, n, dim, 2, 4, _C4), _taps(fl, n, dim, 4, n - 3, _C8), _taps(fl, n, dim, n - 3, n - 1, _C4)]
    return torch.cat([zero, one, *mid, last], dim)


def _dplus(f, dim, order):
    """D+ along `dim`: D- one row further on, the last row zero: 4 taps on
    [1, n-3], 8 on [3, n-5], plain differences on rows 0 and n-2."""
    n = f.shape[dim]
    return torch.cat([_dminus(f, dim, order).narrow(dim, 1, n - 1), torch.zeros_like(f.narrow(dim, 0, 1))], dim)


def _sponge(nb, n, half):
    """The Gaussian tapers of cpu_modelling_kernels.cpp:123-199, which the
    reference holds in float: damping d and sqrt-like d1 per padded row, at
    integer or half nodes."""
    q = np.float32
    i = np.arange(nb, dtype=np.float32)
    t = q(0.05) * (i + q(0.5)) if half else q(0.05) * (i + q(1.0) - q(1.0))
    d, d1 = np.exp(-(t * t)).astype(q), np.exp(-0.5 * (t * t).astype(np.float64)).astype(q)
    one = np.ones(n + (1 if half else 0), q)
    k = nb - 1 if half else nb
    return [np.concatenate([v[:k][::-1], one, v]).astype(np.float64) for v in (d, d1)]


def _pad(v, nb):
    """Edge replication into the sponge (cpumodelling.cpp:39-60)."""
    nx, nz = v.shape
    ix = (torch.arange(nx + 2 * nb, device=v.device) - nb).clamp(0, nx - 1)
    iz = (torch.arange(nz + 2 * nb, device=v.device) - nb).clamp(0, nz - 1)
    return v[ix][:, iz]


class _Scheme:
    """The scheme on one model in 64 bits: all shots of the model at once."""

    def __init__(self, c, vp, rho, src, rec):
        self.c, nb, h = c, c["nb"], np.float32(c["h"])
        self.fd_nt, self.real_nt, self.every, self.nts = _times(c)
        dev = vp.device
        nx, nz = vp.shape
        self.vp, self.rho = vp, rho
        kap, b = _pad(vp * vp * rho, nb), _pad(1.0 / rho, nb)
        nnx, nnz = kap.shape
        if c["surface"]:
            kap = kap * (torch.arange(nnz, device=dev) > nb)
        bz = torch.cat([0.5 * (b[:, 1:] + b[:, :-1]), torch.zeros_like(b[:, :1])], 1)
        bx = torch.cat([0.5 * (b[1:] + b[:-1]), bz[-2:-1]], 0)
        dtd = float(np.float32(c["dt"]) * (np.float32(1.0) / h))
        tab = lambda n, half: [torch.from_numpy(v).to(dev) for v in _sponge(nb, n, half)]  # noqa: E731
        (ax, ax1), (az, az1), (hx, hx1), (hz, hz1) = tab(nx, False), tab(nz, False), tab(nx, True), tab(nz, True)
        self.damp = ax[:, None], az[None, :], hx[:, None], hz[None, :]
        self.kx, self.kz = dtd * ax1[:, None] * kap, dtd * az1[None, :] * kap
        self.lx, self.lz = dtd * hx1[:, None] * bx, dtd * hz1[None, :] * bz
        inv = np.float32(1.0) / h
        cell = lambda p: int(np.float32(p) * inv) + nb  # noqa: E731
        self.src = torch.tensor([[cell(x), cell(z)] for x, z in src], device=dev)
        self.rec = torch.tensor([[cell(x), cell(z)] for x, z in rec], device=dev)
        # injected amplitude per unit of w[kt]: dt kappa_src / (dx dz)
        self.amp = float(np.float32(c["dt"])) / float(h * h) * kap[self.src[:, 0], self.src[:, 1]]
        self.shape = (len(src), nnx, nnz)

    def wavelet(self, dev):
        q, f = np.float32, float(np.float32(self.c["f"]))
        t = (np.arange(self.nts, dtype=np.float32) * q(self.c["dt"])).astype(np.float64)
        a2 = (3.141592654 * f * (t - 1.5 * math.sqrt(6.0) / (3.141592654 * f))) ** 2
        w = np.zeros(self.fd_nt)
        w[: self.nts] = (1.0 - 2.0 * a2) * np.exp(-a2)
        return torch.from_numpy(w).to(dev)

    def step(self, st, w, params):
        """One FD step; `w`: the source sample per shot, or None after the wavelet."""
        px, pz, vx, vz = st
        kx, kz, lx, lz, amp = params
        ax, az, hx, hz = self.damp
        order = self.c["order"]
        px = ax * px + kx * _dminus(vx, 1, order)
        pz = az * pz + kz * _dminus(vz, 2, order)
        if w is not None:
            s = torch.arange(len(amp), device=amp.device)
            px = px.index_put((s, self.src[:, 0], self.src[:, 1]), w * amp, accumulate=True)
        p = px + pz
        vx = hx * vx + lx * _dplus(p, 1, order)
        vz = hz * vz + lz * _dplus(p, 2, order)
        return (px, pz, vx, vz), p

    def advance(self, k0, k1, w, params, *st):
        """Steps [k0, k1): the state after them and the samples recorded."""
        got = []
        for kt in range(k0, k1):
            st, p = self.step(st, w[:, kt] if kt <= self.nts else None, params)
            if (kt + 1) % self.every == 0 and (kt + 1) // self.every <= self.real_nt:
                got.append(p[:, self.rec[:, 0], self.rec[:, 1]])
        return (*st, torch.stack(got, 2) if got else st[0].new_zeros(self.shape[0], len(self.rec), 0))

    def traces(self, w, segment):
        """[shots][nrec][real_nt]; differentiable with recomputation per segment."""
        from torch.utils.checkpoint import checkpoint
        params = (self.kx, self.kz, self.lx, self.lz, self.amp)
        st = tuple(torch.zeros(self.shape, dtype=torch.float64, device=self.kx.device) for _ in range(4))
        parts = []
        for k0 in range(0, self.fd_nt, segment):
            k1 = min(self.fd_nt, k0 + segment)
            if torch.is_grad_enabled():
                *st, got = checkpoint(self.advance, k0, k1, w, params, *st, use_reentrant=False)
            else:
                *st, got = self.advance(k0, k1, w, params, *st)
            parts.append(got)
        out = torch.cat(parts, 2)
        left = self.real_nt - out.shape[2]
        return torch.cat([out, out.new_zeros(*out.shape[:2], left)], 2) if left else out


def exact(case, seed):
    c = dict(case)
    ins = _inputs(c, seed)
    if c["kind"] not in ("gradient", "autograd"):
        shots = []
        with torch.no_grad():
            for vp, rho, src, rec in ins:
                m = _Scheme(c, vp.double(), rho.double(), src, rec)
                w = m.wavelet(vp.device).expand(len(src), -1)
                shots += list(m.traces(w, m.fd_nt))
                del m
        if c["kind"] == "module":
            return [t.cpu().numpy() for t in shots]
        return shots[0] if c["kind"] == "static" else torch.cat([t.reshape(-1) for t in shots])
    vp, rho, src, rec = ins[0]
    vp, rho = vp.double().requires_grad_(), rho.double().requires_grad_()
    m = _Scheme(c, vp, rho, src, rec)
    w = m.wavelet(vp.device).repeat(len(src), 1).requires_grad_()
    seis = m.traces(w, 20).reshape(-1)
    d = _data(c, seed, ins).double()
    if c["kind"] == "gradient" and not c["misfit"]:
        (seis * d).sum().backward()
    else:
        loss = 0.5 * ((seis - d) ** 2).sum()
        loss.backward()
    if c["kind"] == "autograd":
        return {"seis": seis.detach(), "vp": vp.grad, "rho": rho.grad}
    out = {"vp": vp.grad, "rho": rho.grad, "wavelet": w.grad.cpu().numpy()}
    if c["misfit"]:
        out["misfit"] = float(loss)
    return out
