"""The work that programs have this library do, as timed cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (a context, its inputs, pinned read-back buffers), ``run`` is one pass
through the public entry points and returns what the pass computed.

Kinds of case:

* ``thermal``: a short run from its initial condition.  The jittered thermal is
  written on the device, the model advances ``steps`` steps in one call, and the
  program reads the gridded fields and (``parcels``) the whole parcel state
  back, as at an output time.  The FP64 form's state comes as FP64; the mixed
  form's, whose values are FP32, goes to FP32 tensors on the GPU (its tags, whole
  numbers, to int64).
* ``callbacks``: the five components called one at a time, in the order a MONC
  host calls them, on the plume set-up of the host's own configuration.
* ``restart``: a stored mid-run state is uploaded, advanced and read back;
  parcels split, are mixed away and are added in every step.
* ``interp``: par2grid of four fields and grid2par of six at uniform random
  positions, all results read back.
* ``invert``: vort2vel's inversion alone on a gridded vorticity.
* ``ensemble``: independent thermals of uneven sizes stepped together.
* ``static``: par2grid on device arrays for callers without a context.
"""
import ctypes as C
import math
import os

# an ensemble steps its members on streams of their own: more hardware queues
# than the default 8 (read when the process creates its CUDA context)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import torch  # noqa: E402

import pmpic_b200 as pm  # noqa: E402

LX, LY, LZ = 2 * math.pi, 2 * math.pi, math.pi
# the fields that a step leaves defined (mixing uses the gridded vorticity and buoyancy as scratch)
FIELDS = ["u", "v", "w", "dp", "dq", "dr", "vol"]


def listed():
    return [
        # a solver component without a context of its own, on a small box
        {"name": "static_16x16x12", "kind": "static", "nx": 16, "ny": 16, "nz": 12, "per_cell": 8},
        # the plain plume at its smallest configuration: 32^3, FP64, 20 steps of 0.01
        {"name": "thermal_32_fp64", "kind": "thermal", "nx": 32, "ny": 32, "nz": 32, "precision": "fp64",
         "steps": 20, "dt": 0.01, "parcels": True},
        # an ensemble's member sizes run alone, 50 steps each: a length that is no power of two
        {"name": "thermal_48_mixed", "kind": "thermal", "nx": 48, "ny": 48, "nz": 48, "precision": "mixed",
         "steps": 50, "dt": 0.32 / 48, "parcels": True},
        {"name": "thermal_96_mixed", "kind": "thermal", "nx": 96, "ny": 96, "nz": 96, "precision": "mixed",
         "steps": 50, "dt": 0.32 / 96, "parcels": True},
        # the plain form at a production size
        {"name": "thermal_128_fp64", "kind": "thermal", "nx": 128, "ny": 128, "nz": 128, "precision": "fp64",
         "steps": 20, "dt": 0.0025, "parcels": True},
        # the largest: the mixed form's 256^3 plume.  Its 134 M parcels stay on the device
        # (a program reads them at checkpoints only); the gridded fields are read.
        {"name": "thermal_256_mixed", "kind": "thermal", "nx": 256, "ny": 256, "nz": 256, "precision": "mixed",
         "steps": 20, "dt": 0.0025, "parcels": False},
        # the host's own plume configuration, one output interval (ten steps of 0.1)
        {"name": "callbacks_32_fp64", "kind": "callbacks", "nx": 32, "ny": 32, "nz": 32, "precision": "fp64",
         "steps": 10, "dt": 0.1},
        {"name": "callbacks_64_mixed", "kind": "callbacks", "nx": 64, "ny": 64, "nz": 64, "precision": "mixed",
         "steps": 10, "dt": 0.05},
        # a ragged box with all of the splitting and mixing bookkeeping at work
        {"name": "restart_72x40x50_fp64", "kind": "restart", "nx": 72, "ny": 40, "nz": 50, "precision": "fp64",
         "steps": 5, "dt": 0.01},
        # interpolation alone: 16.8 M parcels at random positions
        {"name": "interp_128_fp64", "kind": "interp", "nx": 128, "ny": 128, "nz": 128, "precision": "fp64"},
        # the inversion alone
        {"name": "invert_256_fp64", "kind": "invert", "nx": 256, "ny": 256, "nz": 256, "precision": "fp64"},
        # eight members of uneven sizes
        {"name": "ensemble_8_mixed", "kind": "ensemble", "sizes": "32,48,64,64,32,96,48,32", "precision": "mixed",
         "steps": 20},
    ]


def _smooth(n):
    for f in (2, 3, 5):
        while n % f == 0:
            n //= f
    return n == 1


def _size(rng, lo, hi):
    """An even length with the factors 2, 3 and 5 alone, spread over the logarithm of the range."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((n for n in range(lo, hi + 1, 2) if _smooth(n)), key=lambda n: abs(n - want))


def draw(rng):
    kind = rng.choice(["thermal", "thermal", "thermal", "callbacks", "restart", "interp", "invert", "ensemble",
                       "static"])
    if kind == "static":
        nx, ny = 2 * rng.randint(4, 12), 2 * rng.randint(4, 12)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": rng.randint(4, 24), "per_cell": rng.randint(1, 8)}
    precision = rng.choice(["fp64", "mixed"])
    if kind == "ensemble":
        sizes = [rng.choice([32, 48, 64, 96]) for _ in range(rng.randint(3, 8))]
        return {"kind": kind, "sizes": ",".join(map(str, sizes)), "precision": precision,
                "steps": rng.randint(5, 25)}
    if kind == "invert":
        return {"kind": kind, "nx": _size(rng, 32, 256), "ny": _size(rng, 32, 256), "nz": rng.randint(32, 256),
                "precision": precision}
    # cells near cubic in the box, the number of levels any (odd ones too)
    nx = _size(rng, 24, 160 if kind in ("thermal", "interp") else 80)
    ny = max(16, _size(rng, 16, nx if nx > 16 else 18)) if rng.random() < 0.5 else nx
    nz = rng.randint(max(9, nx // 3), nx)
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision}
    if kind == "thermal":
        case.update(steps=rng.randint(10, 50), dt=0.32 / max(nx, ny, nz), parcels=True)
    elif kind == "callbacks":
        case.update(steps=rng.randint(4, 10), dt=0.05)
    elif kind == "restart":
        case.update(steps=rng.randint(2, 5), dt=0.01)
    return case


# ---- reading results back ------------------------------------------------------
class Readback:
    """Pinned host buffers of one context's results, filled through the C ABI."""

    def __init__(self, ctx, cap=0, fields=(), props=()):
        self.ctx, self.cap, self.fields, self.props = ctx, cap, list(fields), list(props)
        # parcels fill the first n slots; the rest stays zero
        self.out = torch.zeros(11, cap, dtype=torch.float64, pin_memory=True) if cap else None
        self.grid = torch.empty(len(self.fields), ctx.nz + 1, ctx.ny, ctx.nx, dtype=torch.float64, pin_memory=True)
        self.prop = torch.empty(len(self.props), ctx.max_parcels, dtype=torch.float64, pin_memory=True)

    @staticmethod
    def _p(t):
        return C.cast(t.data_ptr(), C.POINTER(C.c_double))

    def _form(self, t):
        """FP64 values as they are; the mixed form's FP32 values as FP32 on the GPU."""
        return t if self.ctx.precision == "fp64" else t.to("cuda").to(torch.float32)

    def grids(self):
        for i, f in enumerate(self.fields):
            self.ctx._check(pm.lib().pmpic_download_grid(self.ctx._h, pm.GRID[f], self._p(self.grid[i])))
        g = self._form(self.grid)
        return {f: g[i] for i, f in enumerate(self.fields)}

    def parcels(self):
        n = C.c_int64()
        self.ctx._check(pm.lib().pmpic_download_parcels(self.ctx._h, self.cap, C.byref(n),
                                                        *[self._p(self.out[i]) for i in range(11)]))
        got = {}
        for i, k in enumerate(pm.IO_PROPS):
            t = self.out[i]
            if k == "tag" and self.ctx.precision == "mixed":
                got[k] = t.to("cuda").to(torch.int64)
            else:
                got[k] = self._form(t)
        return got

    def properties(self):
        n = self.ctx.n
        for i, k in enumerate(self.props):
            self.ctx._check(pm.lib().pmpic_get_property(self.ctx._h, pm.PROP[k], n, self._p(self.prop[i])))
        return {k: self._form(self.prop[i, :n]) for i, k in enumerate(self.props)}


def _model(ctx, back, parcels):
    """The results of a run: fields, parcels, and the step information."""
    info = ctx.info()
    out = {"grid": back.grids(), "n": int(info.n_parcels), "dtm": float(info.dtm),
           "split": int(info.n_split), "removed": int(info.n_removed), "added": int(info.n_added)}
    if parcels:
        out["parcel"] = back.parcels()
    return out


# ---- inputs ----------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _uniform(g, lo, hi, n):
    return torch.rand(n, generator=g, dtype=torch.float64, device="cuda") * (hi - lo) + lo


def _thermal(seed, nx, ny, nz, member=0):
    """A thermal of the ensemble's ranges: radius, excess and humidity, its own jitter."""
    r = torch.Generator().manual_seed(int(seed) * 131 + member)
    u = torch.rand(5, generator=r, dtype=torch.float64).tolist()
    return dict(nx=nx, ny=ny, nz=nz, lx=LX, ly=LY, lz=LZ, seed=int(seed) * 1009 + member,
                radius=0.25 + 0.25 * u[0], excess=0.5 + u[1], h_in=0.8 + 0.2 * u[2],
                xc=math.pi + 0.4 * (u[3] - 0.5), yc=math.pi + 0.4 * (u[4] - 0.5))


def _fourier(g, x, y, z, modes=16, kmax=8):
    """Sum of random Fourier modes with 0 < |k| <= kmax: periodic in x and y, cos in z."""
    out = torch.zeros(torch.broadcast_shapes(x.shape, y.shape, z.shape), dtype=torch.float64, device="cuda")
    done = 0
    while done < modes:
        a, b, m = torch.randint(-kmax, kmax + 1, (3,), generator=g, device="cuda").tolist()
        m = abs(m)
        amp, ph = torch.randn(1, generator=g, device="cuda").item(), torch.rand(1, generator=g, device="cuda").item()
        if 0 < a * a + b * b + m * m <= kmax * kmax:
            out += amp * torch.cos(2 * math.pi * (a * x / LX + b * y / LY + ph)) * torch.cos(math.pi * m * z / LZ)
            done += 1
    return out


def _interp_inputs(case, seed):
    """Random positions, the cell volume share, four parcel fields and six grids."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = 8 * nx * ny * nz
    g = _gen(seed)
    x, y, z = (_uniform(g, 0.0, h, n) for h in (LX, LY, LZ))
    par = {"x": x, "y": y, "z": z, "vol": torch.full_like(x, LX / nx * LY / ny * LZ / nz / 8)}
    for k in ("p", "q", "r", "b"):
        par[k] = _fourier(g, x, y, z)
    zg = torch.arange(nz + 1, dtype=torch.float64, device="cuda").view(-1, 1, 1) * (LZ / nz)
    yg = torch.arange(ny, dtype=torch.float64, device="cuda").view(1, -1, 1) * (LY / ny)
    xg = torch.arange(nx, dtype=torch.float64, device="cuda").view(1, 1, -1) * (LX / nx)
    return par, {k: _fourier(g, xg, yg, zg) for k in ("u", "v", "w", "dp", "dq", "dr")}


def _vorticity(case, seed):
    """Divergence-free random vorticity, k^-5/3 spectrum up to |k| = 64, unit RMS, free-slip walls: the curl
    of a random field with B_x, B_y ~ cos(kz z) and B_z ~ sin(kz z)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = _gen(seed)
    f = dict(dtype=torch.float64, device="cuda")
    kx = torch.arange(nx // 2 + 1, **f).view(1, 1, -1)
    ky = (torch.fft.fftfreq(ny, **f) * ny).view(1, -1, 1)
    kz = torch.arange(min(64, nz - 1) + 1, **f).view(-1, 1, 1)
    kk = torch.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
    amp = torch.where((kk > 0) & (kk <= min(64, nx // 3, ny // 3)), kk.clamp(min=1.0) ** (-11 / 6), 0.0 * kk)
    cx, cy, cz = (amp * torch.complex(torch.randn(amp.shape, generator=g, **f), torch.randn(amp.shape, generator=g, **f))
                  for _ in range(3))
    zk = torch.arange(nz + 1, **f).view(-1, 1) * math.pi / nz
    sin, cos = torch.sin(zk * kz.view(1, -1)), torch.cos(zk * kz.view(1, -1))

    def synth(w, basis):
        planes = torch.fft.irfft2(w, s=(ny, nx)) * (nx * ny)
        return (basis @ planes.reshape(planes.shape[0], -1)).view(nz + 1, ny, nx)
    p = synth(1j * ky * cz + kz * cy, sin)
    q = synth(-kz * cx - 1j * kx * cz, sin)
    r = synth(1j * kx * cy - 1j * ky * cx, cos)
    s = 1.0 / torch.sqrt(((p * p + q * q + r * r).mean() / 3))
    return p * s, q * s, r * s


def _midrun(case, seed):
    """A developed state: jittered parcels, volumes halved by earlier splits (some below the mixing
    threshold), stretches up to the splitting threshold, some cells nearly emptied, vortical."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = _gen(seed)
    cell = torch.arange(nx * ny * nz, device="cuda").repeat_interleave(8)
    n = cell.numel()
    sub = torch.arange(8, device="cuda").repeat(nx * ny * nz)
    d = [LX / nx, LY / ny, LZ / nz]
    ijk = [cell // (ny * nz), cell // nz % ny, cell % nz]
    abc = [sub // 4, sub // 2 % 2, sub % 2]
    x, y, z = (d[v] * (ijk[v] + (abc[v] + 0.5 + _uniform(g, -0.3, 0.3, n)) / 2) for v in range(3))
    halvings = (_uniform(g, 0, 1, n).clamp(min=1e-9).log() / math.log(0.4)).floor().clamp(max=5)
    st = {"x": x, "y": y, "z": z, "vol": d[0] * d[1] * d[2] / 8 * 2.0 ** -halvings}
    for k in ("p", "q", "r"):
        st[k] = 2.0 * _fourier(g, x, y, z, modes=6, kmax=4)
    st["b"] = 0.2 * _fourier(g, x, y, z, modes=6, kmax=4)
    st["h"] = 0.3 * (1 - z / LZ)
    st["stretch"] = _uniform(g, 0, 4, n)
    st["tag"] = torch.arange(n, dtype=torch.float64, device="cuda")
    empty = torch.rand(nx * ny * nz, generator=g, device="cuda") < 0.002
    keep = ~(empty[cell] & (sub >= 2))
    return {k: v[keep] for k, v in st.items()}


# ---- prepare and run ---------------------------------------------------------------
def _context(case, cap):
    return pm.Context(case["nx"], case["ny"], case["nz"], LX, LY, LZ, dtm=case.get("dt", 0.01),
                      dtmax=case.get("dt", 0.01), max_parcels=cap, precision=case["precision"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        sizes = [int(s) for s in case["sizes"].split(",")]
        ens = pm.Ensemble([dict(nx=s, ny=s, nz=s, dtm=0.32 / s, dtmax=0.32 / s, max_parcels=int(1.15 * 8 * s ** 3),
                                precision=case["precision"]) for s in sizes])
        therm = [_thermal(seed, s, s, s, m) for m, s in enumerate(sizes)]
        for m, t in zip(ens.members, therm):
            m.setup_thermal(**t)
        ens.autotune()
        ens.set_concurrency(len(sizes))
        return {"case": case, "ens": ens, "thermal": therm,
                "back": [Readback(m, 0, ["u", "v", "w", "vol"]) for m in ens.members]}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = 8 * nx * ny * nz
    if kind == "static":
        g = _gen(seed)
        n = case["per_cell"] * nx * ny * nz
        par = [_uniform(g, 0.0, h, n) for h in (LX, LY, LZ)]
        par += [_uniform(g, 0.5, 1.5, n) * (LX * LY * LZ / n), torch.randn(n, generator=g, dtype=torch.float64, device="cuda")]
        return {"case": case, "par": par, "out": torch.empty(nz + 1, ny, nx, dtype=torch.float64, device="cuda")}
    if kind == "thermal":
        ctx = _context(case, int((1.15 if case["parcels"] else 1.02) * n) + 64)
        return {"case": case, "ctx": ctx, "thermal": _thermal(seed, nx, ny, nz),
                "back": Readback(ctx, ctx.max_parcels if case["parcels"] else 0, FIELDS)}
    if kind == "callbacks":
        # the box and plume of the host's configuration; the perturbation of its shape from the seed
        ctx = pm.Context(nx, ny, nz, 6.28, 6.28, 6.28, dtm=case["dt"], dtmax=case["dt"],
                         max_parcels=int(2.5 * n) + 4096, precision=case["precision"])
        e = torch.rand(3, generator=torch.Generator().manual_seed(int(seed)), dtype=torch.float64).tolist()
        return {"case": case, "ctx": ctx, "e": tuple(v - 0.5 for v in e), "back": Readback(ctx, ctx.max_parcels, FIELDS)}
    if kind == "restart":
        ctx = _context(case, 4 * n)
        host = {k: v.cpu().pin_memory() for k, v in _midrun(case, seed).items()}
        return {"case": case, "ctx": ctx, "host": host, "back": Readback(ctx, ctx.max_parcels, FIELDS)}
    if kind == "interp":
        ctx = _context(case, n)
        par, grids = _interp_inputs(case, seed)
        ctx.upload(**{k: v.cpu().numpy() for k, v in par.items()})
        for k, v in grids.items():
            ctx.set_grid(k, v.cpu().numpy())
        return {"case": case, "ctx": ctx,
                "back": Readback(ctx, 0, ["p", "q", "r", "b"], ["dxdt", "dydt", "dzdt", "dpdt", "dqdt", "drdt"])}
    if kind == "invert":
        ctx = _context(case, 16)
        for k, v in zip(("p", "q", "r"), _vorticity(case, seed)):
            ctx.set_grid(k, v.cpu().numpy())
        return {"case": case, "ctx": ctx, "back": Readback(ctx, 0, ["u", "v", "w"])}
    raise ValueError(kind)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "static":
        out = state["out"]
        rc = pm.lib().pmpic_par2grid_static(case["nx"], case["ny"], case["nz"], LX, LY, LZ, state["par"][0].numel(),
                                            *[t.data_ptr() for t in state["par"]], out.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream)
        if rc:
            raise pm.PmpicError(rc, "pmpic_par2grid_static")
        return out
    if kind == "ensemble":
        ens = state["ens"]
        for m, t in zip(ens.members, state["thermal"]):
            m.setup_thermal(**t)
        ens.step(case["steps"])
        return [{"grid": b.grids(), "n": m.n} for m, b in zip(ens.members, state["back"])]
    ctx, back = state["ctx"], state["back"]
    if kind == "thermal":
        ctx.setup_thermal(**state["thermal"])
        ctx.step(case["steps"])
        return _model(ctx, back, case["parcels"])
    if kind == "callbacks":
        ctx.setup_plume(e_values=state["e"])
        ctx.set_dtm(case["dt"])
        for _ in range(case["steps"]):
            for _ in range(4):
                ctx.vort2vel()
                ctx.vorticity_tendency()
                ctx.rk4_integrator()
                ctx.parcel_splitting()
                ctx.parcel_mixing()
            ctx.info()  # the host's synopsis reads the step information
        return _model(ctx, back, True)
    if kind == "restart":
        host = state["host"]
        ctx._check(pm.lib().pmpic_upload_parcels(ctx._h, host["x"].numel(),
                                                 *[Readback._p(host[k]) for k in pm.IO_PROPS]))
        ctx.set_dtm(case["dt"])
        ctx.step(case["steps"])
        return _model(ctx, back, True)
    if kind == "interp":
        ctx.par2grid_multi(["p", "q", "r", "b"], ["p", "q", "r", "b"])
        ctx.grid2par_multi(["u", "v", "w", "dp", "dq", "dr"], back.props)
        return {"grid": back.grids(), "par": back.properties()}
    ctx.vort2vel_grids()
    return back.grids()


# ---- what a pass cannot do without --------------------------------------------------
def _step_work(n, nx, ny, nz, word):
    """Bytes and operations of one model step.  Per substep a parcel's 9 gridded values (position, volume,
    vorticity, buoyancy, humidity) are read for par2grid and its RK4 state (6 values, their step's start
    and their sums) is read and written, once each; the grids are read and written once per transform
    (6 forward or inverse in the inversion and its correction each, 9 in the tendency)."""
    nph = (nz + 1) * ny * nx
    par = 4 * 9 + (6 + 18) + 2 * (18 + 12) + (12 + 6)
    lg = math.log2(nx) + math.log2(ny)
    return (n * par * word + 4 * nph * 2 * 21 * word, 4 * (n * 350.0 + nph * (21 * 2.5 * lg + 120)))


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        w = [_step_work(8 * s ** 3, s, s, s, 8 if case["precision"] == "fp64" else 4)
             for s in map(int, case["sizes"].split(","))]
        return {"bytes": case["steps"] * sum(b for b, _ in w), "flops": case["steps"] * sum(f for _, f in w)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nph = (nz + 1) * ny * nx
    word = 8 if case.get("precision", "fp64") == "fp64" else 4
    n = case.get("per_cell", 8) * nx * ny * nz
    if kind == "static":
        return {"bytes": 40 * n + 8 * nph, "flops": 60 * n}
    if kind == "interp":  # positions, volume and four fields in, six values out; four grids out, six in
        return {"bytes": word * (14 * n + 10 * nph), "flops": 240.0 * n}
    if kind == "invert":  # three grids in, three out
        lg = math.log2(nx) + math.log2(ny)
        return {"bytes": word * 6 * nph, "flops": nph * (9 * 2.5 * lg + 80)}
    b, f = _step_work(n, nx, ny, nz, word)
    return {"bytes": case["steps"] * b, "flops": case["steps"] * f}


# ---- 64-bit values --------------------------------------------------------------------
def _exact_par2grid(pos, vol, fields, nx, ny, nz):
    """Volume-weighted trilinear means of the fields at the grid points, (nz+1, ny, nx) each."""
    d = (LX / nx, LY / ny, LZ / nz)
    c = [torch.floor(p / h) for p, h in zip(pos, d)]
    f = [p / h - k for p, h, k in zip(pos, d, c)]
    c = [k.long() for k in c]
    tot = torch.zeros(len(fields) + 1, (nz + 1) * ny * nx, dtype=torch.float64, device="cuda")
    for u in range(8):
        a, b, e = u & 1, u >> 1 & 1, u >> 2
        w = vol * (f[0] if a else 1 - f[0]) * (f[1] if b else 1 - f[1]) * (f[2] if e else 1 - f[2])
        at = ((c[2] + e) * ny + (c[1] + b) % ny) * nx + (c[0] + a) % nx
        tot[-1].index_add_(0, at, w)
        for q, v in enumerate(fields):
            tot[q].index_add_(0, at, w * v)
    wt = torch.where(tot[-1] == 0, torch.ones_like(tot[-1]), tot[-1])
    return [(t / wt).view(nz + 1, ny, nx).cpu() for t in tot[:-1]]


def _exact_grid2par(pos, grids, nx, ny, nz):
    d = (LX / nx, LY / ny, LZ / nz)
    c = [torch.floor(p / h) for p, h in zip(pos, d)]
    f = [p / h - k for p, h, k in zip(pos, d, c)]
    c = [k.long() for k in c]
    out = [torch.zeros_like(pos[0]) for _ in grids]
    for u in range(8):
        a, b, e = u & 1, u >> 1 & 1, u >> 2
        w = (f[0] if a else 1 - f[0]) * (f[1] if b else 1 - f[1]) * (f[2] if e else 1 - f[2])
        at = ((c[2] + e) * ny + (c[1] + b) % ny) * nx + (c[0] + a) % nx
        for o, gr in zip(out, grids):
            o += w * gr.reshape(-1)[at]
    return [o.cpu() for o in out]


def _exact_invert(p, q, r):
    """The inversion in complex form: the correction to a divergence-free vorticity, then the velocity
    u = curl of the vector potential, with the compact fourth-order z operators and their boundary rows."""
    nz1, ny, nx = p.shape
    dz = LZ / (nz1 - 1)
    dev, f64 = p.device, torch.float64
    lit = lambda a, b: float(torch.tensor(a, dtype=torch.float32) / torch.tensor(b, dtype=torch.float32))  # noqa: E731
    f16, f13, f112, f56 = lit(1, 6), lit(1, 3), lit(1, 12), lit(5, 6)
    f23 = lit(2, 3)
    mx = torch.arange(nx // 2 + 1, dtype=f64, device=dev).view(1, -1)
    my = (torch.fft.fftfreq(ny, dtype=f64, device=dev) * ny).view(-1, 1)
    kx, ky = 2 * math.pi * mx / LX, 2 * math.pi * my / LY
    k2 = kx ** 2 + ky ** 2
    keep = ((mx / LX) ** 2 + (my / LY) ** 2 <= ((nx / 2 / LX) ** 2 + (ny / 2 / LY) ** 2) * 2 / 9).to(f64)
    dx = 1j * torch.where(mx == nx // 2, 0.0 * kx, kx)  # a real field's derivative has no Nyquist mode
    dy = 1j * torch.where(my.abs() == ny / 2, 0.0 * ky, ky)

    def solve(lo, di, up, rhs):
        """Thomas recurrence over levels; lo, di, up are per-level scalars or (ny, nx/2+1) arrays."""
        n = len(rhs)
        cp, x = [None] * n, [None] * n
        den = di[0] + torch.zeros_like(k2)
        x[0] = rhs[0] / den
        for k in range(1, n):
            cp[k] = up[k - 1] / den
            den = di[k] - lo[k] * cp[k]
            x[k] = (rhs[k] - lo[k] * x[k - 1]) / den
        for k in range(n - 2, -1, -1):
            x[k] = x[k] - cp[k + 1] * x[k + 1]
        return torch.stack(x)

    def laplinv(f, df0):
        n, i2 = nz1, 1 / dz / dz
        lo, di, up = [i2 - f112 * k2] * n, [-2 * i2 - f56 * k2] * n, [i2 - f112 * k2] * n
        rhs = [None] * n
        for k in range(1, n - 1):
            rhs[k] = f112 * f[k - 1] + f56 * f[k] + f112 * f[k + 1]
        if df0:
            di[0] = di[n - 1] = -i2 - f13 * k2
            up[0] = lo[n - 1] = i2 - f16 * k2
            rhs[0], rhs[n - 1] = f13 * f[0] + f16 * f[1], f13 * f[n - 1] + f16 * f[n - 2]
        else:
            one = torch.ones_like(k2)
            di[0] = di[n - 1] = one
            up[0] = lo[n - 1] = 0 * one
            rhs[0] = rhs[n - 1] = torch.zeros_like(f[0])
        for v in (lo, di, up):
            for k in range(n):
                v[k] = torch.where(k2 == 0, torch.ones_like(k2) if v is di else 0 * k2, v[k])
        return torch.where(k2 == 0, f, solve(lo, di, up, rhs))

    def diffz(f, bot=None, top=None):
        n = nz1
        lo, di, up = [f16] * n, [f23] * n, [f16] * n
        lo[n - 1], up[0] = (f13, f13) if bot is not None else (0.0, 0.0)
        di[0] = di[n - 1] = 1.0
        rhs = [None] * n
        for k in range(1, n - 1):
            rhs[k] = (f[k + 1] - f[k - 1]) / 2 / dz
        if bot is None:
            rhs[0] = rhs[n - 1] = torch.zeros_like(f[0])
        else:
            rhs[0], rhs[n - 1] = f[1] / dz - f16 * bot * dz, -f[n - 2] / dz + f16 * top * dz
        return solve(lo, di, up, rhs)

    a, b, c = (torch.fft.rfft2(g) for g in (p, q, r))
    dc = torch.empty_like(c)
    dc[1:-1] = (c[2:] - c[:-2]) * (0.5 / dz)
    dc[0] = (4 * c[1] - c[2] - 3 * c[0]) * (0.5 / dz)
    dc[-1] = (c[-3] + 3 * c[-1] - 4 * c[-2]) * (0.5 / dz)
    f = dx * a + dy * b + dc
    f[:, 0, 0] = 0
    lam = laplinv(f, True) * keep
    a, b = a - dx * lam, b - dy * lam
    c = c - diffz(lam)
    c[0] = 0
    abot, atop, bbot, btop = a[0], a[-1], b[0], b[-1]

    def mean_flow(col):
        v = torch.zeros(nz1, dtype=f64, device=dev)
        v[1:] = torch.cumsum(dz / 2 * (col[1:] + col[:-1]), 0)
        return v - lit(1, nz1) * (v[:-1] + 0.5 * v[-1]).sum()
    ubar, vbar = mean_flow(b[:, 0, 0].real), -mean_flow(a[:, 0, 0].real)
    a, b, c = laplinv(a, False), laplinv(b, False), laplinv(c, True)
    u = diffz(b, bbot, btop) - dy * c
    v = dx * c - diffz(a, abot, atop)
    w = dy * a - dx * b
    u[:, 0, 0], v[:, 0, 0] = ubar.to(u.dtype), vbar.to(v.dtype)
    return [torch.fft.irfft2(g, s=(ny, nx)).cpu() for g in (u, v, w)]


def exact(case, seed):
    """64-bit values of the interpolations and the inversion; a whole model run has none."""
    kind = case["kind"]
    if kind == "static":
        par = prepare(case, seed)["par"]
        return _exact_par2grid(par[:3], par[3], par[4:], case["nx"], case["ny"], case["nz"])[0]
    if kind == "interp":
        par, grids = _interp_inputs(case, seed)
        pos, size = [par[k] for k in ("x", "y", "z")], (case["nx"], case["ny"], case["nz"])
        g = _exact_par2grid(pos, par["vol"], [par[k] for k in ("p", "q", "r", "b")], *size)
        v = _exact_grid2par(pos, list(grids.values()), *size)
        return {"grid": dict(zip(("p", "q", "r", "b"), g)),
                "par": dict(zip(("dxdt", "dydt", "dzdt", "dpdt", "dqdt", "drdt"), v))}
    if kind == "invert":
        return dict(zip(("u", "v", "w"), _exact_invert(*_vorticity(case, seed))))
    return None
