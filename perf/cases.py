"""The timed cases of the particle step: what a driver of this framework has it do.

Every case goes through ``romspath_b200.Tracker`` (and ``adjoint.Adjoint``), as
a user's program does.  Three kinds:

``step``      one ``Tracker.step``, the particle columns read where they are, on
              the device (``Tracker.device_state``): a driver that analyses the
              particles on the GPU after every internal step.
``interval``  one frame interval of a run, as the benchmark's end-to-end loop
              makes it: the interval's internal steps in one ``step_n`` call, the
              output record behind them, the next frame uploaded from page-locked
              host arrays while they run, then the record's columns on the host.
``adjoint``   release attribution: the particles set, ``forward`` over two frame
              intervals, the loss of the final positions, ``backward``.

Grids, frames and releases are the shapes of ``romspath_b200.synth`` (sigma-
coordinate grids, a double gyre with an M2 tide, parabolic diffusivities, land,
Stokes drift), made on the GPU in this file; the seed moves the tide's phase, the
islands, the particles and their noise.
"""
import math
import types

import numpy as np
import torch

from romspath_b200 import Tracker, synth
from romspath_b200 import adjoint as adj

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
DT, IDT, DELTAT = 3600, 300, 30.0          # frame interval, internal step, VTurb sub-step (s)
F64 = torch.float64


def _case(name, kind, form, nx, ny, N, n, **kw):
    c = {"name": name, "kind": kind, "form": form, "nx": nx, "ny": ny, "N": N, "n": n, "vturb": True, "hturb": False,
         "stokes": False, "diag": False, "land": "corner", "nested": False, "nsteps": 12}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest run of the test suite: one step of a handful of particles, all latency
        _case("tiny step f64", "step", "f64", 24, 20, 6, 500, hturb=True),
        # the plain method's grid and release (130 x 98 x 20, 10,000 particles), step by step
        _case("130x98 step f64", "step", "f64", 130, 98, 20, 10_000),
        # an ordinary exact run on sizes that fill no tile or block
        _case("odd interval f64", "interval", "f64", 257, 191, 25, 131_071, hturb=True, land="islands"),
        # the exact form at scale: FP32 frames with Stokes drift, HTurb, islands, a million particles
        _case("512x384 interval f32", "interval", "f32", 512, 384, 30, 1_048_576, hturb=True, stokes=True,
              land="islands"),
        # the same run without the random walk (deterministic trajectories)
        _case("512x384 advection f32", "interval", "f32", 512, 384, 30, 1_048_576, vturb=False, stokes=True,
              land="islands"),
        # the mixed form's latency: the small release, step by step
        _case("130x98 step mixed", "step", "mixed", 130, 98, 20, 10_000),
        # the benchmark's default workload, one frame interval end to end
        _case("512x384 interval mixed", "interval", "mixed", 512, 384, 30, 1_048_576, hturb=True, stokes=True,
              land="islands"),
        # the precision study's workload: many particles on a grid that stays in cache
        _case("130x98 interval mixed", "interval", "mixed", 130, 98, 20, 4_194_304),
        # fixed-point fields with the output diagnostics (salt, temp, bottom stress), odd sizes
        _case("odd diagnostics int16", "interval", "mixed-i16", 301, 215, 17, 300_007, hturb=True, diag=True,
              land="islands"),
        # a parent with two children (5x and 3x), particles handed between them
        _case("nested interval mixed", "interval", "mixed", 400, 300, 30, 1_500_000, hturb=True, stokes=True,
              land="islands", nested=True),
        # the same layout, small, in the exact form
        _case("nested step f64", "step", "f64", 120, 90, 12, 20_011, hturb=True, land="islands", nested=True),
        # release attribution on the plain method's grid: forward and backward over two intervals
        _case("adjoint f64", "adjoint", "f64", 130, 98, 20, 65_536, nsteps=24),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "interval", "interval", "interval", "interval", "adjoint"])
    form = "f64" if kind == "adjoint" else rng.choice(["f64", "f32", "mixed", "mixed", "mixed", "mixed-i16"])
    exact_form = form in ("f64", "f32")
    nx = logu(48, 480)
    ny = max(40, int(nx * rng.uniform(0.6, 0.9)))
    # attribution ensembles come in whole warps; the other releases in any number
    n = 32 * logu(16, 1_900) if kind == "adjoint" else logu(500, 400_000 if exact_form else 1_400_000)
    nested = kind != "adjoint" and nx >= 80 and rng.random() < 0.2
    return _case("", kind, form, nx, ny, rng.randint(6, 34), n,
                 vturb=kind == "adjoint" or rng.random() < 0.85, hturb=rng.random() < 0.5,
                 stokes=rng.random() < 0.4, diag=kind == "interval" and not nested and rng.random() < 0.2,
                 land=rng.choice(["corner", "islands", "none"]), nested=nested,
                 nsteps=24 if kind == "adjoint" else 12)


# ------------------------------------------------------------------ inputs

def _specs(case, seed):
    nx, ny, N = case["nx"], case["ny"], case["N"]
    P = synth.GridSpec(nx, ny, N, land=case["land"], land_seed=seed, stokes=case["stokes"], diag=case["diag"])
    if not case["nested"]:
        return [P]
    lx, ly = (nx - 1) * P.dx, (ny - 1) * P.dy

    def child(r, fx, fy, px, py):
        return synth.GridSpec(int(fx * nx) // r * r, int(fy * ny) // r * r, N, land="none", stokes=case["stokes"],
                              dx=P.dx / r, dy=P.dy / r, x0=int(px * nx) * P.dx, y0=int(py * ny) * P.dy, eddy=0.1,
                              gyre_lx=lx, gyre_ly=ly)
    P.gyre_lx, P.gyre_ly = lx, ly
    return [child(5, 0.75, 0.83, 0.625, 0.5), child(3, 0.6, 0.6, 0.15, 0.2), P]


def _params(case):
    p = synth.config_params("cfg1")
    p.update(idt=IDT, dt=DT, deltat=DELTAT, vturb_on=int(case["vturb"]), hturb_on=int(case["hturb"]),
             constant_hturb=[1.0] * 5)
    if case["diag"]:
        p.update(salttemp_on=1, salttemp_mean=1, write_bottom=1)
    return p


def _t0(seed):
    return float(np.random.default_rng([seed, 1]).uniform(0.0, synth.M2_PERIOD))


def _dev(a, dtype=F64):
    """A Fortran-ordered array as its transpose on the device: [j][i]."""
    return torch.as_tensor(np.ascontiguousarray(np.asarray(a).T), device=DEV).to(dtype)


def _fields(spec, grid, t):
    """A frame at model time t: FP64 tensors [k][j][i] (zeta [j][i]), synth.make_frame's formulas."""
    nx, ny = spec.xi_rho, spec.eta_rho
    h, m, mu, mv = (_dev(grid[k]) for k in ("h", "mask_rho", "mask_u", "mask_v"))
    x = spec.x0 + torch.arange(nx, dtype=F64, device=DEV) * spec.dx
    y = spec.y0 + torch.arange(ny, dtype=F64, device=DEV) * spec.dy
    lx = spec.gyre_lx or (nx - 1) * spec.dx
    ly = spec.gyre_ly or (ny - 1) * spec.dy
    om, kx = 2.0 * math.pi / synth.M2_PERIOD, 2.0 * math.pi / lx

    def lev(a):
        return torch.as_tensor(a, dtype=F64, device=DEV)[:, None, None]

    def gyre(xp, yp):
        a = 0.1 * math.sin(2.0 * math.pi / 864000.0 * t)
        b, xs, ys = 1.0 - 2.0 * a, 2.0 * xp / lx, yp / ly
        f, fx = a * xs * xs + b * xs, 2.0 * a * xs + b
        u = -0.3 * torch.sin(math.pi * f) * torch.cos(math.pi * ys)
        v = 0.3 * ly * torch.cos(math.pi * f) * torch.sin(math.pi * ys) * fx * (2.0 / lx)
        if spec.eddy > 0.0:
            k = 2.0 * math.pi / 20000.0
            u = u - spec.eddy * torch.sin(k * xp) * torch.cos(k * yp)
            v = v + spec.eddy * torch.cos(k * xp) * torch.sin(k * yp)
        return u, v

    zeta = 0.5 * torch.cos(om * t - kx * x)[None, :] * m
    S_r = (spec.hc * lev(grid["s_rho"]) + h * lev(grid["cs_r"])) / (spec.hc + h)
    S_w = (spec.hc * lev(grid["s_w"]) + h * lev(grid["cs_w"])) / (spec.hc + h)
    z_r, z_w = zeta + (zeta + h) * S_r, zeta + (zeta + h) * S_w
    zu, zv = 0.5 * (z_r[..., :-1] + z_r[..., 1:]), 0.5 * (z_r[:, :-1, :] + z_r[:, 1:, :])
    xu, yv = x[:-1] + 0.5 * spec.dx, y[:-1] + 0.5 * spec.dy
    out = {"zeta": zeta,
           "u": (gyre(xu[None, :], y[:, None])[0] * torch.exp(zu / 100.0) + 0.1 * torch.cos(om * t - kx * xu)) * mu,
           "v": gyre(x[None, :], yv[:, None])[1] * torch.exp(zv / 100.0) * mv,
           "w": -(z_w + h) * (0.1 * kx * torch.sin(om * t - kx * x)) * m}
    xi = (z_w + h) / (zeta + h)
    out["aks"] = (1e-2 * (0.75 + 0.25 * math.cos(2.0 * om * t)) * 4.0 * xi * (1.0 - xi)).clamp(min=0.0) * m
    if spec.stokes:
        out["su"] = 0.05 * torch.exp(zu / 5.0) * math.cos(math.radians(30.0)) * mu
        out["sv"] = 0.05 * torch.exp(zv / 5.0) * math.sin(math.radians(30.0)) * mv
    if spec.diag:
        tide = torch.sin(om * t - kx * x)
        out["salt"] = (33.0 + 2.0 * (1.0 - torch.exp(z_r / 30.0)) + 0.3 * tide) * m
        out["temp"] = (8.0 + 10.0 * torch.exp(z_r / 40.0) - 0.5 * tide) * m
        out["bustr"] = 2.5e-3 * out["u"][0] * out["u"][0].abs()
        out["bvstr"] = 2.5e-3 * out["v"][0] * out["v"][0].abs()
    return out


def _src_dtype(case):
    """The exact FP64 form's frames come in double precision, the others' in single."""
    return F64 if case["form"] == "f64" else torch.float32


def _host_frame(fields, dtype, pinned):
    """The frame as a reader hands it over: Fortran-ordered host arrays."""
    out, keep = {}, []
    for k, a in fields.items():
        t = torch.empty(a.shape, dtype=dtype, pin_memory=pinned and DEV.type == "cuda")
        t.copy_(a)
        keep.append(t)
        out[k] = t.numpy().transpose(*range(a.dim() - 1, -1, -1))
    out["_keep"] = keep
    return out


def _inputs(case, seed, nframes):
    specs = _specs(case, seed)
    grids = [synth.make_grid(s) for s in specs]
    t0 = _t0(seed)
    frames = [[_fields(s, g, t0 + DT * k) for s, g in zip(specs, grids)] for k in range(nframes)]
    zeta0 = frames[0][-1]["zeta"].cpu().numpy().T
    if case["nested"]:
        rel = synth.nested_release(specs, grids, None, case["n"], seed=seed, child_frac=0.25)
    else:
        rel = synth.uniform_release(specs[0], grids[0], {"zeta": zeta0}, case["n"], seed=seed)
    return specs, grids, frames, rel


def _interval(p):
    """External step 3 + p: frame times, ring slots and its internal steps (run_External_Timestep's loop)."""
    ets = 3 + p
    ex = (float((ets - 2) * DT), float((ets - 1) * DT), float(ets * DT))
    tb, tc, tf = p % 3 + 1, (p + 1) % 3 + 1, (p + 2) % 3 + 1
    return [types.SimpleNamespace(ex=ex, ix=tuple(ex[1] + float(q * IDT) for q in (i - 1, i, i + 1)), ets=ets, tb=tb,
                                  tc=tc, tf=tf) for i in range(DT // IDT)]


def _frame_of(k):
    """Frame number k of the run from the pool of four: 0 1 2 3 2 1 0 ..., each next to its neighbours in time."""
    k %= 6
    return k if k < 4 else 6 - k


# --------------------------------------------------------- prepare and run

class _Column:
    """A particle column in the tracker's device memory; a tensor made of it keeps the tracker alive."""

    def __init__(self, tracker, ptr, n, typestr):
        self.tracker = tracker
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


COLUMNS = {"x": "<f8", "y": "<f8", "z": "<f8", "age": "<f8", "status": "<f8", "wd": "<f8", "zeta": "<f8",
           "bath": "<f8", "gid": "<i4", "isin": "|i1"}


def prepare(case, seed):
    S = types.SimpleNamespace(case=case, p=0, i=0)
    kind, mixed = case["kind"], case["form"].startswith("mixed")
    specs, grids, frames, rel = _inputs(case, seed, 4 if kind == "interval" else 3)
    scl = off = None
    if case["nested"]:
        scl, off = synth.nest_maps(specs)
    S.T = Tracker(specs, grids, _params(case), case["n"], field_dtype=case["form"], stokes=case["stokes"],
                  seed=seed + 1, scl=scl, off=off, resort=12 if kind == "interval" else 0)
    S.frames = [[_host_frame(f, _src_dtype(case), kind == "interval") for f in fr] for fr in frames]
    for slot in (1, 2, 3):
        for g in range(len(specs)):
            S.T.upload_frame(g + 1, slot, S.frames[slot - 1][g])
    S.T.locate(rel)
    if kind == "adjoint":
        c = S.T.get_particles()
        S.start = [c["x"], c["y"], c["z"], rel.dob, c["age"], c["status"], c["gid"], c["isin"]]
        S.A = adj.Adjoint(S.T)
        S.A.load_frames(3, lambda ng, k: S.frames[k - 1][ng - 1])
        S.steps = adj.step_table(case["nsteps"] * IDT / 86400.0, DT, IDT)[0]
        S.target = (0.5 * case["nx"], 0.5 * case["ny"])
    elif kind == "interval":
        names = ["lon", "lat", "zp", "age", "status", "gid"]
        if case["diag"]:
            names += ["salt", "temp", "hob", "bustr", "bvstr"]
        S.rec = {k: torch.empty(case["n"], dtype=F64, pin_memory=DEV.type == "cuda") for k in names}
        S.out = {k: v.numpy() for k, v in S.rec.items()}
    else:
        st = S.T.device_state()
        S.cols = {k: torch.as_tensor(_Column(S.T, getattr(st, k), case["n"], t), device=DEV)
                  for k, t in COLUMNS.items()}
        S.stream = torch.cuda.ExternalStream(st.stream)
    S.mixed = mixed
    return S


# The mixed forms hold positions and depths in FP32: their columns are taken at
# that width.  Status keeps its whole part there: 1.1 and 1.2 mark a reflection
# within the last step, which the last bit of an FP32 depth decides.
FP32_COLUMNS = ("x", "y", "z", "wd", "zeta", "bath", "lon", "lat", "zp", "salt", "temp", "hob", "bustr", "bvstr")


def _taken(cols, mixed):
    if not mixed:
        return dict(cols)
    return {k: v.float() if k in FP32_COLUMNS else v.floor() if k == "status" else v for k, v in cols.items()}


def run(S):
    case, T = S.case, S.T
    if case["kind"] == "adjoint":
        T.set_particles(*S.start)
        S.A.forward(S.steps, kappa=1.0, checkpoint_every=12)
        end = T.get_particles()
        loss, gx, gy = adj.attribution_loss(end["x"], end["y"], S.target)
        dx, dy, dz, dk = S.A.backward(gx, gy, np.zeros_like(gx))
        return {"x": end["x"], "y": end["y"], "z": end["z"], "loss": loss, "dx": dx, "dy": dy, "dz": dz, "dk": dk}
    if case["kind"] == "interval":
        steps = _interval(S.p)
        T.step_n(steps)
        T.output_record_async(len(steps), S.out)
        for g, f in enumerate(S.frames[_frame_of(S.p + 3)]):
            T.upload_frame(g + 1, steps[0].tb, f)
        T.output_wait()
        S.p += 1
        return _taken(S.rec, S.mixed)
    it = _interval(0)[S.i]
    S.i = (S.i + 1) % (DT // IDT)
    T.step(it.ex, it.ix, it.ets, it.tb, it.tc, it.tf)
    if not S.mixed:
        return S.cols
    T.device_state()                       # writes x, y, z from the compensated columns
    with torch.cuda.stream(S.stream):
        return _taken(S.cols, True)


def work(case):
    """Per internal step: the fields' live slots that the particles' stencils can reach, each once; the particle
    state in and out; for the random walk one fit (factor, two substitutions, the sum) of its np points."""
    bpv = {"f64": 8, "f32": 4}.get(case["form"], 2)
    cells = case["nx"] * case["ny"] * (2.2 if case["nested"] else 1.0)
    n, N, ns = case["n"], case["N"], 1 if case["kind"] == "step" else case["nsteps"]
    fields = 4 if case["vturb"] else 3
    gather = min(3 * bpv * fields * (N + 1) * cells, 3 * bpv * n * (4 * 3 * 8 + (4 * (N + 1) if case["vturb"] else 0)))
    flops = 4 * 300 + (30 * (N + 1) + 40 * 4 * (N + 1) + 10 * 80 if case["vturb"] else 0)
    total = {"bytes": ns * (gather + 150 * n), "flops": ns * n * flops}
    if case["kind"] == "interval":
        total["bytes"] += (8 if case["form"] == "f64" else 4) * cells * (4 * N + 3) + 48 * n
    if case["kind"] == "adjoint":              # each step again, with its four derivatives
        total = {k: 5 * v for k, v in total.items()}
    return {k: float(v) for k, v in total.items()}


# ------------------------------------------------- the model in 64 bits
#
# update_particles (ROMSPath.f90:608-1008) as plain torch in FP64, over all
# particles at once, Vtransform 2, away from the grid's edge cells.  The steps
# are differentiable, so that autograd gives the adjoint's gradients.

class _G:
    """One grid with its frames interpolated in time to a step's ix(2)."""

    def __init__(self, spec, grid):
        self.nx, self.ny, self.N, self.hc = spec.xi_rho, spec.eta_rho, spec.N, spec.hc
        for k in ("h", "pm", "pn", "mask_rho", "mask_u", "mask_v", "lon_rho", "lat_rho"):
            setattr(self, k, _dev(grid[k]).reshape(-1))
        for k in ("s_rho", "cs_r", "s_w", "cs_w"):
            setattr(self, k, torch.as_tensor(grid[k], dtype=F64, device=DEV)[:, None])

    def set_time(self, f3, a, auvw):
        """f3: the b, c, f frames; a, auvw: their Lagrange weights (u, v, w at the first external step: b, b, c)."""
        u = [f["u"] + f["su"] if "su" in f else f["u"] for f in f3]
        v = [f["v"] + f["sv"] if "sv" in f else f["v"] for f in f3]

        def mix(w, fs):
            return (w[0] * fs[0] + w[1] * fs[1] + w[2] * fs[2]).reshape(fs[0].shape[0], -1)
        self.u, self.v, self.w = mix(auvw, u), mix(auvw, v), mix(auvw, [f["w"] for f in f3])
        self.aks = mix(a, [f["aks"] for f in f3])
        self.zeta = mix(a, [f["zeta"] for f in f3]).reshape(-1)
        self.f3, self.a = f3, a


def _dot(w, a, o):
    return w[0] * a[o[0]] + w[1] * a[o[1]] + w[2] * a[o[2]] + w[3] * a[o[3]]


def _corners(ix, jx, ni, nj):
    i0, i1 = ix.clamp(1, ni) - 1, (ix + 1).clamp(1, ni) - 1
    j0, j1 = (jx.clamp(1, nj) - 1) * ni, ((jx + 1).clamp(1, nj) - 1) * ni
    return [j0 + i0, j0 + i1, j1 + i1, j1 + i0]


def _bilinear(X, Y):
    return [(1 - X) * (1 - Y), X * (1 - Y), X * Y, (1 - X) * Y]


def _rho(g, x, y):
    """Corner indices, bilinear and inverse-distance weights, and the weights of w and AKs."""
    I, J = torch.floor(x.detach()), torch.floor(y.detach())
    X, Y = x - I, y - J
    o = _corners(I.long(), J.long(), g.nx, g.ny)
    cb = _bilinear(X, Y)
    m = [g.mask_rho[k] for k in o]
    d = [X * X + Y * Y, (1 - X) ** 2 + Y * Y, (1 - X) ** 2 + (1 - Y) ** 2, X * X + (1 - Y) ** 2]
    w = [mk / torch.sqrt(dk) for mk, dk in zip(m, d)]
    tot = w[0] + w[1] + w[2] + w[3]
    safe = torch.where(tot == 0, torch.ones_like(tot), tot)
    ci = [wk / safe for wk in w]
    wet = m[0] + m[1] + m[2] + m[3] >= 4
    return o, cb, ci, [torch.where(wet, b, c) for b, c in zip(cb, ci)]


def _uv(g, x, y, f, mask, is_u, L):
    ni, nj = (g.nx - 1, g.ny) if is_u else (g.nx, g.ny - 1)
    xs, ys = (x - 0.5, y) if is_u else (x, y - 0.5)
    I, J = torch.floor(xs.detach()), torch.floor(ys.detach())
    o = _corners(I.long(), J.long(), ni, nj)
    m = [mask[k] for k in o]
    return _level(f, o, [b * (mk != 0) for b, mk in zip(_bilinear(xs - I, ys - J), m)], L)


def _pick(lv, z):
    """Bracket of z among the levels lv (nz, n) and its weights: the end level itself beyond the ends."""
    nz = lv.shape[0]
    c = (lv <= z).sum(0)
    ib, it = c.clamp(min=1), (c + 1).clamp(max=nz)
    zb, zt = lv.gather(0, (ib - 1)[None])[0], lv.gather(0, (it - 1)[None])[0]
    same = ib == it
    Z = torch.where(same, torch.full_like(z, 0.5), (z - zb) / torch.where(same, torch.ones_like(z), zt - zb))
    return ib - 1, it - 1, 1 - Z, Z


def _level(f, o, w, L):
    ib, it, wb, wt = L
    plane = f.shape[1]
    flat = f.reshape(-1)
    return wb * _dot(w, flat, [ib * plane + k for k in o]) + wt * _dot(w, flat, [it * plane + k for k in o])


def _z_levels(g, s, cs, zeta, h):
    return zeta + (zeta + h) * ((g.hc * s + h * cs) / (g.hc + h))


def _currents(g, x, y, z):
    o, cb, ci, cw = _rho(g, x, y)
    h, zeta = _dot(cb, g.h, o), _dot(ci, g.zeta, o)
    z = torch.where(z < -h, -h + float(np.float32(0.001)), z)
    z = torch.where(z > zeta, zeta - float(np.float32(0.001)), z)
    Lr = _pick(_z_levels(g, g.s_rho, g.cs_r, zeta, h), z)
    Lw = _pick(_z_levels(g, g.s_w, g.cs_w, zeta, h), z)
    u = _uv(g, x, y, g.u, g.mask_u, True, Lr)
    v = _uv(g, x, y, g.v, g.mask_v, False, Lr)
    return u, v, _level(g.w, o, cw, Lw), z, (o, cw, h, zeta)


def _normal(pid, step, d, seed):
    """Philox4x32-10 at counter (pid, step, d/2), Box-Muller's cosine branch (pdf_module.f90:26-40)."""
    M = 0xFFFFFFFF
    c = [pid, torch.full_like(pid, step & M), torch.full_like(pid, step >> 32), torch.full_like(pid, d >> 1)]
    k0, k1 = seed & M, seed >> 32
    for r in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & M) ^ c[1] ^ k0, p1 & M, ((p0 >> 32) & M) ^ c[3] ^ k1, p0 & M]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    a, b = (c[2], c[3]) if d & 1 else (c[0], c[1])
    u1, u2 = (a.double() + 0.5) / 2.0 ** 32, (b.double() + 0.5) / 2.0 ** 32
    return torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2)


def _solve(y, hb, p, serr):
    """chol1d (pppack.f90:1428) on uniform breaks: u, and sum qu^2 dy^2."""
    n = y.shape[0]
    r2, c = (serr / hb) ** 2, 6.0 * (1.0 - p)
    D, E, F = c * 6.0 * r2 + 4.0 * p * hb, c * -4.0 * r2 + p * hb, c * r2
    zero = torch.zeros_like(hb)
    a1, a2, b1 = D, E, D
    up, uc, r2p = zero, (y[2] - 2.0 * y[1] + y[0]) / hb, zero
    s1, s2, q = [None] * n, [None] * n, [None] * n
    for i in range(1, n - 2):
        Fi = F if i < n - 3 else zero
        q1, q2 = a2 / a1, Fi / a1
        s1[i], s2[i], q[i] = q1, q2, uc / a1
        un = (y[i + 2] - 2.0 * y[i + 1] + y[i]) / hb - q1 * uc - r2p * up
        a1, a2, b1 = b1 - q1 * a2, E - q1 * Fi, D - q2 * Fi
        up, uc, r2p = uc, un, q2
    u = [zero] * n
    u[n - 2] = uc / a1
    for i in range(n - 3, 0, -1):
        u[i] = q[i] - u[i + 1] * s1[i] - u[i + 2] * s2[i]
    prev, tot = zero, zero
    for i in range(1, n):
        raw = (u[i] - u[i - 1]) / hb
        tot = tot + (raw - prev) ** 2
        prev = raw
    return u, (tot + prev ** 2) * serr ** 2


@torch.no_grad()
def _smoothing(y, hb, serr, s):
    """smooth's secant search for p (pppack.f90:5108-5317)."""
    u, sm = _solve(y, hb, torch.zeros_like(hb), serr)
    sf = 36.0 * sm
    utru = sum(hb * (u[i - 1] * (u[i - 1] + u[i]) + u[i] * u[i]) for i in range(1, len(u)))
    del u
    p = torch.zeros_like(hb)
    live = torch.nonzero(sf > s)[:, 0]
    if live.numel() == 0:
        return p
    Y, H, oos = y[:, live], hb[live], 1.0 / math.sqrt(s)
    sf, utru = sf[live], utru[live]
    of = 1.0 / torch.sqrt(sf)
    q, pq, ps = -(of - oos) * sf / (6.0 * utru * of), torch.zeros_like(sf), of
    for _ in range(100):
        sf = 36.0 * _solve(Y, H, q / (1.0 + q), serr)[1] / (1.0 + q) ** 2
        p[live] = q / (1.0 + q)
        keep = torch.nonzero(~((sf - s).abs() <= 0.01 * s))[:, 0]
        if keep.numel() == 0:
            break
        of = 1.0 / torch.sqrt(sf)
        q, pq, ps = q - (q - pq) / (of - ps) * (of - oos), q, of
        if keep.numel() < live.numel():
            live, Y, H, q, pq, ps = live[keep], Y[:, keep], H[keep], q[keep], pq[keep], ps[keep]
    return p


def _vturb(g, P, stage, z0, pid, step, seed, kappa):
    o, cw, h, zeta = stage
    sw = g.N + 1
    n = int(sw * P["sub"])
    zc = _z_levels(g, g.s_w, g.cs_w, zeta, h)
    kh = kappa * torch.stack([_dot(cw, g.aks[k], o) for k in range(sw)])
    z1, hb = zc[0], (zc[-1] - zc[0]) / (n - 1)
    rows = [kh[0]]
    for i in range(1, n - 1):
        x = z1 + i * hb
        j = ((zc <= x).sum(0) - 1).clamp(0, sw - 2)[None]
        zl, zh, kl, kk = zc.gather(0, j)[0], zc.gather(0, j + 1)[0], kh.gather(0, j)[0], kh.gather(0, j + 1)[0]
        m = (kl - kk) / (zl - zh)
        rows.append(m * x + (kl - m * zl))
    y = torch.stack(rows + [kh[-1]])
    serr = P["serr"]
    p = _smoothing(y.detach(), hb.detach(), serr, P["smth"])
    u = torch.stack(_solve(y, hb, p, serr)[0])
    zero = torch.zeros_like(hb)[None]
    raw = torch.cat([zero, (u[1:] - u[:-1]) / hb, zero])
    a1, a3 = y - 6.0 * (1.0 - p) * serr ** 2 * (raw[1:] - raw[:-1]), u * (6.0 * p)

    def fit(x, deriv):
        i = torch.floor((x - z1) / hb).detach().nan_to_num(0.0).clamp(0, n - 2).long()[None]
        c1, d1, c3, d3 = (a.gather(0, k)[0] for a in (a1, a3) for k in (i, i + 1))
        c4 = (d3 - c3) / hb
        c2 = (d1 - c1) / hb - (c3 + c4 / 3.0 * hb) / 2.0 * hb
        t = x - (z1 + i[0] * hb)
        return (c4 / 2.0 * t + c3) * t + c2 if deriv else ((c4 / 3.0 * t + c3) / 2.0 * t + c2) * t + c1

    depth, back, z = -h, torch.full_like(z0, P["aksback"]), z0
    for k in range(1, IDT // int(DELTAT) + 1):
        kp = torch.where((z <= depth) | (z >= zeta), torch.zeros_like(z), fit(z, True)) * DELTAT
        zm = z + 0.5 * kp
        K = fit(zm, False)
        K = torch.where((zm < depth) | (zm > zeta) | (K < back), back, K)
        z = z + kp + _normal(pid, step, 1 + k, seed) * torch.sqrt(2.0 * K * DELTAT)
        z = torch.where(z <= depth, depth + (z - depth).abs(), z)
        z = torch.where(z >= zeta, zeta - (z - zeta).abs(), z)
    return z - z0


def _inside(g, x, y):
    """bounds (boundary_module.f90:43-143): in the grid's water, and beyond its open boundary."""
    I, J = torch.floor(x).long(), torch.floor(y).long()
    X, Y = x - I, y - J
    deep = (I > 1) & (J > 1) & (I < g.nx - 1) & (J < g.ny - 1)
    o = _corners(I, J, g.nx, g.ny)
    m11, m21, m22, m12 = (g.mask_rho[k] == 1 for k in o)
    nm = m11.long() + m21.long() + m22.long() + m12.long()
    tri = torch.where(~m11, X + Y >= 1, torch.where(~m22, X + Y <= 1, torch.where(~m21, Y >= X, Y <= X)))
    e = float(np.float32(0.1))
    two = ((m11 & (X < e) & (Y < e)) | (m21 & (X > 1 - e) & (Y < e)) | (m22 & (X > 1 - e) & (Y > 1 - e)) |
           (m12 & (X < e) & (Y > 1 - e)))
    return deep & ((nm == 4) | ((nm == 3) & tri) | ((nm == 2) & two)), ~deep


def _advance(g, P, case, x, y, z, pid, step, seed, kappa):
    """Displacements of one internal step of particles in grid g."""
    o, cb, _, _ = _rho(g, x, y)
    pm, pn = _dot(cb, g.pm, o), _dot(cb, g.pn, o)
    u, v, w, zp, stage = _currents(g, x, y, z)
    ku, kv, kw = u * pm, v * pn, w
    su, sv, sw = ku, kv, kw
    for c in (2.0, 2.0, 1.0):
        u, v, w, _, _ = _currents(g, x + ku * (IDT / 2.0), y + kv * (IDT / 2.0), zp + kw * (IDT / 2.0))
        ku, kv, kw = u * pm, v * pn, w
        su, sv, sw = su + c * ku, sv + c * kv, sw + c * kw
    dx, dy, dz = IDT * su / 6.0, IDT * sv / 6.0, IDT * sw / 6.0
    if case["hturb"]:
        sc = math.sqrt(2.0 * P["constant_hturb"][0] * IDT)
        dx = dx + _normal(pid, step, 0, seed) * sc * pm
        dy = dy + _normal(pid, step, 1, seed) * sc * pn
    if case["vturb"]:
        dz = dz + _vturb(g, P, stage, zp, pid, step, seed, kappa)
    return dx, dy, dz


def _surface(g, x, y):
    o, cb, ci, _ = _rho(g, x, y)
    return -_dot(cb, g.h, o), _dot(ci, g.zeta, o)


def _exact_step(gs, scl, off, P, case, st, step, seed, kappa=1.0):
    """One update_particles of every particle (chunks of about a million); st: the columns, replaced."""
    n, ng = st["x"].numel(), len(gs)
    new = {k: [] for k in ("x", "y", "z", "status", "gid", "isin", "wd", "zeta", "bath")}
    for c0 in range(0, n, 1 << 20):
        sl = slice(c0, c0 + (1 << 20))
        x, y, z, gid = st["x"][sl], st["y"][sl], st["z"][sl], st["gid"][sl]
        pid = torch.arange(n, device=DEV)[sl]
        nx, ny, dz = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
        for g in range(ng):
            k = torch.nonzero(gid == g + 1)[:, 0] if ng > 1 else slice(None)
            if ng > 1 and k.numel() == 0:
                continue
            a, b, c = _advance(gs[g], P, case, x[k], y[k], z[k], pid[k], step, seed, kappa)
            if ng == 1:
                nx, ny, dz = x + a, y + b, c
            else:
                nx[k], ny[k], dz[k] = x[k] + a, y[k] + b, c
        tx, ty, to = nx, ny, gid
        if ng == 1:
            ins, out = _inside(gs[0], nx.detach(), ny.detach())
        else:
            ins, out = torch.zeros_like(gid, dtype=torch.bool), torch.zeros_like(gid, dtype=torch.bool)
            for g in range(ng):
                s = torch.as_tensor(scl[:, g, :], device=DEV)[gid - 1]
                f = torch.as_tensor(off[:, g, :], device=DEV)[gid - 1]
                mx, my = s[:, 0] * nx + f[:, 0], s[:, 1] * ny + f[:, 1]
                tx, ty = torch.where(ins, tx, mx), torch.where(ins, ty, my)
                i_g, o_g = _inside(gs[g], mx, my)
                out = torch.where(ins, out, o_g)
                to = torch.where(i_g & ~ins, torch.full_like(to, g + 1), to)
                ins = ins | i_g
        if ng == 1:
            depth, zeta = _surface(gs[0], tx, ty)
        else:
            depth, zeta = torch.zeros_like(tx), torch.zeros_like(tx)
            for g in range(ng):
                k = torch.nonzero(to == g + 1)[:, 0]
                if k.numel():
                    depth[k], zeta[k] = _surface(gs[g], tx[k], ty[k])
        nz = z + dz
        bot = nz < depth
        nz = torch.where(bot, depth + (nz - depth).abs(), nz)
        top = nz > zeta
        nz = torch.where(top, zeta - (nz - zeta).abs(), nz)
        mark = torch.where(bot, float(np.float32(1.2)), torch.where(top, float(np.float32(1.1)), 1.0))
        new["x"].append(torch.where(ins, tx, x))
        new["y"].append(torch.where(ins, ty, y))
        new["z"].append(torch.where(ins, nz, z))
        new["status"].append(torch.where(ins, mark, torch.where(out, -8.0, -9.0)).double())
        new["gid"].append(torch.where(ins, to, torch.where(out, torch.full_like(to, ng), gid)))
        new["isin"].append((ins | ~out).to(torch.int8))
        new["wd"].append(-depth + zeta)
        new["zeta"].append(zeta)
        new["bath"].append(-depth)
    st.update({k: torch.cat(v) for k, v in new.items()})
    st["age"] = st["age"] + float(IDT)


def _diagnostics(g, st):
    """ROMSPath.f90:935-986 after a step (one grid): bottom stress at the lowest height above bottom, salt and temp."""
    x, y, z = st["x"], st["y"], st["z"]
    b = st["bath"] + z
    hit = b <= st["hob"]
    st["hob"] = torch.minimum(b, st["hob"])
    one = (torch.zeros_like(x, dtype=torch.long),) * 2 + (torch.full_like(x, 0.5),) * 2
    for k, m, is_u in (("bustr", g.mask_u, True), ("bvstr", g.mask_v, False)):
        f = sum(a * q[k] for a, q in zip(g.a, g.f3)).reshape(1, -1)
        st[k] = torch.where(hit, _uv(g, x, y, f, m, is_u, one), st[k])
    o, _, ci, cw = _rho(g, x, y)
    for a, f in zip(g.a, g.f3):
        L = _pick(_z_levels(g, g.s_rho, g.cs_r, _dot(ci, f["zeta"].reshape(-1), o), st["bath"]), z)
        for k in ("salt", "temp"):
            st[k] = st[k] + a * _level(f[k].reshape(g.N, -1), o, cw, L)


def _start(gs, specs, grids, frames, rel, case):
    """ini_ROMSPath's ownership loop (ROMSPath.f90:367-432)."""
    n = case["n"]
    st = {"z": torch.as_tensor(rel.z, device=DEV), "age": torch.zeros(n, dtype=F64, device=DEV)}
    ones = torch.ones(n, dtype=F64, device=DEV)
    x, y, z, gid = ones, ones, st["z"], torch.full((n,), len(gs), device=DEV)
    got = torch.zeros_like(ones, dtype=torch.bool)
    for g, G in enumerate(gs):
        ix, jx = torch.as_tensor(rel.ipos[g], device=DEV), torch.as_tensor(rel.jpos[g], device=DEV)
        ins, _ = _inside(G, ix, jx)
        take = ins & ~got
        o, cb, ci, _ = _rho(G, ix, jx)
        surf = _dot(ci, frames[0][g]["zeta"].reshape(-1), o)
        z = torch.where(take & (z >= surf), surf - 0.01, z)
        x, y, gid, got = torch.where(take, ix, x), torch.where(take, jx, y), torch.where(take, g + 1, gid), got | ins
    st.update(x=x, y=y, z=z, gid=gid)
    for k in ("salt", "temp", "bustr", "bvstr"):
        st[k] = torch.zeros_like(ones)
    st["hob"] = 9999.0 * ones
    return st


def _weights(it):
    e, t = it.ex, it.ix[1]
    a = [(t - e[1]) * (t - e[2]) / ((e[0] - e[1]) * (e[0] - e[2])),
         (t - e[0]) * (t - e[2]) / ((e[1] - e[0]) * (e[1] - e[2])),
         (t - e[0]) * (t - e[1]) / ((e[2] - e[0]) * (e[2] - e[1]))]
    return a, ([a[0] + a[1], a[2], 0.0] if it.ets == 1 else a)


def exact(case, seed):
    if DEV.type != "cuda" and case["n"] * case["nsteps"] > 50_000:
        return None                            # over 20 seconds on host cores
    specs, grids, frames, rel = _inputs(case, seed, 3)
    frames = [[{k: v.to(_src_dtype(case)).double() for k, v in f.items()} for f in fr] for fr in frames]
    gs = [_G(s, g) for s, g in zip(specs, grids)]
    scl, off = synth.nest_maps(specs) if case["nested"] else (None, None)
    P, st = _params(case), _start(gs, specs, grids, frames, rel, case)
    if case["kind"] == "adjoint":
        return _exact_adjoint(gs[0], P, case, st, frames, seed)
    steps = _interval(0)[: 1 if case["kind"] == "step" else None]
    if case["diag"]:                           # the writer's sums start at the particle's own initial value
        gs[0].set_time([f[0] for f in frames], [0.0, 1.0, 0.0], [0.0, 1.0, 0.0])
        o, cb, ci, _ = _rho(gs[0], st["x"], st["y"])
        st["bath"] = _dot(cb, gs[0].h, o)
        hob = st["hob"]
        _diagnostics(gs[0], st)
        st.update(hob=hob, bustr=torch.zeros_like(hob), bvstr=torch.zeros_like(hob))
    for k, it in enumerate(steps):
        a, auvw = _weights(it)
        for g, G in enumerate(gs):
            G.set_time([f[g] for f in frames], a, auvw)
        _exact_step(gs, scl, off, P, case, st, k, seed + 1)
        if case["diag"]:
            _diagnostics(gs[0], st)
    if case["form"].startswith("mixed"):
        st["status"] = st["status"].floor()
    if case["kind"] == "step":
        return {k: st[k] for k in COLUMNS}
    out = {"lon": torch.zeros_like(st["x"]), "lat": torch.zeros_like(st["x"]), "zp": st["z"], "age": st["age"],
           "status": st["status"], "gid": st["gid"].double()}
    for g, G in enumerate(gs):
        k = torch.nonzero(st["gid"] == g + 1)[:, 0]
        o, cb, _, _ = _rho(G, st["x"][k], st["y"][k])
        out["lon"][k], out["lat"][k] = _dot(cb, G.lon_rho, o), _dot(cb, G.lat_rho, o)
    if case["diag"]:
        out.update({k: st[k] / len(steps) for k in ("salt", "temp")}, **{k: st[k] for k in ("hob", "bustr", "bvstr")})
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_adjoint(g, P, case, st, frames, seed):
    table = adj.step_table(case["nsteps"] * IDT / 86400.0, DT, IDT)[0]

    def go(state, it, kappa):
        a, auvw = _weights(it)
        g.set_time([frames[k - 1][0] for k in (it.frame_b, it.frame_c, it.frame_f)], a, auvw)
        _exact_step([g], None, None, P, case, state, it.step_index, seed + 1, kappa)

    saved = []
    for it in table:
        saved.append(dict(st))
        with torch.no_grad():
            go(st, it, 1.0)
    x, y = st["x"], st["y"]
    dx, dy = x - 0.5 * case["nx"], y - 0.5 * case["ny"]
    k = torch.exp(-(dx * dx + dy * dy) / 50.0)
    lam, dk = [-k * dx / 25.0, -k * dy / 25.0, torch.zeros_like(k)], 0.0
    for it, s in zip(reversed(table), reversed(saved)):
        lv = [s[c].clone().requires_grad_(True) for c in ("x", "y", "z")]
        kap = torch.ones((), dtype=F64, device=DEV, requires_grad=True)
        s = dict(s, x=lv[0], y=lv[1], z=lv[2])
        go(s, it, kap)
        gr = torch.autograd.grad([s["x"], s["y"], s["z"]], lv + [kap], lam, allow_unused=True)
        lam = [torch.zeros_like(k) if q is None else q for q in gr[:3]]
        dk += 0.0 if gr[3] is None else float(gr[3])
    out = {"x": x, "y": y, "z": st["z"], "dx": lam[0], "dy": lam[1], "dz": lam[2]}
    return {**{q: v.cpu().numpy() for q, v in out.items()}, "loss": float(k.sum()), "dk": dk}
