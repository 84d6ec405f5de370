"""The work this framework is used for, as cases that can be timed and checked.

A case of kind

* ``box`` is one output interval of a periodic two-beam (Weibel) run: a number
  of steps, then the energies and the fields as a run writes them (FP64 runs
  with ``particles`` also the particle arrays, as a restart file takes them);
* ``cyl`` is the same for the cylindrical plasma wakefield, on the theta grid
  or on the azimuthal modes 0 and 1;
* ``ensemble`` steps many small runs together and reads each one's energies
  and fields;
* ``adjoint`` is one forward run and its reverse sweep.

A pass goes on from where the last one left the run, as a simulation does.
What an FP32 run did to its particles shows in its fields and energies: the
particle arrays of that form have no order of their own to compare by.
``exact`` restates the steps in FP64 with plain torch, from the same initial
particles.  Runs of more than a few ten million particles are loaded by the
device's own loader and have no restatement (it would take minutes).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pictor_b200 import Particles, PicConfig, Simulation, init_scale
from pictor_b200.adjoint import Adjoint
from pictor_b200.simulation import Fields, step_many

COMPONENTS = ("Ex", "Ey", "Ez", "Bx", "By", "Bz")


def _box(name, nx, ny, nz, ppc, precision, **kw):
    """ppc: particles per cell and species; nz = 1 is a 2D run."""
    c = dict(name=name, kind="box", nx=nx, ny=ny, nz=nz, ppc=ppc, precision=precision, steps=20, drift=0.3,
             sigma=0.02, fdtd="yee", filter=0, exact_charge=0, particles=False, loader="host")
    c.update(kw)
    return c


def _cyl(name, nr, nz, precision, modes, **kw):
    c = dict(name=name, kind="cyl", nx=nr, ny=8, nz=nz, precision=precision, modes=modes, steps=20, thermal=0.01,
             bunch=1 << 16)
    c.update(kw)
    return c


def listed():
    return [
        # a parameter-scan run too small to fill the GPU: launches and latency
        _box("box2d_small_fp32", 64, 64, 1, 4, "fp32", drift=0.5, sigma=0.05),
        # a short FP64 verification run on a ragged grid, written out whole for a restart
        _box("box2d_small_fp64", 93, 70, 1, 8, "fp64", drift=0.5, sigma=0.05, fdtd="lehe", particles=True),
        # the 2D Weibel configuration in the reference's precision and layout
        _box("box2d_fp64", 256, 256, 1, 16, "fp64", drift=0.5, sigma=0.05),
        # a large 2D FP32 run, 12.6 M particles
        _box("box2d_fp32", 1024, 768, 1, 8, "fp32"),
        # a small ragged 3D FP32 run with the solver's options on: Lehe stencil, filtered and exactly
        # charge-conserving current, a fill that is no power of two
        _box("box3d_options_fp32", 67, 45, 37, 5, "fp32", fdtd="lehe", filter=2, exact_charge=1, sigma=0.05),
        # a 3D run in the reference's precision, 6.3 M particles
        _box("box3d_fp64", 96, 64, 64, 8, "fp64"),
        # the headline's plasma on 1/32 of its grid, 16.8 M particles
        _box("box3d_fp32", 128, 128, 64, 8, "fp32"),
        # the headline: 3D Weibel, 512 x 256 x 256 cells, 537 M particles
        _box("box3d_headline_fp32", 512, 256, 256, 8, "fp32", loader="device"),
        # plasma wakefield on modes 0 and 1, FP32 fields and particles, 8.4 M particles
        _cyl("cyl_modal_fp32", 128, 1024, "fp32", 2),
        # the same on the theta grid in the reference's precision
        _cyl("cyl_fp64", 64, 512, "fp64", 0),
        # a scan of 16 Weibel runs of uneven size stepped together
        dict(name="ensemble_fp32", kind="ensemble", runs=16, unit=32, precision="fp32", steps=20),
        # gradient of the magnetic energy of a 2D run with respect to the initial particles
        dict(name="adjoint_fp32", kind="adjoint", nx=128, ny=128, ppc=8, precision="fp32", steps=64, every=16,
             drift=0.4, sigma=0.05),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["box2", "box2", "box3", "box3", "box3", "cyl", "ensemble", "adjoint"])
    if kind in ("box2", "box3"):
        prec = rng.choice(["fp32", "fp32", "fp64"])
        ppc = rng.choice([2, 3, 4, 6, 8, 11, 16, 32 if kind == "box2" else 12])
        cells = _log(rng, 3000, 12e6 / ppc)
        if kind == "box2":
            nx = max(24, int(math.sqrt(cells) * rng.uniform(0.6, 1.6)))
            dims = (nx, max(24, cells // nx), 1)
        else:
            a = cells ** (1.0 / 3.0)
            nx, ny = max(13, int(a * rng.uniform(0.7, 1.8))), max(13, int(a * rng.uniform(0.7, 1.3)))
            dims = (nx, ny, max(13, cells // (nx * ny)))
        c = _box("", *dims, ppc, prec, drift=rng.choice([0.1, 0.3, 0.5, 0.9]), sigma=rng.choice([0.01, 0.03, 0.1]),
                 fdtd=rng.choice(["yee", "yee", "lehe"]), filter=rng.choice([0, 0, 0, 1, 3]),
                 exact_charge=int(prec == "fp32" and rng.random() < 0.25),
                 particles=prec == "fp64" and ppc * cells < 500000)
    elif kind == "cyl":
        c = _cyl("", _log(rng, 24, 160), _log(rng, 60, 1024), rng.choice(["fp32", "fp64"]), rng.choice([0, 2]))
    elif kind == "ensemble":
        c = dict(kind="ensemble", runs=rng.randint(3, 24), unit=rng.choice([24, 29, 32, 40]), precision="fp32", steps=20)
    else:
        c = dict(kind="adjoint", nx=_log(rng, 24, 160), ny=_log(rng, 24, 160), ppc=rng.choice([2, 5, 8]),
                 precision=rng.choice(["fp32", "fp64"]), steps=rng.choice([20, 40, 64]), every=rng.choice([7, 16]),
                 drift=rng.choice([0.2, 0.4]), sigma=0.05)
    c.pop("name", None)
    return c


# --- initial particles (torch, on the GPU, FP64) -------------------------------
def _beams(nx, ny, nz, ppc, drift, sigma, seed):
    """Two counter-streaming neutral beams along x: every ion sits on an
    electron, half of each pair set moves with +drift and half with -drift.
    Positions in cells from the first interior cell (2D: z in [0, 1))."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = ppc * nx * ny * nz
    size = torch.tensor([nx, ny, nz], dtype=torch.float64, device="cuda")[:, None]
    pos = torch.rand((3, n), generator=g, dtype=torch.float64, device="cuda") * size
    sign = torch.where(torch.arange(n, device="cuda") % 2 == 0, 1.0, -1.0).double()
    gamma = 1.0 / math.sqrt(1.0 - drift * drift)
    out = []
    for _ in range(2):
        u = torch.randn((3, n), generator=g, dtype=torch.float64, device="cuda") * sigma
        u[0] += sign * (gamma * drift)
        out.append(u)
    pos, u = torch.cat([pos, pos], 1), torch.cat(out, 1)
    q = torch.cat([torch.ones(n, dtype=torch.float64, device="cuda"), -torch.ones(n, dtype=torch.float64, device="cuda")])
    flv = torch.cat([torch.full((n,), 1, dtype=torch.int32, device="cuda"),
                     torch.full((n,), 2, dtype=torch.int32, device="cuda")])
    return q, pos, u, flv


def _plasma(case, seed):
    """Electrons placed evenly, 2 x 2 x 2 per cell, weights growing with the
    radius, and a Gaussian bunch (gamma = 50) on the axis; positions in cells
    from the first interior cell, whose radius is -1/2."""
    nr, nt, nz, c = case["nx"], case["ny"], case["nz"], 0.3
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    ax = [(torch.arange(2 * n, dtype=torch.float64, device="cuda") + 0.5) / 2 for n in (nr, nt, nz)]
    X, Y, Z = (a.reshape(-1) for a in torch.meshgrid(*ax, indexing="ij"))
    keep = X > 0.5
    X, Y, Z = X[keep], Y[keep], Z[keep]
    dth = 2.0 * math.pi / nt
    wt = (X - 0.5) * dth
    u = torch.randn((3, X.numel()), generator=g, dtype=torch.float64, device="cuda") * (case["thermal"] * c)
    m, sr, sz = case["bunch"], nr / 12.0, nz / 40.0
    b = torch.randn((3, m), generator=g, dtype=torch.float64, device="cuda")
    bx, by, bz = b[0] * sr, b[1] * sr, b[2] * sz + 0.3 * nz
    r = torch.hypot(bx, by)
    th = torch.remainder(torch.atan2(by, bx), 2.0 * math.pi) / dth
    ok = (r < nr - 2.0) & (bz >= 0) & (bz < nz) & (th < nt)
    r, th, bz = r[ok], th[ok], bz[ok]
    wb = torch.full_like(r, 0.1 * 8 * (2.0 * math.pi) ** 1.5 * sr * sr * sz / m)
    ub = torch.zeros((3, r.numel()), dtype=torch.float64, device="cuda")
    ub[2] = c * math.sqrt(50.0 * 50.0 - 1.0)
    pos = torch.stack([torch.cat([X, r + 0.5]), torch.cat([Y, th]), torch.cat([Z, bz])])
    q = -torch.cat([wt, wb])
    return q, pos, torch.cat([u, ub], 1), torch.full((q.numel(),), 2, dtype=torch.int32, device="cuda")


def _host(q, pos, u, flv, low):
    a = [t.cpu().numpy() for t in (q, pos[0] + low[0], pos[1] + low[1], pos[2] + low[2], u[0], u[1], u[2], flv)]
    return Particles(*a)


def _pinned_fields(shape):
    n = shape[0] * shape[1] * shape[2]
    buf = torch.empty((6, n), dtype=torch.float64, pin_memory=True).numpy()
    return Fields(*(buf[k].reshape(shape, order="F") for k in range(6)))


# --- prepare / run ------------------------------------------------------------
CARTESIAN, CYL = 0.45, 0.3


def _units(case):
    """Courant number, skin depth in cells, particles per cell and species."""
    return (CYL, 10.0, 8) if case["kind"] == "cyl" else (CARTESIAN, 2.0, case["ppc"])


def _scale(case):
    return _units(case)[0], init_scale(*_units(case))


def _make_box(case, seed):
    c, sc = _scale(case)
    dims = 3 if case["nz"] > 1 else 2
    n = 2 * case["ppc"] * case["nx"] * case["ny"] * case["nz"]
    # the FP64 form appends the wrapped particles until the next reorder
    cap = int(n * (1.04 if case["precision"] == "fp32" else 1.5)) + (1 << 16)
    sim = Simulation(PicConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], dims=dims, c=c, qi=sc["qi"],
                               precision=case["precision"], fdtd=case["fdtd"], capacity=cap, reorder_period=20,
                               curr_filter=case["filter"], exact_charge=case["exact_charge"]))
    if case["loader"] == "device":
        t = 2.0 * case["sigma"] ** 2
        sim.init_weibel(case["ppc"], 0.5, case["drift"], t, t, int(seed) & 0x7FFFFFFF)
    else:
        p = _beams(case["nx"], case["ny"], case["nz"], case["ppc"], case["drift"], case["sigma"], seed)
        sim.load_particles(_host(*p, (3.0, 3.0, 3.0 if dims == 3 else 1.0)))
    sim.reorder()
    return sim, sc


def _ensemble_runs(case):
    u, out = case["unit"], []
    for r in range(case["runs"]):
        out.append(_box("", u * (2 + (5 * r) % 7), u * (2 + (3 * r) % 5), 1, (4, 8, 16, 12)[r % 4], case["precision"],
                        drift=0.1 + 0.8 * ((7 * r) % 16) / 16.0, sigma=0.01 + 0.09 * ((3 * r) % 8) / 8.0,
                        steps=case["steps"]))
    return out


def prepare(case, seed):
    if case["kind"] == "box":
        sim, sc = _make_box(case, seed)
        return {"case": case, "sim": sim, "masse": sc["masse"], "out": _pinned_fields(sim.cfg.shape)}
    if case["kind"] == "cyl":
        c, sc = _scale(case)
        p = _plasma(case, seed)
        sim = Simulation(PicConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], dims=3, c=c, qi=sc["qi"], fdtd="lehe",
                                   geom="cylindrical", precision=case["precision"], capacity=2 * p[0].numel() + 4096,
                                   reorder_period=20, rmin=-0.5, inc_axis=1, cyl_modes=case["modes"]))
        sim.load_particles(_host(*p, (3.0, 3.0, 3.0)))
        sim.reorder()
        return {"case": case, "sim": sim, "masse": sc["masse"], "out": _pinned_fields(sim.cfg.shape)}
    if case["kind"] == "ensemble":
        made = [_make_box(b, int(seed) + 7919 * k) for k, b in enumerate(_ensemble_runs(case))]
        return {"case": case, "sims": [s for s, _ in made], "masse": [sc["masse"] for _, sc in made],
                "out": [_pinned_fields(s.cfg.shape) for s, _ in made]}
    c, sc = _scale(case)
    n = 2 * case["ppc"] * case["nx"] * case["ny"]
    adj = Adjoint(PicConfig(nx=case["nx"], ny=case["ny"], dims=2, c=c, qi=sc["qi"], precision=case["precision"],
                            capacity=n + 4096, reorder_period=0))
    p = _beams(case["nx"], case["ny"], 1, case["ppc"], case["drift"], case["sigma"], seed)
    adj.load_particles(_host(*p, (3.0, 3.0, 1.0)))
    return {"case": case, "adj": adj}


def _energies(d):
    # the Gauss residual is rounding noise of the field updates and is left out
    return np.array([d["B2"], d["E2"], *(k for k in d["kinetic"] if k != 0.0)])


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        j = state["adj"].forward(case["steps"], case["every"])
        g = state["adj"].gradient()
        return {"objective": np.array([j]), **{k: g[k] for k in ("u", "v", "w", "x", "y")}}
    if case["kind"] == "ensemble":
        step_many(state["sims"], case["steps"])
        out = {"energy": [], "fields": []}
        for sim, masse, buf in zip(state["sims"], state["masse"], state["out"]):
            out["energy"].append(_energies(sim.diagnostics(masse)))
            f = sim.fetch_fields(False, out=buf)
            out["fields"].append(np.stack([getattr(f, k).T.reshape(-1) for k in COMPONENTS]))
        out["energy"] = np.stack(out["energy"])
        return out
    sim = state["sim"]
    sim.step(case["steps"])
    d = sim.diagnostics(state["masse"])
    f = sim.fetch_fields(False, out=state["out"])
    out = {"energy": _energies(d), **{k: getattr(f, k).T for k in COMPONENTS}}
    if case["kind"] == "box":
        out["rho_max"] = np.array([d["rho_max"]])
        if case["particles"]:
            p = sim.fetch_particles()
            out["particles"] = {k: getattr(p, k) for k in Particles.NAMES}
    return out


def work(case):
    """Bytes: every step reads and writes the particle state and the fields
    once (the state of all but the smallest runs is larger than any cache),
    and the pass writes its output once.  Flops: gather, push and deposit of a
    particle, counted from the formulas."""
    if case["kind"] == "ensemble":
        w = [work(b) for b in _ensemble_runs(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    fp32 = case["precision"] == "fp32"
    word = 4 if fp32 else 8
    nz = case.get("nz", 1)
    cells = case["nx"] * case["ny"] * nz
    n = 8.0 * cells if case["kind"] == "cyl" else 2.0 * case["ppc"] * cells
    part = (60 if nz > 1 else 52) if fp32 else 108
    flops = 250 if nz > 1 else 160
    if case["kind"] == "adjoint":
        # forward, recomputation and reverse sweep of every step
        return {"bytes": 3 * case["steps"] * (n * 12 * word + cells * 12 * word) + n * 40, "flops": 5.0 * case["steps"] * n * flops}
    out = 6 * 8 * cells + (60 * n if case.get("particles") else 0)
    if case["kind"] == "cyl":
        flops *= 2
    # fields: both B half steps read E and B and write B, the E step reads E, B, J and writes E; J written once
    return {"bytes": case["steps"] * (n * part + cells * 33 * word) + out, "flops": float(case["steps"]) * n * flops}


def tolerance(case):
    """About four times the largest distance of an output from ``exact`` over
    the listed and some drawn cases.  The weakest components (Bx of a box, Bz
    of the wakefield) carry the rounding of the strong ones: FP32 boxes are
    up to 5e-4 off, the FP32 wakefield 9e-4, the FP32 gradient 1.5e-2 (the
    reverse sweep amplifies the rounding as the run does), FP64 boxes and
    gradients up to 5e-13 and the FP64 wakefield 6e-11 (atomic sums, and the
    small steps next to the axis)."""
    if case["precision"] == "fp64":
        return {"rel": 5e-10 if case["kind"] == "cyl" else 1e-11}
    return {"rel": {"box": 2e-3, "ensemble": 2e-3, "cyl": 4e-3, "adjoint": 3e-2}[case["kind"]]}


# --- the same steps in FP64 with plain torch ----------------------------------
def _r(F, ax, s):
    """F at index + s along axis ax (0 = x, 1 = y, 2 = z) of a periodic (nz, ny, nx) grid."""
    return torch.roll(F, -s, dims=2 - ax)


def _charge(case):
    """Courant number and the charge (and mass) of a particle of unit weight, ions as heavy as electrons."""
    c, skin, epc = _units(case)
    return c, (c / skin) ** 2 / (2.0 * epc)


def _lehe(dims, c):
    s = math.sin(0.5 * math.pi * c)
    dx = 0.25 * (1.0 - s * s / (c * c))
    if dims == 3:
        return {"a": (1 - 0.25 - 0.25 - 3 * dx, 1 - 0.25, 1 - 0.25), "b": {(0, 1): 0.125, (0, 2): 0.125, (1, 0): 0.125, (1, 2): 0.0,
                                                                      (2, 0): 0.125, (2, 1): 0.0}, "d": (dx, 0.0, 0.0)}
    return {"a": (1 - 0.25 - 3 * dx, 1 - 0.25, 1.0), "b": {(0, 1): 0.125, (1, 0): 0.125}, "d": (dx, 0.0, 0.0)}


def _grad(F, ax, L):
    """Forward difference along ax, with Lehe's transverse and long-range terms when L is given."""
    D = _r(F, ax, 1) - F
    if L is None:
        return D
    out = L["a"][ax] * D + L["d"][ax] * (_r(F, ax, 2) - _r(F, ax, -1))
    for (a, t), b in L["b"].items():
        if a == ax and b:
            out = out + b * (_r(D, t, 1) + _r(D, t, -1))
    return out


def _bhalf(E, B, h, dims, L):
    Ex, Ey, Ez = E
    Bx, By, Bz = B
    bx = Bx - h * _grad(Ez, 1, L)
    by = By + h * _grad(Ez, 0, L)
    if dims == 3:
        bx, by = bx + h * _grad(Ey, 2, L), by - h * _grad(Ex, 2, L)
    return [bx, by, Bz - h * _grad(Ey, 0, L) + h * _grad(Ex, 1, L)]


def _estep(E, B, J, fc, dims):
    Bx, By, Bz = B
    ex = E[0] + fc * (Bz - _r(Bz, 1, -1)) - J[0]
    ey = E[1] - fc * (Bz - _r(Bz, 0, -1)) - J[1]
    ez = E[2] + fc * (By - _r(By, 0, -1)) - fc * (Bx - _r(Bx, 1, -1)) - J[2]
    if dims == 3:
        ex, ey = ex - fc * (By - _r(By, 2, -1)), ey + fc * (Bx - _r(Bx, 2, -1))
    return [ex, ey, ez]


def _nodes(E, B, dims):
    """Node averages of the staggered fields, (cells, 6)."""
    def av(F, *axes):
        for a in axes:
            if a < dims:
                F = 0.5 * (F + _r(F, a, -1))
        return F
    return torch.stack([av(E[0], 0), av(E[1], 1), av(E[2], 2), av(B[0], 1, 2), av(B[1], 0, 2), av(B[2], 0, 1)], -1).reshape(-1, 6)


def _corners(n, dims, cell, d):
    """Flat indices and trilinear weights of the corners of each particle's cell."""
    for c in range(1 << dims):
        bit = [(c >> a) & 1 for a in range(dims)]
        ix = [torch.remainder(cell[a] + bit[a], n[a]) for a in range(dims)]
        flat = ix[0] + n[0] * (ix[1] + (n[1] * ix[2] if dims == 3 else 0))
        w = 1.0
        for a in range(dims):
            w = w * (d[a] if bit[a] else 1.0 - d[a])
        yield flat, w


def _boris(c, pE, pB, u):
    """Half kick, rotation, half kick of momenta u (in units of c); returns new momenta and displacement factor."""
    u0 = c * u + pE
    t = pB / torch.sqrt(c * c + (u0 * u0).sum(0))
    s = 2.0 / (1.0 + (t * t).sum(0))
    u1 = (u0 + torch.linalg.cross(u0, t, dim=0)) * s
    u0 = u0 + torch.linalg.cross(u1, t, dim=0) + pE
    return u0, c * c / torch.sqrt(c * c + (u0 * u0).sum(0))


def _relay(a, b):
    i, j = torch.floor(a.detach()), torch.floor(b.detach())
    return torch.minimum(torch.minimum(i, j) + 1.0, torch.maximum(torch.maximum(i, j), 0.5 * (a + b)))


def _segment(n, dims, a, b, base, q, xc):
    """(component, flat index, value) of the current of the straight segment a -> b inside cell `base`."""
    F = [q * (b[k] - a[k]) for k in range(3)]
    W = [0.5 * (a[k] + b[k]) - base[k] for k in range(dims)]
    C = F[0] * (b[1] - a[1]) * (b[2] - a[2]) / 12.0 if xc else None
    ib = [base[k].long() for k in range(dims)]
    for comp in range(3):
        axes = [k for k in range(dims) if k != comp]
        for m in range(1 << len(axes)):
            ix, w, sign = list(ib), F[comp], 1.0
            for p, k in enumerate(axes):
                hit = (m >> p) & 1
                ix[k] = ix[k] + hit
                w = w * (W[k] if hit else 1.0 - W[k])
                sign = -sign if hit else sign
            if xc:
                w = w + sign * C
            ix = [torch.remainder(ix[k], n[k]) for k in range(dims)]
            yield comp, ix[0] + n[0] * (ix[1] + (n[1] * ix[2] if dims == 3 else 0)), w


def _box_steps(case, seed, grad=False):
    """FP64 steps; returns fields, particles, energies; with grad the inputs keep their graph and the objective is summed."""
    c, qi = _charge(case)
    nz = case.get("nz", 1)
    dims = 3 if nz > 1 else 2
    n = (case["nx"], case["ny"], nz)
    q, pos, u, flv = _beams(*n, case["ppc"], case["drift"], case["sigma"], seed)
    if grad:
        pos, u = pos.requires_grad_(), u.requires_grad_()
        leaf = (pos, u)
    x = [pos[k] for k in range(3)]
    qm = torch.where(flv == 1, 1.0, -1.0).double()
    fp64_z = dims == 2 and case["precision"] == "fp64" and not grad
    L = _lehe(dims, c) if case.get("fdtd") == "lehe" else None
    zero = torch.zeros((nz, n[1], n[0]), dtype=torch.float64, device="cuda")
    E, B, obj = [zero] * 3, [zero] * 3, 0.0
    for _ in range(case["steps"]):
        B = _bhalf(E, B, 0.5 * c, dims, L)
        cell = [torch.floor(x[k].detach()).long() for k in range(dims)]
        d = [x[k] - cell[k] for k in range(dims)]
        V, F6 = _nodes(E, B, dims), 0.0
        for flat, w in _corners(n, dims, cell, d):
            F6 = F6 + w[:, None] * V[flat]
        F6 = F6.T * (0.5 * qm)
        u0, gg = _boris(c, F6[:3], F6[3:], u)
        u = u0 / c
        new = [x[k] + u[k] * gg for k in range(3)]
        mid = [_relay(x[k], new[k]) if k < dims or fp64_z else 0.5 * (x[k] + new[k]) for k in range(3)]
        J = [torch.zeros(zero.numel(), dtype=torch.float64, device="cuda") for _ in range(3)]
        qq = q * qi
        for a, b, at in ((x, mid, x), (mid, new, new)):
            for comp, flat, w in _segment(n, dims, a, b, [torch.floor(at[k].detach()) for k in range(dims)], qq,
                                          dims == 3 and case.get("exact_charge")):
                J[comp] = J[comp].index_add(0, flat, w) if grad else J[comp].index_add_(0, flat, w)
        J = [j.reshape(zero.shape) for j in J]
        x = [new[k] - n[k] * torch.floor(new[k].detach() / n[k]) for k in range(3)]
        B = _bhalf(E, B, 0.5 * c, dims, L)
        for _f in range(case.get("filter", 0)):
            for a in range(dims):
                J = [0.25 * _r(j, a, -1) + 0.5 * j + 0.25 * _r(j, a, 1) for j in J]
        E = _estep(E, B, J, c, dims)
        if grad:
            obj = obj + 0.5 * sum((b * b).sum() for b in B)
    if grad:
        gp, gu = torch.autograd.grad(obj, leaf)
        return {"objective": obj.detach().reshape(1), "u": gu[0], "v": gu[1], "w": gu[2], "x": gp[0], "y": gp[1]}
    wt = [torch.tensor([sum(float((b * b).sum()) for b in F)], dtype=torch.float64) for F in (B, E)]
    gm = torch.sqrt(1.0 + (u * u).sum(0)) - 1.0
    rho = torch.zeros(zero.numel(), dtype=torch.float64, device="cuda")
    cell = [torch.floor(x[k]).long() for k in range(dims)]
    for flat, w in _corners(n, dims, cell, [x[k] - cell[k] for k in range(dims)]):
        rho.index_add_(0, flat, w * torch.clamp(q, min=0.0) * qi)
    kin = [float((gm * (flv == f)).sum()) * qi * c * c for f in (1, 2)]
    return {"E": E, "B": B, "energy": torch.tensor([float(wt[0]), float(wt[1]), *kin], dtype=torch.float64),
            "rho_max": rho.max().reshape(1)}


def _ghosted(F, n, dims):
    for a in range(dims):
        F = torch.index_select(F, 2 - a, torch.remainder(torch.arange(-2, n[a] + 3, device=F.device), n[a]))
    return F


def _box_exact(case, seed):
    r = _box_steps(case, seed)
    n, dims = (case["nx"], case["ny"], case["nz"]), 3 if case["nz"] > 1 else 2
    fields = [_ghosted(F, n, dims) for F in (*r["E"], *r["B"])]
    out = {"energy": r["energy"], **dict(zip(COMPONENTS, fields)), "rho_max": r["rho_max"]}
    if case["particles"]:
        out["particles"] = None   # their order in the arrays is the library's
    return out


# The cylinder: arrays (mz, my, mx) with the ghost layers (2 low, 3 high);
# index i of r stands at radius i - 2 - 1/2 (0-based), the axis at i = 2.5.
class _Cyl:
    def __init__(self, case):
        self.nr, self.nt, self.nz = case["nx"], case["ny"], case["nz"]
        self.m = (self.nr + 5, self.nt + 5, self.nz + 5)
        self.c, self.qi = _charge(case)
        self.dth = 2.0 * math.pi / self.nt
        i = torch.arange(self.m[0], dtype=torch.float64, device="cuda")
        self.r = i - 2.5
        p = torch.arange(self.m[1], device="cuda") + self.nt // 2
        self.partner = torch.where(p > self.m[1] - 4, p - self.nt, p)   # the cell across the axis
        s = math.sin(0.5 * math.pi * self.c)
        dz = 0.25 * (1.0 - s * s / self.c ** 2)
        self.beta, self.bz_y, self.dz = 0.125, 0.125 / self.dth ** 2, dz
        self.az = 1.0 - 2 * 0.125 - 2 * self.bz_y - 3 * dz

    def zeros(self):
        return [torch.zeros(self.m[::-1], dtype=torch.float64, device="cuda") for _ in range(3)]

    def halo(self, F):
        jt = torch.remainder(torch.arange(-2, self.nt + 3, device="cuda"), self.nt) + 2
        kz = torch.remainder(torch.arange(-2, self.nz + 3, device="cuda"), self.nz) + 2
        return [f[kz][:, jt] for f in F]

    def gx(self, F, w=None):
        G = F if w is None else w * F
        D = _r(G, 0, 1) - G
        return (1 - 2 * self.beta) * D + self.beta * (_r(D, 2, 1) + _r(D, 2, -1))

    def gy(self, F):
        D = _r(F, 1, 1) - F
        return (1 - 2 * self.beta) * D + self.beta * (_r(D, 2, 1) + _r(D, 2, -1))

    def gz(self, F):
        D = _r(F, 2, 1) - F
        return (self.az * D + self.beta * (_r(D, 0, 1) + _r(D, 0, -1)) + self.bz_y * (_r(D, 1, 1) + _r(D, 1, -1)) +
                self.dz * (_r(F, 2, 2) - _r(F, 2, -1)))

    def bhalf(self, E, B):
        h, r, s = 0.5 * self.c, self.r, slice(3, self.m[0] - 1)
        Ex, Ey, Ez = E
        B = [b.clone() for b in B]
        axis = -h * (4.0 / self.nt) * Ey[:, 2:-3, 3].sum(1)
        B[0][..., s] += (-h * self.gy(Ez) / (r * self.dth) + h * self.gz(Ey))[..., s]
        B[1][..., s] += (-h * self.gz(Ex) + h * self.gx(Ez))[..., s]
        B[2][..., s] -= (h * (self.gx(Ey, r) - self.gy(Ex) / self.dth) / (r + 0.5))[..., s]
        B[2][..., 2] = (B[2][:, 2, 2] + axis)[:, None]
        p = self.partner
        B[1][..., 2] = 0.5 * (B[1][..., 3] - B[1][:, p, 3])
        B[1][..., 1] = -B[1][:, p, 3]
        B[0][..., 2] = -B[0][:, p, 3]
        B[2][..., 1] = B[2][:, p, 3]
        return self.halo(B)

    def e_axis(self, E):
        p = self.partner
        E[0][..., 2] = 0.5 * (E[0][..., 3] - E[0][:, p, 3])
        E[0][..., 1] = -E[0][:, p, 3]
        E[1][..., 2] = -E[1][:, p, 3]
        E[2][..., 2] = E[2][:, p, 3]
        return self.halo(E)

    def estep(self, E, B):
        c, r, s = self.c, self.r, slice(3, self.m[0] - 3)
        Bx, By, Bz = B
        E = [e.clone() for e in E]
        E[0][..., s] += (c * (Bz - _r(Bz, 1, -1)) / ((r + 0.5) * self.dth) - c * (By - _r(By, 2, -1)))[..., s]
        E[1][..., s] += (c * (Bx - _r(Bx, 2, -1)) - c * (Bz - _r(Bz, 0, -1)))[..., s]
        E[2][..., s] += (c * ((r + 0.5) * By - _r((r + 0.5) * By, 0, -1)) / r -
                         c * (Bx - _r(Bx, 1, -1)) / (r * self.dth))[..., s]
        return self.e_axis(E)

    def add_current(self, E, J):
        r, s = self.r, slice(3, self.m[0] - 3)
        for k, w in enumerate(((r + 0.5) * self.dth, torch.ones_like(r), r * self.dth)):
            E[k][..., s] -= (J[k] / w)[..., s]
        return self.e_axis(E)

    def fold(self, J, modes):
        """Periodic images in theta and z added, the modes above 1 taken out when asked."""
        out = []
        for j in J:
            for dim, n in ((0, self.nz), (1, self.nt)):
                idx = torch.remainder(torch.arange(-2, n + 3, device="cuda"), n)
                j = torch.zeros((n, *j.shape[1:]) if dim == 0 else (j.shape[0], n, j.shape[2]), dtype=j.dtype,
                                device="cuda").index_add_(dim, idx, j)
            if modes:
                f = torch.fft.rfft(j, dim=1)
                f[:, modes:] = 0
                j = torch.fft.irfft(f, n=self.nt, dim=1)
            pad = torch.zeros(self.m[::-1], dtype=j.dtype, device="cuda")
            pad[2:-3, 2:-3] = j
            out.append(pad)
        return out

    def gather(self, V, x, y, z):
        out, cell = 0.0, [torch.floor(a).long() for a in (x, y, z)]
        d = [a - b for a, b in zip((x, y, z), cell)]
        for c in range(8):
            b = [(c >> k) & 1 for k in range(3)]
            w = 1.0
            for k in range(3):
                w = w * (d[k] if b[k] else 1.0 - d[k])
            flat = (cell[0] + b[0]) + self.m[0] * ((cell[1] + b[1]) + self.m[1] * (cell[2] + b[2]))
            out = out + w[:, None] * V[flat]
        return out.T

    def kick(self, F6, u0):
        t = F6[3:] / torch.sqrt(self.c ** 2 + (u0 * u0).sum(0))
        s = 2.0 / (1.0 + (t * t).sum(0))
        u1 = (u0 + torch.linalg.cross(u0, t, dim=0)) * s
        return u0 + torch.linalg.cross(u1, t, dim=0) + F6[:3]

    def deposit(self, J, a, b, q, second_in_first):
        mid = [_relay(a[k], b[k]) for k in range(3)]
        base = [torch.floor(v) for v in a]
        for p, e, at in ((a, mid, a), (mid, b, b)):
            own = [torch.floor(v) for v in at]
            # the weights belong to the segment's own cell; the main mover adds both segments to the first's cell
            to = base if second_in_first else own
            shift = [to[k] - own[k] for k in range(3)]
            for comp, ix, w in _segment_cells([p[k] + shift[k] for k in range(3)], [e[k] + shift[k] for k in range(3)], to, q):
                J[comp].view(-1).index_add_(0, ix[0] + self.m[0] * (ix[1] + self.m[1] * ix[2]), w)

    def substeps(self, V, J, x, u, q):
        """The particles near the axis, moved in steps that turn at most 0.45 theta cells."""
        c, qm = self.c, -0.25
        t, dt = torch.zeros_like(q), torch.ones_like(q)
        u, on = u.clone(), torch.ones_like(q, dtype=torch.bool)
        while bool(on.any()):
            k = on.nonzero()[:, 0]
            xs, us, h = [a[k] for a in x], u[:, k], torch.minimum(dt[k], 1.0 - t[k])
            F6 = self.gather(V, *xs) * qm * h
            u0 = self.kick(F6, c * us + F6[:3])
            u1, v1, w1 = u0[0] / c, u0[1] / c, u0[2] / c
            gg = c * c / torch.sqrt(c * c + (u0 * u0).sum(0))
            r0 = xs[0] - 2.5
            x1, y1 = r0 + u1 * gg * h, v1 * gg * h
            r1 = torch.sqrt(x1 * x1 + y1 * y1)
            turn = torch.where(x1 > 0, torch.atan(y1 / x1) / self.dth, torch.zeros_like(x1))
            ok = turn.abs() <= 0.45
            front = x1 > 0
            nx = torch.where(front, r1, x1) + 2.5
            a = torch.where(front, (r0 * u0[0] + (u0[0] * u1 * gg * h + u0[1] * y1)) / r1, u1)
            b = torch.where(front, u0[1] * r0 / r1, v1)
            new = [nx, xs[1] + turn, xs[2] + w1 * gg * h]
            F6 = self.gather(V, *[torch.where(ok, n, o) for n, o in zip(new, xs)]) * qm * h
            u2 = self.kick(F6, torch.stack([a, b, u0[2]]) + F6[:3]) / c
            g, kg = ok, k[ok]
            self.deposit(J, [a_[g] for a_ in xs], [n[g] for n in new], q[kg], False)
            over = new[0] < 2.5
            new[0] = torch.where(over, 5.0 - new[0], new[0])
            new[1] = new[1] + torch.where(over, 0.5 * self.nt, 0.0)
            u2 = torch.stack([torch.where(over, -u2[0], u2[0]), torch.where(over, -u2[1], u2[1]), u2[2]])
            new[1] = torch.where(new[1] > self.nt + 2.0, new[1] - self.nt, new[1])
            new[1] = torch.where(new[1] < 2.0, new[1] + self.nt, new[1])
            for a_, n in zip(x, new):
                a_[kg] = n[g]
            u[:, kg] = u2[:, g]
            t[kg] += h[g]
            dt[k] = torch.where(ok, dt[k] * 1.7, dt[k] * 0.5)
            on = t < 1.0
        return x, u

    def move(self, E, B, x, u, q):
        c, qm = self.c, -0.25
        V = _nodes(E, B, 3)
        J = self.zeros()
        F6 = self.gather(V, *x) * qm
        u0 = self.kick(F6, c * u + F6[:3])
        u1, v1 = u0[0] / c, u0[1] / c
        gg = c * c / torch.sqrt(c * c + (u0 * u0).sum(0))
        r0 = x[0] - 2.5
        x1, y1 = r0 + u1 * gg, v1 * gg
        r1 = torch.sqrt(x1 * x1 + y1 * y1)
        near = x[0] < 3.5
        new = [r1 + 2.5, x[1] + torch.atan(y1 / x1) / self.dth, x[2] + u[2] * gg]
        new = [torch.where(near, o, n) for n, o in zip(new, x)]
        a = (r0 * u0[0] + (u0[0] * u1 * gg + u0[1] * y1)) / r1
        b = u0[1] * r0 / r1
        F6 = self.gather(V, *new) * qm
        un = self.kick(F6, torch.stack([a, b, u0[2]]) + F6[:3]) / c
        qq, far = q * self.qi, ~near
        self.deposit(J, [v[far] for v in x], [v[far] for v in new], qq[far], True)
        if bool(near.any()):
            xs, us = self.substeps(V, J, [v[near].clone() for v in x], u[:, near], qq[near])
            for v, s in zip(new, xs):
                v[near] = s
            un[:, near] = us
        J[1][..., 3] -= J[1][..., 2]
        J[2][..., 3] -= J[2][..., 2]
        J[0][..., 2] = 0
        J[1][..., 1] = 0
        J[2][..., 1] = 0
        keep = (new[0] <= self.nr + 2.0) & (new[0] >= 2.0)
        new = [v[keep] for v in new]
        for k, n in ((1, self.nt), (2, self.nz)):
            new[k] = torch.remainder(new[k] - 2.0, n) + 2.0
        return J, new, un[:, keep], q[keep]


def _segment_cells(a, b, base, q):
    F = [q * (b[k] - a[k]) for k in range(3)]
    W = [0.5 * (a[k] + b[k]) - base[k] for k in range(3)]
    ib = [v.long() for v in base]
    for comp in range(3):
        axes = [k for k in range(3) if k != comp]
        for m in range(4):
            ix, w = list(ib), F[comp]
            for p, k in enumerate(axes):
                hit = (m >> p) & 1
                ix[k] = ix[k] + hit
                w = w * (W[k] if hit else 1.0 - W[k])
            yield comp, ix, w


def _cyl_exact(case, seed):
    S = _Cyl(case)
    q, pos, u, _ = _plasma(case, seed)
    x = [pos[k] + 2.0 for k in range(3)]
    E, B = S.zeros(), S.zeros()
    for _ in range(case["steps"]):
        B = S.bhalf(E, B)
        J, x, u, q = S.move(E, B, x, u, q)
        B = S.bhalf(E, B)
        E = S.estep(E, B)
        E = S.add_current(E, S.fold(J, case["modes"]))
    r, c = S.r[3:-3], S.c
    I = (slice(2, -3), slice(2, -3), slice(3, -3))
    en = [float(sum((w * f[I] ** 2).sum() for w, f in zip(ws, F))) * S.dth
          for ws, F in (((r, r + 0.5, r + 0.5), B), ((r + 0.5, r, r), E))]
    kin = float(((torch.sqrt(1.0 + (u * u).sum(0)) - 1.0) * q.abs()).sum()) * S.qi * c * c
    return {"energy": torch.tensor([*en, kin], dtype=torch.float64), **dict(zip(COMPONENTS, (*E, *B)))}


def exact(case, seed):
    if case["kind"] == "cyl":
        return _cyl_exact(case, seed)
    if case["kind"] == "adjoint":
        return _box_steps(case, seed, grad=True)
    if case["kind"] == "ensemble":
        out = {"energy": [], "fields": []}
        for k, b in enumerate(_ensemble_runs(case)):
            r = _box_exact(b, int(seed) + 7919 * k)
            out["energy"].append(r["energy"])
            out["fields"].append(torch.stack([r[n].reshape(-1) for n in COMPONENTS]))
        out["energy"] = torch.stack(out["energy"])
        return out
    if case["loader"] == "device":
        return None
    return _box_exact(case, seed)
