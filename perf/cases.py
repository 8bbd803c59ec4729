"""Cases for timing the library through its public entry points.

A case is one call a user's program makes on a model it has set up: a formal solve
(device buffers or the drop-in ``core.Model`` call), the level-population loop, an
image, a batch of models, or a forward + backward pass of the differentiable imager or
formal solve.  Geometries are those of ``magritte_gb300.synthetic``; they do not depend
on the seed and are kept per process, the fields on them (velocity, temperature) are
drawn from the seed.
"""
import ctypes as C
import math
from dataclasses import replace
from functools import lru_cache

import numpy as np
import torch

from magritte_gb300 import _abi, adjoint, healpix, loader, synthetic

CC = 2.99792458e8
CC_SQUARED = 8.98755179e16  # as the library's constant
HH = 6.62607004e-34
KB = 1.38064852e-23
AMU = 1.66053904e-27
T_CMB = 2.72548

# The formal-solve parameters of core.Parameters that exact() restates.
MAX_WIDTH_FRACTION = 0.35
MIN_OPACITY = 1.0e-26
MIN_LINE_OPACITY = 1.0e-13
MIN_LINE_EMISSIVITY = 1.0e-50
MAX_INTERPOLATION_DIFF = 1.4
MAX_DISTANCE = 10.0


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a test-sized cube, where launches and latency count
        dict(name="cube10_fp64", family="solve", geometry="cube", n=10, nside=1, nlev=2, nquads=5,
             precision="fp64", approx="CloseLines", entry="device"),
        # the plain FP64 workload (20^3 cube, 12 rays, one line x 11) as the drop-in call, results on the host
        dict(name="cube20_fp64_host", family="solve", geometry="cube", n=20, nside=1, nlev=2, nquads=11,
             precision="fp64", approx="CloseLines", entry="host"),
        # the benchmark's family at a middle, odd size
        dict(name="sphere33_split", family="solve", geometry="sphere", n=33, nside=2, nlev=5, nquads=31,
             precision="split", approx="CloseLines", entry="device"),
        # the benchmark itself: the largest formal solve
        dict(name="sphere64_split", family="solve", geometry="sphere", n=64, nside=2, nlev=5, nquads=31,
             precision="split", approx="CloseLines", entry="device"),
        # the reference's own arithmetic on the same family
        dict(name="sphere24_fp64", family="solve", geometry="sphere", n=24, nside=2, nlev=5, nquads=31,
             precision="fp64", approx="CloseLines", entry="device"),
        # a 1D spherically symmetric model (200 shells, 50 rays, 50 quadrature points), drop-in call
        dict(name="shells200_fp64", family="shells", npoints=200, nrays=50, nquads=50, precision="fp64"),
        # short characteristics on a small sphere cutout, results on the host
        dict(name="shortchar20_split", family="shortchar", n=20, nside=1, nlev=4, nquads=21, precision="split"),
        # many small models of 2k-20k points in one batch
        dict(name="batch8_split", family="batch", models=8, pmax=20000, precision="split"),
        # level populations of a wind on an unstructured mesh: 8 iterations, Ng every 4
        dict(name="ali4k_split", family="ali", npoints=4000, nside=2, nlev=10, nquads=21, iterations=8,
             precision="split"),
        # an image of the same kind of model, odd pixel counts, 41 frequencies
        dict(name="image_fp64", family="image", npoints=20000, nlev=10, nx=151, ny=97, nfreqs=41, precision="fp64"),
        # a fitting step on an image: forward, loss and gradients of every field
        dict(name="image_grad", family="image_grad", npoints=5000, nlev=10, nx=64, ny=64, nfreqs=41),
        # a fitting step on the mean intensity
        dict(name="solve_grad", family="solve_grad", n=13, nside=1, nlev=4, nquads=15),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    family = rng.choice(["solve"] * 6 + ["shells", "shortchar", "batch", "ali", "image", "image_grad", "solve_grad"])
    precision = rng.choice(["fp64", "split"])
    if family == "solve":
        geometry = rng.choice(["cube", "sphere"])
        nside, nlev, nquads = rng.choice([1, 2]), rng.randint(2, 6), rng.randint(5, 31)
        if geometry == "cube":
            nlev = 2  # the cube carries a single line
        # ray pairs x frequencies x path length of the largest listed case bound the size
        cap = 4.0e8 * 37 / (10.0 if precision == "fp64" else 1.0) / (6.0 if geometry == "cube" else 1.0)
        n = int(round(_log(rng, 8, 56)))
        while n > 8 and n**4 * 0.5 * 6 * nside**2 * (nlev - 1) * nquads > cap:
            n -= 1
        return dict(family=family, geometry=geometry, n=n, nside=nside, nlev=nlev, nquads=nquads, precision=precision,
                    approx=rng.choice(["CloseLines"] * 4 + ["OneLine", "None"]),
                    entry="host" if n <= 24 and rng.random() < 0.3 else "device")
    if family == "shells":
        return dict(family=family, npoints=rng.randint(50, 200), nrays=2 * rng.randint(10, 40),
                    nquads=rng.randint(11, 60), precision=precision)
    if family == "shortchar":
        return dict(family=family, n=rng.randint(9, 21), nside=1, nlev=rng.randint(2, 5), nquads=rng.randint(7, 25),
                    precision=precision)
    if family == "batch":
        return dict(family=family, models=rng.randint(2, 10), pmax=rng.randint(4000, 16000), precision="split")
    if family == "ali":
        return dict(family=family, npoints=int(_log(rng, 800, 4000)), nside=rng.choice([1, 2]), nlev=rng.randint(4, 10),
                    nquads=rng.randint(9, 21), iterations=rng.randint(4, 8), precision="split")
    if family == "image":
        return dict(family=family, npoints=int(_log(rng, 2000, 20000)), nlev=rng.randint(4, 10), nx=rng.randint(33, 160),
                    ny=rng.randint(33, 160), nfreqs=rng.randint(17, 64), precision=precision)
    if family == "image_grad":
        return dict(family=family, npoints=int(_log(rng, 1500, 5000)), nlev=rng.randint(4, 10), nx=rng.randint(24, 64),
                    ny=rng.randint(24, 64), nfreqs=rng.randint(11, 41))
    return dict(family=family, n=rng.randint(8, 13), nside=1, nlev=rng.randint(2, 4), nquads=rng.randint(5, 15))


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
@lru_cache(maxsize=32)
def _base(geometry, n, nside, nlev, nquads):
    if geometry == "cube":
        return synthetic.grid_cube(n=n, nside=nside, nquads=nquads)
    if geometry == "sphere":
        return synthetic.grid_sphere(n=n, nside=nside, nquads=nquads, nlev=nlev)
    if geometry == "cutout":
        return synthetic.batch_model(npoints=n, nside=nside, nquads=nquads, nlev=nlev)
    return synthetic.nlte_sphere(npoints=n, nside=nside, nquads=nquads, nlev=nlev, nside_out=8)


def _wind(raw, rng, sigma=0.3e3):
    """The unstructured wind with turbulent velocity noise and 5 % temperature noise."""
    P = raw.npoints
    return replace(raw, velocity=raw.velocity + rng.normal(0.0, sigma, size=(P, 3)) / CC,
                   temperature=raw.temperature * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, size=P)))


def _raw(case, seed):
    rng = np.random.default_rng(seed)
    f = case["family"]
    if f in ("solve", "shortchar", "solve_grad"):
        geometry = case.get("geometry", "sphere")
        raw = _base(geometry, case["n"], case["nside"], case["nlev"], case["nquads"])
        P = raw.npoints
        if geometry == "cube":
            return replace(raw, temperature=rng.uniform(20.0, 100.0, size=P),
                           velocity=rng.normal(0.0, 1.0e3, size=(P, 3)) / CC)
        # grid_sphere's radial outflow 5-15 km/s with its own noise replaced by the seed's
        rel = raw.position - 0.5 * (raw.position.min(axis=0) + raw.position.max(axis=0))
        r = np.sqrt(np.sum(rel * rel, axis=1))
        rhat = rel / np.maximum(r, 1e-300)[:, None]
        vr = 5.0e3 + 10.0e3 * r / r.max()
        return replace(raw, velocity=(vr[:, None] * rhat + rng.normal(0.0, 0.5e3, size=(P, 3))) / CC)
    if f == "shells":
        raw = synthetic.density_distribution_1d("a", case["npoints"], case["nrays"], case["nquads"])
        P = raw.npoints
        v = np.zeros((P, 3))
        v[:, 0] = np.linspace(0.0, 2.0e3, P) * rng.uniform(0.5, 1.5) / CC
        return replace(raw, temperature=20.0 * (1.0 + 0.1 * rng.uniform(-1.0, 1.0, size=P)), velocity=v)
    nside = case.get("nside", 1)
    return _wind(_base("wind", case["npoints"], nside, case["nlev"], case.get("nquads", 5)), rng)


def _batch_raws(case, seed):
    """The models of a batch: point counts spread over [2k, pmax], 12 or 48 rays, 2-5-level
    rotors, 11 / 21 / 31 quadrature points (the mix is the case's, the fields are the seed's)."""
    out = []
    for i in range(case["models"]):
        t = (i + 0.5) / case["models"]
        n = int(2000 * (case["pmax"] / 2000.0) ** t)
        raw = _base("cutout", n, 1 + i % 2, 2 + (i * 7) % 4, (11, 21, 31)[i % 3])
        rng = np.random.default_rng([seed, i])
        P = raw.npoints
        out.append(replace(raw, temperature=rng.uniform(20.0, 100.0, size=P),
                           velocity=rng.normal(0.0, 1.0e3, size=(P, 3)) / CC))
    return out


def _model(raw, precision, approx="CloseLines", image=None):
    model = loader.to_core(raw, precision=precision, approx=approx)
    if image:
        model.compute_spectral_discretisation(*image)
    else:
        model.compute_spectral_discretisation()
    model.compute_inverse_line_widths()
    model.compute_LTE_level_populations()
    return model


def _band(raw, nfreqs):
    """nfreqs image frequencies over +-20 km/s about the first line."""
    f0 = float(raw.linedata[0].frequency[0])
    dd = 20.0e3 / CC
    return f0 * (1.0 - dd), f0 * (1.0 + dd), nfreqs


class Resident(_abi.DeviceModel):
    """A core.Model's device copy behind the device-model calls (the core.Model owns it)."""

    def __init__(self, model):
        prm = model.parameters
        self.model = model
        self.h = C.c_void_p(model.upload())
        self.P, self.F, self.L, self.R = prm.npoints(), prm.nfreqs(), prm.nlines(), prm.hnrays()

    def close(self):
        self.h = None


def _f64(x):
    return torch.tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")


def prepare(case, seed):
    f = case["family"]
    if f == "batch":
        devs = [Resident(_model(r, case["precision"])) for r in _batch_raws(case, seed)]
        return dict(case=case, devs=devs, batch=_abi.Batch(devs),
                    J=[torch.empty((d.P, d.F), dtype=torch.float64, device="cuda") for d in devs],
                    lam=[torch.empty((d.P, d.L), dtype=torch.float64, device="cuda") for d in devs])
    raw = _raw(case, seed)
    if f in ("image", "image_grad"):
        image = _band(raw, case["nfreqs"])
        model = _model(raw, case.get("precision", "fp64"), image=image)
        if f == "image":
            return dict(case=case, dev=Resident(model))
        solver = adjoint.NewImager(model, case["nx"], case["ny"])
    else:
        model = _model(raw, case.get("precision", "fp64"), case.get("approx", "CloseLines"))
        if f == "solve_grad":
            solver = adjoint.FormalSolver(model)
    if f in ("image_grad", "solve_grad"):
        rng = np.random.default_rng([seed, 1])
        if f == "image_grad":
            target = rng.uniform(0.5, 1.5, size=(case["nx"] * case["ny"], case["nfreqs"])) * 1.0e-16
        else:
            target = rng.uniform(0.5, 1.5, size=(raw.npoints, solver.F)) * 1.0e-17
        return dict(case=case, solver=solver, target=_f64(target),
                    fields=[_f64(x) for x in (raw.velocity, raw.temperature, raw.vturb2, raw.abundance)])
    if f == "ali":
        prm = model.parameters
        prm.store_u = False
        prm.use_adaptive_Ng_acceleration = False
        prm.Ng_acceleration_mem_limit = 4
        prm.pop_prec = 0.0  # every iteration runs
        return dict(case=case, model=model)
    if f == "shells" or case.get("entry") == "host":
        model.upload()
        return dict(case=case, model=model)
    dev = Resident(model)
    state = dict(case=case, dev=dev)
    if f == "solve":
        state["J"] = torch.empty((dev.P, dev.F), dtype=torch.float64, device="cuda")
        state["lam"] = torch.empty((dev.P, dev.L), dtype=torch.float64, device="cuda")
    return state


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
# the direction a fitting step looks along, off the axes
DIRECTION = np.array([0.48, 0.36, 0.8])


def run(state):
    case = state["case"]
    f = case["family"]
    if f == "batch":
        state["batch"].formal_solve_fo2_device(case["precision"], [t.data_ptr() for t in state["J"]],
                                               [t.data_ptr() for t in state["lam"]])
        state["batch"].timings()  # waits for the batch and reports its errors
        return dict(J=state["J"], lam=state["lam"])
    if f == "ali":
        model = state["model"]
        model.compute_LTE_level_populations()
        model.compute_level_populations(True, case["iterations"])
        sp = model.lines.lineProducingSpecies[0]
        return dict(population=np.array(sp.population).reshape(model.parameters.npoints(), -1),
                    emissivity=np.array(model.lines.emissivity))
    if f in ("image_grad", "solve_grad"):
        fields = [t.detach().requires_grad_(True) for t in state["fields"]]
        out = state["solver"](DIRECTION, *fields) if f == "image_grad" else state["solver"](*fields)
        scale = 1.0e16 if f == "image_grad" else 1.0e17
        (((out - state["target"]) * scale) ** 2).sum().backward()
        return dict(out=out.detach(), grad=[t.grad for t in fields])
    if f == "image":
        return state["dev"].image_new(DIRECTION, case["nx"], case["ny"], case["precision"])
    if f == "shortchar":
        out = state["dev"].formal_solve_sc0(case["precision"])
        return dict(J=out["J"], lam=out["lambda_diag"])
    if f == "shells" or case.get("entry") == "host":
        model = state["model"]
        model.compute_radiation_field_feautrier_order_2()
        return dict(J=np.array(model.radiation.J), u=np.array(model.radiation.u),
                    lam=np.array(model.lines.lineProducingSpecies[0].lambda_diag))
    dev = state["dev"]
    dev.formal_solve_fo2_device(case["precision"], state["J"].data_ptr(), lam_dev=state["lam"].data_ptr())
    dev.sync()  # waits for the solve and reports its errors
    return dict(J=state["J"], lam=state["lam"])


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
# FP operations per element of a ray and frequency (frequency offset, profile or erf
# difference, optical depth, one elimination row) and per neighbour looked at by a trace
ELEMENT_FLOPS, NEIGHBOUR_FLOPS = 40.0, 20.0


def work(case):
    f = case["family"]
    if f == "batch":
        rs = _batch_raws(case, 0)
        parts = [_solve_work(r.npoints, len(r.neighbors), r.nrays // 2, r.linedata[0].nrad, r.nquads,
                             0.5 * r.npoints ** (1 / 3)) for r in rs]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if f in ("image", "image_grad"):
        P, E, L = case["npoints"] + 960, 15.5 * case["npoints"], case["nlev"] - 1
        px, steps = case["nx"] * case["ny"], 2.0 * case["npoints"] ** (1 / 3)
        times = 4.0 if f == "image_grad" else 1.0
        return {"bytes": P * 64 + E * 4 + P * L * 32 + 8.0 * px * case["nfreqs"] * (1 + (f == "image_grad")),
                "flops": times * px * steps * (case["nfreqs"] * ELEMENT_FLOPS + 15.5 * NEIGHBOUR_FLOPS)}
    if f == "shells":
        P, R, Q = case["npoints"], case["nrays"] // 2, case["nquads"]
        return {"bytes": 8.0 * (P * 12 + P * Q * 2 + R * P * Q), "flops": ELEMENT_FLOPS * P * R * Q * P}
    L = case["nlev"] - 1
    if f == "ali":
        P = case["npoints"] + 960
        w = _solve_work(P, 15.5 * P, 6 * case["nside"] ** 2, L, case["nquads"], 1.2 * case["npoints"] ** (1 / 3))
        return {k: v * case["iterations"] for k, v in w.items()}
    cube = case.get("geometry") == "cube"
    P = case["n"] ** 3 * (1.0 if cube else math.pi / 6)
    w = _solve_work(P, 24.0 * P, 6 * case["nside"] ** 2, L, case["nquads"], 0.6 * case["n"])
    return {k: v * (4.0 if f == "solve_grad" else 1.0) for k, v in w.items()}


def _solve_work(P, E, R, L, Q, steps):
    """Points, velocities, neighbour lists, line data and frequencies in, J and the ALO out;
    ``steps`` the elements of an average ray pair."""
    return {"bytes": P * 64.0 + 4.0 * E + P * L * 40.0 + 16.0 * P * L * Q + 8.0 * P * L,
            "flops": P * R * steps * (L * Q * ELEMENT_FLOPS + 26 * NEIGHBOUR_FLOPS)}


# --------------------------------------------------------------------------
# The formal solve in 64 bits, as plain torch
# --------------------------------------------------------------------------
EXACT_SOLVES = 1.2e8  # elements x frequencies that exact() takes on


def exact(case, seed):
    f = case["family"]
    if f == "batch":
        if case["pmax"] > 20000 or case["models"] > 10:
            return None
        parts = [_exact_solve(r, "CloseLines") for r in _batch_raws(case, seed)]
        return dict(J=[p[0] for p in parts], lam=[p[1] for p in parts])
    if f != "solve":
        return None
    raw = _raw(case, seed)
    if raw.npoints * (raw.nrays // 2) * raw.linedata[0].nrad * raw.nquads > EXACT_SOLVES:
        return None
    J, lam = _exact_solve(raw, case["approx"])
    return dict(J=J, lam=lam, u=None) if case["entry"] == "host" else dict(J=J, lam=lam)


def _exact_solve(raw, approx):
    """J [P][F] and the ALO diagonal [P][L] of a second-order Feautrier solve along every ray
    pair: lines in LTE, interpolation points where the opacity per particle jumps, Gaussian
    profiles, line-integrated optical depths where the Doppler shift jumps."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    d = dict(dtype=torch.float64, device=dev)
    t = lambda x: torch.tensor(np.ascontiguousarray(x), **d)
    ti = lambda x: torch.tensor(np.ascontiguousarray(x).astype(np.int64), device=dev)
    ld, P, Q, L = raw.linedata[0], raw.npoints, raw.nquads, raw.linedata[0].nrad
    R = raw.nrays // 2
    T, vt2 = t(raw.temperature), t(raw.vturb2)
    line = t(ld.frequency)
    w = torch.sqrt(2.0 * KB / (AMU * CC_SQUARED) * ld.inverse_mass * T + vt2)  # width / line frequency
    pop = t(ld.weight) * torch.exp(-t(ld.energy) / (KB * T[:, None]))
    tot = t(raw.abundance[:, ld.num])
    pop = pop * (tot / pop.sum(1))[:, None]
    up, lo = pop[:, ti(ld.irad)], pop[:, ti(ld.jrad)]
    em = (line * HH / (4 * math.pi) * t(ld.A) * up).clamp(min=MIN_LINE_EMISSIVITY)
    op = (line * HH / (4 * math.pi) * (lo * t(ld.Ba) - up * t(ld.Bs))).clamp(min=MIN_LINE_OPACITY)
    iw = 1.0 / (line * w[:, None])
    crit = op / tot[:, None]
    src = em / op
    nu = (line[:, None] + (line * w[:, None])[:, :, None] * t(raw.quad_roots[0]))  # [P][L][Q]
    dsm = MAX_WIDTH_FRACTION * w
    dirs, pos, vel = t(raw.ray_direction), t(raw.position), t(raw.velocity)
    n_nb = raw.n_neighbors.astype(np.int64)
    cum = np.concatenate([[0], np.cumsum(n_nb)])
    K = int(n_nb.max())
    table = np.zeros((P, K), np.int64)
    mask = np.arange(K)[None, :] < n_nb[:, None]
    table[mask] = raw.neighbors
    table, mask = torch.tensor(table, device=dev), torch.tensor(mask, device=dev)
    bdy = torch.zeros(P, dtype=torch.bool, device=dev)
    bdy[ti(raw.boundary2point)] = True
    antipode = healpix.antipodes(raw.ray_direction)
    order = torch.arange(K, device=dev)
    log_diff = math.log(MAX_INTERPOLATION_DIFF)

    def planck(p, freq):
        """The boundary's black body (cosmic background), 0 at interior points."""
        return torch.where(bdy[p][:, None], 2 * HH / CC_SQUARED * freq**3 / torch.expm1(HH * freq / (KB * T_CMB)), 0.0)

    def trace(o, direction):
        """Steps (next point, distance, shift) of the half rays from o until a boundary point."""
        cur, Z = o.clone(), torch.zeros(len(o), **d)
        alive = torch.ones(len(o), dtype=torch.bool, device=dev)
        pts, dzs, shs = [], [], []
        po, vo = pos[o], vel[o]
        while True:
            nb = table[cur]
            rel = pos[nb] - po[:, None]
            Zn = (rel[..., 0] * direction[0] + rel[..., 1] * direction[1]) + rel[..., 2] * direction[2]
            d2 = ((rel[..., 0] * rel[..., 0] + rel[..., 1] * rel[..., 1]) + rel[..., 2] * rel[..., 2]) - Zn * Zn
            ok = mask[cur] & (Zn > Z[:, None]) & alive[:, None]
            alive = alive & ok.any(1)
            if not bool(alive.any()):
                break
            d2 = torch.where(ok, d2, math.inf)
            first = torch.where(d2 == d2.min(1, keepdim=True).values, order, K).min(1).values.clamp(max=K - 1)
            nxt = torch.where(alive, nb.gather(1, first[:, None])[:, 0], -1)
            dz = Zn.gather(1, first[:, None])[:, 0] - Z
            Z = torch.where(alive, Z + dz, Z)
            dv = vel[nxt.clamp(min=0)] - vo
            shs.append(1.0 + ((dv[:, 0] * direction[0] + dv[:, 1] * direction[1]) + dv[:, 2] * direction[2]))
            pts.append(nxt)
            dzs.append(dz)
            cur = torch.where(alive, nxt, cur)
            alive = alive & ~bdy[cur]
        if not pts:
            return None, None, None, torch.zeros(len(o), dtype=torch.long, device=dev)
        pts = torch.stack(pts)
        return pts, torch.stack(dzs), torch.stack(shs), (pts >= 0).sum(0)

    def ilog(x, e, l):
        a, b = x[e["nr"], l], x[e["ni"], l]
        return a * (b / a) ** e["fac"]

    def ilin(x, e, l):
        a, b = x[e["nr"], l], x[e["ni"], l]
        return (b - a) * e["fac"] + a

    def lines_of(l, left, right):
        """(line, where it counts) for the lines within reach of [left, right]."""
        if approx == "OneLine":
            return [(l, None)]
        if approx == "None":
            return [(m, None) for m in range(L)]
        found = []
        for m in range(L):
            hit = (line[m] >= left) & (line[m] <= right)
            if bool(hit.any()):
                found.append((m, hit))
        return found

    def profile(width, x):
        y = width[:, None] * x
        return width[:, None] / math.sqrt(math.pi) * torch.exp(-y * y)

    def eta_chi(e, l, f):
        f = f * e["sh"][:, None]
        reach = MAX_DISTANCE * f * w[e["nr"]][:, None]
        eta, chi = torch.zeros_like(f), torch.full_like(f, MIN_OPACITY)
        for m, hit in lines_of(l, f - reach, f + reach):
            p = profile(ilin(iw, e, m), f - line[m])
            p = p if hit is None else torch.where(hit, p, 0.0)
            eta = eta + p * ilog(em, e, m)[:, None]
            chi = chi + p * ilog(op, e, m)[:, None]
        return eta / chi, chi

    def erf_diff(b, a):
        """erf(b) - erf(a) without cancellation where both lie on one side."""
        plus, minus = (a > 0.5) & (b > 0.5), (a < -0.5) & (b < -0.5)
        far = torch.special.erfc(a.abs()) - torch.special.erfc(b.abs())
        return torch.where(plus, far, torch.where(minus, -far, torch.erf(b) - torch.erf(a)))

    def pair(a, b, dz, l, f):
        """(optical depth, source at a, source at b) between the elements a and b."""
        large = ((b["sh"] - a["sh"]).abs() > torch.minimum(dsm[a["nr"]], dsm[b["nr"]]))[:, None]
        z = dz[:, None]
        (Sa, ca), (Sb, cb) = eta_chi(a, l, f), eta_chi(b, l, f)
        dtau = 0.5 * (ca + cb) * z
        if not bool(large.any()):
            return dtau, Sa, Sb
        fa, fb = f * a["sh"][:, None], f * b["sh"][:, None]
        left, right = torch.minimum(fa, fb), torch.maximum(fa, fb)
        reach = MAX_DISTANCE * right * torch.maximum(w[a["nr"]], w[b["nr"]])[:, None]
        sd, sa, sb = torch.zeros_like(f), torch.zeros_like(f), torch.zeros_like(f)
        for m, hit in lines_of(l, left - reach, right + reach):
            width = 0.5 * (ilin(iw, a, m) + ilin(iw, b, m))
            opac = 0.5 * (ilog(op, a, m) + ilog(op, b, m))[:, None]
            xb, xa = (line[m] - fb) * width[:, None], (line[m] - fa) * width[:, None]
            same = fa == fb
            mean = width[:, None] * opac * 0.5 * erf_diff(xb, xa) / torch.where(same, 1.0, xb - xa)
            mean = torch.where(same, profile(width, fa - line[m]) * opac, mean)
            dt = z * (mean + MIN_OPACITY)
            dt = dt if hit is None else torch.where(hit, dt, 0.0)
            sd = sd + dt
            sa = sa + dt * ilog(src, a, m)[:, None]
            sb = sb + dt * ilog(src, b, m)[:, None]
        if approx == "OneLine":
            La, Lb = ilog(src, a, l)[:, None].expand_as(f), ilog(src, b, l)[:, None].expand_as(f)
        else:
            if approx == "CloseLines":
                sd = torch.where(sd > -MIN_OPACITY * z, torch.maximum(sd, MIN_OPACITY * z), sd)
            La, Lb = sa / sd, sb / sd
        return torch.where(large, sd, dtau), torch.where(large, La, Sa), torch.where(large, Lb, Sb)

    def sweep(o, half, l, f, forward):
        """The elimination from a half ray's far end to the origin: G = F / (1 + F), the
        modified source, the last pair's optical depth and its source at the origin."""
        pts, dzs, shs, steps = half
        n = len(o)
        G, Su, dt_prev, S_in = (torch.zeros_like(f) for _ in range(4))
        if pts is None:
            return G, Su, dt_prev, S_in, steps > 0
        ray = torch.arange(n, device=dev)
        here = torch.cat([o[None], pts.clamp(min=0)])   # [s] the point step s leaves from
        sh = torch.cat([torch.ones(1, n, **d), shs])
        ratio = (crit[here[1:], l] / crit[here[:-1], l]).log().abs()
        count = torch.ceil(ratio / log_diff).clamp(min=1.0)
        s = steps - 1
        i = count[s.clamp(min=0), ray]

        def element(s, i):
            k = s.clamp(min=0)
            c = count[k, ray]
            origin = s < 0
            frac = i / c
            shift = torch.where(c > 1, sh[k, ray] + frac * (sh[k + 1, ray] - sh[k, ray]), sh[k + 1, ray])
            return dict(nr=torch.where(origin, o, here[k + 1, ray]), ni=torch.where(origin, o, here[k, ray]),
                        fac=torch.where(origin | (c == 1), 0.0, 1.0 - frac), sh=torch.where(origin, 1.0, shift),
                        dz=dzs[k, ray] / c)

        def inward(s, i):
            last = i <= 1
            s2 = torch.where(last, s - 1, s)
            return s2, torch.where(last, count[s2.clamp(min=0), ray], i - 1)

        a = element(s, i)
        I = planck(a["nr"], f * a["sh"][:, None])
        S_carry = torch.zeros_like(f)
        first = True
        while True:
            live = s >= 0
            if not bool(live.any()):
                break
            s, i = inward(s, i)
            s = torch.where(live, s, -1)
            b = element(s, i)
            dt, Sa, Sb = pair(a, b, a["dz"], l, f)
            if first:
                row = Sa
                Fn = dt * (1.0 + 0.5 * dt)
                Sn = (row * 0.5 * dt * dt + I * dt) / (1.0 + Fn)
            else:
                row = S_carry if forward else Sa
                q, c = dt / dt_prev, 0.5 * (dt + dt_prev) * dt
                Fn = q * G + c
                Sn = (q * Su + row * c) / (1.0 + Fn)
            m = live[:, None]
            G = torch.where(m, Fn / (1.0 + Fn), G)
            Su = torch.where(m, Sn, Su)
            dt_prev = torch.where(m, dt, dt_prev)
            S_carry = torch.where(m, Sb, S_carry)
            a, first = b, False
        return G, Su, dt_prev, S_carry, steps > 0

    J = torch.zeros(P, L, Q, **d)
    lam = torch.zeros(P, L, **d)
    # the ALO's factors at the origin (the opacity at the line centre)
    freq_c = line.expand(P, L)
    chi_c = torch.full((P, L), MIN_OPACITY, **d)
    for m in range(L):
        reach = MAX_DISTANCE * freq_c * w[:, None]
        own = torch.arange(L, device=dev) == m
        hit = {"OneLine": own, "None": torch.ones_like(own)}.get(approx, (line[m] - freq_c).abs() <= reach)
        x = iw[:, m][:, None] * (freq_c - line[m])
        chi_c = chi_c + torch.where(hit, iw[:, m][:, None] / math.sqrt(math.pi) * torch.exp(-x * x) * op[:, m][:, None], 0)
    wq = t(raw.quad_weights[0])
    chunk = max(1, int(2.0e7 / (max(K * 4, Q))))
    for rr in range(R):
        weight = 2.0 * float(raw.ray_weight[rr])
        for o0 in range(0, P, chunk):
            o = torch.arange(o0, min(P, o0 + chunk), device=dev)
            back, fwd = trace(o, dirs[rr]), trace(o, dirs[int(antipode[rr])])
            for l in range(L):
                f = nu[o, l]
                G1, S1, t1, Sc1, top = sweep(o, back, l, f, False)
                G2, S2, t2, Sc, bot = sweep(o, fwd, l, f, True)
                Io = planck(o, f)
                both, none = (top & bot)[:, None], (~top & ~bot)[:, None]
                # interior origin
                q, c = t2 / t1, 0.5 * (t1 + t2) * t2
                D = q * G1 + c + G2
                u, Ld = (q * S1 + Sc * c + S2) / D, c / D
                # the origin at one end: its boundary row
                tt, Ge, Se, end = (torch.where(bot[:, None], y, x)
                                   for x, y in ((t1, t2), (G1, G2), (S1, S2), (Sc1, Sc)))
                De = tt * (1.0 + 0.5 * tt) + Ge
                ue, Le = (end * 0.5 * tt * tt + Io * tt + Se) / De, 0.5 * tt * tt / De
                u = torch.where(none, Io, torch.where(both, u, ue))
                Ld = torch.where(none, 0.0, torch.where(both, Ld, Le))
                J[o, l] += weight * u
                x = iw[o, l][:, None] * (f - line[l])
                phi = iw[o, l][:, None] / math.sqrt(math.pi) * torch.exp(-x * x)
                lam[o, l] += (float(ld.A[l]) * wq * weight * f * phi * Ld / chi_c[o, l][:, None]).sum(1)
    return J.reshape(P, L * Q), lam
