"""The work that programs have this solver do, as a list of timed cases.

A case is one pass through the public entry points of bfpn_gpu_b200:

  beam    a context that is kept between beams: init_beam, depth steps, the IDD
          and proxy history and, where the case asks for it, the spot plane and
          the energy moments at the last depth (--spot-depths and
          --save-energy-moments of the command line)
  resume  a checkpoint taken up and written again: the four state arrays go up,
          some depth steps run, the four arrays come back
  serve   a list of independent uneven beams handed to the batch entry point
  dose    the IDD of state arrays that the calling program owns on the GPU

Mixed-precision runs hold their state in float32 (5e-5 of the FP64 dose), and a
program keeps such a dose or checkpoint in float32 too; FP64 runs keep doubles.

`exact` is the same computation restated in 64-bit torch and numpy.
"""
import math
import os

import numpy as np
import torch

from bfpn_gpu_b200 import Context, capi, make_config, read_tables

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TABLES = os.path.join(ROOT, "tests", "golden", "tables")
DENSITY = {"water": 1.0, "bone": 1.85}
LX = 40.0  # the depth range of the command line, cm
EPS = 1e-10


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _beam_case(name, precision, ny, nz, nom, nmu, ng, steps, nx=1000, ly=8.0, energy=230.0, lg=259.0,
               material="water", tables="", straggling=False, legacy=False, lite=False, golden=False,
               per_call=0, planes=False):
    c = dict(kind="beam", precision=precision, ny=ny, nz=nz, nom=nom, nmu=nmu, ng=ng, steps=steps, nx=nx, ly=ly,
             energy=energy, lg=lg, material=material, tables=tables or material, straggling=straggling,
             legacy=legacy, lite=lite, golden=golden, per_call=per_call, planes=planes)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest beam (the smoke run's grid), one call per depth step with
        # the dose read back each time, as an interactive or stepping program does
        _beam_case("tiny_step_by_step", "mixed", 8, 8, 8, 8, 40, 8, nx=160, ly=2.0, energy=40.0, lg=59.0,
                   tables="synthetic500", per_call=1),
        # 100 MeV in water on the small grid of the FP64 method study
        _beam_case("small_fp64", "fp64", 16, 16, 8, 8, 200, 40, nx=400, ly=4.0, energy=100.0, lg=104.0,
                   tables="synthetic200_lg104"),
        # the command line's default grid and precision (10x10, 11x11 angles, 500
        # groups) with the beam options of the published 230 MeV runs
        _beam_case("cli_default_fp64", "fp64", 10, 10, 11, 11, 500, 16, golden=True, planes=True),
        # the 20x20 / 20x20 / 500 beam in both precisions
        _beam_case("water20_mixed", "mixed", 20, 20, 20, 20, 500, 16, planes=True),
        _beam_case("water20_fp64", "fp64", 20, 20, 20, 20, 500, 6),
        # the paper-scale grid
        _beam_case("water80_mixed", "mixed", 80, 80, 20, 20, 500, 6, ly=16.0),
        # a middle-sized treatment beam in bone
        _beam_case("bone48_mixed", "mixed", 48, 48, 16, 16, 400, 8, energy=200.0, lg=210.0, material="bone",
                   planes=True),
        # a ragged grid: no two extents alike, odd angles, straggling on
        _beam_case("ragged_mixed", "mixed", 37, 29, 15, 12, 301, 10, energy=150.0, lg=160.0, straggling=True,
                   planes=True),
        # psi^1 only, for memory-limited scans over the whole depth
        _beam_case("lite_mixed", "mixed", 20, 20, 20, 20, 500, 40, lite=True),
        dict(name="resume_mixed", kind="resume", precision="mixed", ny=12, nz=12, nom=9, nmu=9, ng=250, steps=8),
        # a seeded treatment plan: uneven small beams, batched
        dict(name="serve_uneven", kind="serve", beams=6, ny_max=32, steps=24, set=1),
        dict(name="dose_mixed", kind="dose", precision="mixed", ny=20, nz=20, nom=20, nmu=20, ng=500,
             trapezoidal=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["beam", "lite", "resume", "serve", "dose"], [13, 1, 2, 1, 2])[0]
    precision = rng.choices(["mixed", "fp64"], [2, 1])[0]
    if kind == "serve":
        return dict(kind="serve", beams=rng.randint(2, 8), ny_max=rng.choice([16, 32]), steps=rng.randint(8, 32),
                    set=rng.randint(2, 10000))
    ny = _log_int(rng, 6, 72)
    nz = ny if rng.random() < 0.6 else _log_int(rng, 6, 72)
    nom = rng.randint(5, 20)
    nmu = nom if rng.random() < 0.7 else rng.randint(5, 20)
    ng = _log_int(rng, 40, 500)
    cells = (ny + 1) * (nz + 1) * nom * nmu * ng
    if kind == "resume":
        while cells > 8e6:
            ny, nz, ng = max(5, ny * 3 // 4), max(5, nz * 3 // 4), max(31, ng * 3 // 4)
            cells = (ny + 1) * (nz + 1) * nom * nmu * ng
        return dict(kind="resume", precision=precision, ny=ny, nz=nz, nom=nom, nmu=nmu, ng=ng,
                    steps=rng.randint(2, 10))
    if kind == "dose":
        while cells > 1e8 or (ny + 1) * (nz + 1) * nom * nmu > 4194304:
            ny, nz = ny * 3 // 4, nz * 3 // 4
            cells = (ny + 1) * (nz + 1) * nom * nmu * ng
        return dict(kind="dose", precision=precision, ny=ny, nz=nz, nom=nom, nmu=nmu, ng=ng,
                    trapezoidal=rng.random() < 0.5)
    # FP64 is for method studies, on the smaller grids
    while cells > (3e8 if precision == "mixed" else 6e7):
        ny, nz = ny * 4 // 5, nz * 4 // 5
        cells = (ny + 1) * (nz + 1) * nom * nmu * ng
    energy = max(20.0, 0.5 * ng)
    return _beam_case("", precision, ny, nz, nom, nmu, ng, max(3, min(rng.randint(6, 40), int(1.5e9 / cells))),
                      ly=rng.choice([4.0, 8.0]), energy=energy, lg=energy + 10.0,
                      material=rng.choice(["water", "bone"]), straggling=rng.random() < 0.25,
                      legacy=rng.random() < 0.08, lite=kind == "lite", planes=kind != "lite" and rng.random() < 0.5,
                      per_call=rng.choice([0, 0, 0, 1, 4]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _physical(case, seed):
    """Grid and beam of a single-beam case; the seed moves the beam."""
    r = np.random.default_rng(seed)
    energy = case.get("energy", 0.5 * case["ng"]) * (1.0 - 0.02 * r.random())
    material = case.get("material", "water")
    golden = case.get("golden", False)
    return dict(nx=case.get("nx", 1000), ny=case["ny"], nz=case["nz"], nom=case["nom"], nmu=case["nmu"],
                ng=case["ng"], ly=case.get("ly", 8.0), lz=case.get("ly", 8.0), lu=2.0 if golden else 1.0,
                lv=2.0 if golden else 1.0, lg=case.get("lg", 0.5 * case["ng"] + 10.0), beam_energy=energy,
                sigma_e=0.01 * energy if not golden else 1.0, sigma_yz=float(r.uniform(0.3, 0.6)),
                density=DENSITY[material], energy_density=DENSITY[material], material_name=material,
                eq15_straggling=case.get("straggling", False), legacy_energy=case.get("legacy", False),
                lite_memory=case.get("lite", False), discrete_angle_delta=golden, normalize_initial_mass=golden,
                trapezoidal_yz=golden)


def _uneven(case, seed):
    """The beams of a serving case: energy, material, width, plane, angles and groups each their own."""
    s = np.random.default_rng(case["set"])  # the shapes belong to the case
    r = np.random.default_rng(seed)         # the beams to the seed
    out = []
    for _ in range(case["beams"]):
        energy = float(s.uniform(70.0, 150.0))
        ny = int(s.choice([n for n in (16, 32) if n <= case["ny_max"]]))
        na = int(s.choice([12, 16]))
        material = "water" if s.random() < 0.5 else "bone"
        ng = int(round(2.0 * energy))
        out.append(dict(nx=1000, ny=ny, nz=ny, nom=na, nmu=na, ng=ng, ly=8.0, lz=8.0, lu=1.0, lv=1.0,
                        lg=energy + 10.0, beam_energy=energy * (1.0 - 0.02 * r.random()), sigma_e=0.01 * energy,
                        sigma_yz=float(r.uniform(0.3, 0.8)), density=DENSITY[material],
                        energy_density=DENSITY[material], material_name=material))
    return out


def _device_rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _resume_state(case, seed):
    """F, f, F1, f1 of a beam in mid-depth: a spread Gaussian in y, z, angle and
    energy with some structure, float32 values."""
    ny1, nz1, nom, nmu, ng = case["ny"] + 1, case["nz"] + 1, case["nom"], case["nmu"], case["ng"]
    dev, g = "cuda", _device_rng(seed)

    def bell(n, width):
        x = torch.linspace(-1.0, 1.0, n, device=dev, dtype=torch.float64)
        return torch.exp(-((x / width) ** 2))

    e = torch.arange(ng, device=dev, dtype=torch.float64) / ng
    base = (torch.exp(-(((e - 0.7) / 0.08) ** 2))[:, None, None, None, None] * bell(nz1, 0.4)[:, None, None, None]
            * bell(ny1, 0.35)[:, None, None] * bell(nmu, 0.5)[:, None] * bell(nom, 0.5))
    tail = (torch.exp(-3.0 * (0.8 - e).abs())[:, None, None, None, None] * bell(nz1, 0.6)[:, None, None, None]
            * bell(ny1, 0.6)[:, None, None] * bell(nmu, 0.8)[:, None] * bell(nom, 0.8))

    def noise(a):
        return torch.rand(base.shape, device=dev, generator=g, dtype=torch.float32).double() * a

    F = base * (1.0 + noise(0.2))
    f = base * (noise(0.2) - 0.1)
    F1 = 0.05 * tail * (1.0 + noise(0.2))
    f1 = 0.05 * tail * (noise(0.2) - 0.1)
    return [a.float().double().reshape(-1) for a in (F, f, F1, f1)]


def _dose_arrays(case, seed):
    n = ((case["ny"] + 1) * (case["nz"] + 1), case["nom"] * case["nmu"])
    g = _device_rng(seed)
    dt = torch.float32 if case["precision"] == "mixed" else torch.float64

    def one(lo, hi):
        a = torch.rand((case["ng"],) + n, device="cuda", generator=g, dtype=dt)
        return a.mul_(hi - lo).add_(lo)

    return one(0.0, 1.0), one(-0.1, 0.1), one(0.0, 0.1), one(-0.01, 0.01)


def _dose_weights(case, seed):
    ph = _physical(case, seed)
    t = _Tables(ph, angular=False, table_dir=os.path.join(TABLES, "water"))
    return ph, np.stack([t.w1, t.w2], axis=1).reshape(-1)


def _grid_only(ph):
    return make_config(**ph).grid()


def _precision(case):
    return capi.PREC_MIXED if case["precision"] == "mixed" else capi.PREC_FP64


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        beams = []
        for ph in _uneven(case, seed):
            cfg = make_config(**ph)
            mu, sig = read_tables(os.path.join(TABLES, ph["material_name"]), cfg.ng)
            beams.append(capi.make_beam(cfg.grid(), cfg.phys(), mu, sig, case["steps"], capi.PREC_MIXED))
        return dict(kind=kind, beams=beams)
    if kind == "dose":
        ph, w = _dose_weights(case, seed)
        return dict(kind=kind, grid=_grid_only(ph), precision=_precision(case), trap=case["trapezoidal"],
                    arrays=_dose_arrays(case, seed), weights=torch.from_numpy(w).cuda())
    ph = _physical(case, seed)
    cfg = make_config(**ph)
    mu, sig = read_tables(os.path.join(TABLES, case.get("tables", "water")), cfg.ng)
    ctx = Context(cfg.grid(), cfg.phys(), _precision(case), device=0)
    ctx.load_tables(mu, sig)
    s = dict(kind=kind, ctx=ctx, steps=case["steps"], mixed=case["precision"] == "mixed")
    if kind == "resume":
        ctx.init_beam()
        ctx.step(1)  # the checkpoint is of a beam under way
        s["arrays"] = [a.cpu().numpy() for a in _resume_state(case, seed)]
    else:
        s.update(per_call=case["per_call"] or case["steps"], planes=case["planes"])
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _kept(s, *arrays):
    """Results in the precision of the run's state."""
    t = [torch.from_numpy(np.asarray(a)) for a in arrays]
    return [x.float() for x in t] if s["mixed"] else t


def run(s):
    kind = s["kind"]
    if kind == "serve":
        s["mixed"] = True
        return [_kept(s, idd, proxy) for idd, proxy in capi.batch_run(s["beams"])]
    if kind == "dose":
        out = torch.empty(2, device="cuda", dtype=torch.float64)
        F0, f0, F1, f1 = s["arrays"]
        capi.idd_noalloc(s["grid"], s["precision"], s["trap"], F0.data_ptr(), f0.data_ptr(), F1.data_ptr(),
                         f1.data_ptr(), s["weights"].data_ptr(), out.data_ptr(),
                         stream=torch.cuda.current_stream().cuda_stream)
        return out
    ctx = s["ctx"]
    if kind == "resume":
        for k, a in enumerate(s["arrays"]):
            ctx.set_state(k // 2, k % 2, a)
        idd, proxy = ctx.step(s["steps"])
        return _kept(s, idd, proxy, *[ctx.get_state(k // 2, k % 2) for k in range(4)])
    ctx.init_beam()
    left, idd, proxy = s["steps"], [], []
    while left > 0:
        a, b = ctx.step(min(left, s["per_call"]))
        idd.append(a)
        proxy.append(b)
        left -= s["per_call"]
    out = [np.concatenate(idd), np.concatenate(proxy)]
    if s["planes"]:
        out += [ctx.spot_plane(), ctx.energy_moments()]
    return _kept(s, *out)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _beam_work(ny, nz, nom, nmu, ng, steps, elem, lite=False):
    """Each depth step reads and writes the state once. Operations per cell and array of a step: two transports
    of two limited stages in two directions (about 90 each), four DST passes, two energy sweeps (about 20 each)
    and, per step, the secondary's source from its banded kernels."""
    nyz, na = (ny + 1) * (nz + 1), nom * nmu
    cells = float(nyz * na * ng)
    if lite:
        return 2.0 * cells * elem * steps, 6.0 * cells * steps
    return 8.0 * cells * elem * steps, 4.0 * cells * steps * (180.0 + 4.0 * (nom + nmu) + 40.0)


def work(case):
    kind = case["kind"]
    elem = 8 if case.get("precision") == "fp64" else 4
    if kind == "serve":
        w = [_beam_work(p["ny"], p["nz"], p["nom"], p["nmu"], p["ng"], case["steps"], 4) for p in _uneven(case, 1)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    if kind == "dose":
        cells = (case["ny"] + 1) * (case["nz"] + 1) * case["nom"] * case["nmu"] * case["ng"]
        return {"bytes": 4.0 * cells * elem, "flops": 6.0 * cells}
    b, f = _beam_work(case["ny"], case["nz"], case["nom"], case["nmu"], case["ng"], case["steps"], elem,
                      case.get("lite", False))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same in 64 bits, in torch and numpy
# ---------------------------------------------------------------------------
_COMPOSITION = {
    "bone": [(1, 0.04200), (6, 0.1940), (7, 0.04000), (8, 0.4250), (11, 0.001000), (12, 0.002000), (15, 0.09200),
             (16, 0.003000), (20, 0.2010)],
    "water": [(1, 0.1111), (8, 0.8889)],
}
_MASS = {1: 1.0, 6: 12.0, 7: 14.0, 8: 16.0, 11: 23.0, 12: 24.0, 15: 31.0, 16: 32.0, 20: 40.0}


def _bethe(E, Z):
    beta2 = np.maximum(E * (E + 2.0 * 938.3) / ((E + 938.3) * (E + 938.3)), EPS)
    gamma2 = 1.0 / np.maximum(1.0 - beta2, EPS)
    ion = 19.0 if Z == 1 else 11.2 + 11.7 * Z if Z <= 13 else 52.8 + 8.71 * Z
    arg = np.maximum(2.0 * 0.51099895e6 * beta2 * gamma2 / ion, 1.0 + EPS)
    return 0.307 * (Z / _MASS[Z]) / beta2 * (np.log(arg) - beta2)


class _Tables:
    """Set-up tables of one beam: numpy, the angular kernel and the state on the GPU."""

    def __init__(self, ph, angular=True, table_dir=None):
        self.ph, ng = ph, ph["ng"]
        self.Ng, self.Ny1, self.Nz1, self.Nom, self.Nmu = ng, ph["ny"] + 1, ph["nz"] + 1, ph["nom"], ph["nmu"]
        self.NA = self.Nom * self.Nmu
        self.dt, self.dy, self.dz = LX / ph["nx"], ph["ly"] / ph["ny"], ph["lz"] / ph["nz"]
        self.dg, self.du, self.dv = ph["lg"] / ng, ph["lu"] / (self.Nom + 1), ph["lv"] / (self.Nmu + 1)
        rows = open(os.path.join(table_dir, "cross_total.txt")).read().split()
        self.sigma = np.array([float(x) for x in rows[:ng]])
        i = np.arange(ng + 1)
        E = (i - 0.5) * self.dg + 1.0
        E[0], E[-1] = 1.0, ph["lg"] + 1.0
        mat = sum(w * _bethe(E, z) for z, w in _COMPOSITION[ph["material_name"]])
        wat = sum(w * _bethe(E, z) for z, w in _COMPOSITION["water"])
        b2 = E * (E + 2.0 * 938.3) / (E + 938.3) ** 2
        self.S = (0.170 / b2 * (np.log(1.02e6 * b2 / (1.0 - b2)) - b2 - 4.31) + 0.02) * np.where(
            wat > EPS, mat / np.where(wat > EPS, wat, 1.0), 1.0)
        en = i * self.dg + 1.0
        sig = np.maximum(self.sigma, 0.0)
        # dose per unit psi^1 and psi^2 of a group, over the density
        self.w1 = (0.5 * (self.S[:-1] + self.S[1:]) + 0.5 * (en[:-1] + en[1:]) * sig) * self.dg / ph["density"]
        self.w2 = ((self.S[1:] - self.S[:-1]) / 6.0 * self.dg + (en[1:] - en[:-1]) * sig * self.dg / 6.0) / ph["density"]
        self.Tc = np.full(ng, 8.99e18 * 4.0 * math.pi * 1.6e-19 ** 4 / 1.6e-13 ** 2 / 100.0 * 3.34e29 * 1.2)
        if angular:
            self._angular(table_dir)

    def _angular(self, table_dir):
        ph, ng, dg, NA = self.ph, self.Ng, self.dg, self.NA
        cross = next(f for f in ("data_cross.txt", "data_b.txt") if os.path.exists(os.path.join(table_dir, f)))
        v = [float(x) for x in open(os.path.join(table_dir, cross)).read().split()[:3 * ng]]
        mu = np.zeros(3 * ng)
        mu[:len(v)] = v
        mu = mu.reshape(ng, 3)
        E = (np.arange(ng) + 0.5) * dg + 1.0
        beta = np.sqrt(2.0 * E * 1.6e-13 / 1.673e-27) / (3.0 * 2.998e8)
        eta = 3.0 ** (2.0 / 3.0) * (1.0 / 137.0) ** 2 * (9.10956e-31 / 1.673e-27) ** 2 / (beta * beta)
        mid = np.log((eta + 1.0) / eta) - 1.0 / (eta + 1.0)
        trg = 2.0 * math.pi * 3.34 * 197.3 ** 2 * (1.0 / 137.0) ** 2 / 4.0 * 9.0 / (E * E) * mid / 1000.0
        # energy kernels: [out, src]
        ker = np.zeros((ng, ng))
        for j in range(ng - 1):
            if mu[j, 2] != 0.0:
                k = np.arange(j, ng - 1)
                ker[k + 1, j] = dg / mu[j, 2] * np.exp(-(k - j + 0.5) * dg / mu[j, 2])
        ker = ker[::-1, ::-1].copy()
        ker[np.abs(ker) < 1e-5] = 0.0
        ker *= self.sigma[None, :]
        nxt = np.vstack([ker[1:], np.zeros((1, ng))])
        self.e1, self.e2 = (torch.from_numpy(0.5 * (a + nxt)).cuda() for a in (ker, -ker))
        # directions and the angular kernel [src, in, out]
        u = -0.5 * ph["lu"] + (np.arange(self.Nom) + 1) * self.du
        w = -0.5 * ph["lv"] + (np.arange(self.Nmu) + 1) * self.dv
        oy, oz = np.repeat(-w[::-1], self.Nom), np.tile(-u, self.Nmu)
        self.oy, self.oz = torch.from_numpy(oy.copy()).cuda(), torch.from_numpy(oz.copy()).cuda()
        r2 = 1.0 + oy * oy + oz * oz
        n = np.sqrt(r2)
        c = (1.0 + oy[:, None] * oy[None, :] + oz[:, None] * oz[None, :]) / np.maximum(n[:, None] * n[None, :], EPS)
        theta = torch.from_numpy(np.abs(np.arccos(np.clip(c, -1.0, 1.0)) * 180.0 / math.pi)).cuda()
        weight = torch.from_numpy(r2 ** -1.5).cuda()[:, None]
        self.kv = torch.zeros((ng, NA, NA), device="cuda", dtype=torch.float64)
        for k in range(ng - 1):
            if mu[k, 0] == 0.0 or mu[k, 1] == 0.0:
                continue
            val = theta ** (mu[k, 0] - 1.0) * torch.exp(-theta / mu[k, 1]) * weight
            val[~torch.isfinite(val)] = 0.0
            s = val.sum(0, keepdim=True)
            norm = val / s
            norm[norm < 1e-3] = 0.0
            self.kv[k] = torch.where(s > EPS, norm, val)
        # angular diffusion
        def sine(m):
            a = np.arange(1, m + 1)
            return torch.from_numpy(np.sin(math.pi * np.outer(a, a) / (m + 1))).cuda()
        self.su, self.sv = sine(self.Nom), sine(self.Nmu)
        lu = (2.0 - 2.0 * np.cos(math.pi * np.arange(1, self.Nom + 1) / (self.Nom + 1))) / self.du ** 2
        lv = (2.0 - 2.0 * np.cos(math.pi * np.arange(1, self.Nmu + 1) / (self.Nmu + 1))) / self.dv ** 2
        lam = 0.5 * ph["density"] * trg[:, None, None] * (lv[:, None] + lu[None, :])
        self.fac = torch.from_numpy((2.0 / self.dt - lam) / (2.0 / self.dt + lam) * 4.0
                                    / ((self.Nom + 1.0) * (self.Nmu + 1.0))).cuda()
        # initial beam
        c1, c2 = np.abs(w).min(), np.abs(u).min()
        y = -0.5 * ph["ly"] + np.arange(self.Ny1) * self.dy
        z = -0.5 * ph["lz"] + np.arange(self.Nz1) * self.dz
        a1, a2 = 0.5 / ph["sigma_yz"] ** 2, 0.5 / 1e-6 / 1e-6
        yz = np.exp(-a1 * (z[:, None] ** 2 + y[None, :] ** 2))
        wy, wz = np.ones(self.Ny1), np.ones(self.Nz1)
        if ph.get("trapezoidal_yz"):
            wy[[0, -1]], wz[[0, -1]] = 0.5, 0.5
        self.wyz = torch.from_numpy(wz[:, None] * wy[None, :]).cuda()
        d1, d2 = np.abs(oy) - c1, np.abs(oz) - c2
        if ph.get("discrete_angle_delta"):
            hit = (np.abs(d1) < 0.25 * self.dv) & (np.abs(d2) < 0.25 * self.du)
            ang, angular_mass = hit / (hit.sum() * self.du * self.dv), 1.0
        else:
            ang = np.exp(-a2 * (d1 * d1 + d2 * d2))
            angular_mass = ang.sum() * self.du * self.dv
        beam_e = np.exp(-((E - ph["beam_energy"]) / ph["sigma_e"] / math.sqrt(2.0)) ** 2) / math.sqrt(
            2.0 * math.pi) / ph["sigma_e"]
        scale = 1.0
        if ph.get("normalize_initial_mass"):
            scale = 1.0 / ((wz[:, None] * wy[None, :] * yz).sum() * self.dy * self.dz * angular_mass
                           * beam_e.sum() * dg)
        self.beam = [torch.from_numpy(x).cuda() for x in (beam_e, scale * yz.reshape(-1), ang)]


class _Exact:
    """The depth step in float64; arrays [group, position, angle]."""

    def __init__(self, ph, table_dir):
        self.t = _Tables(ph, table_dir=table_dir)
        self.ph, t = ph, self.t
        e, yz, ang = t.beam
        self.state = [e[:, None, None] * yz[None, :, None] * ang[None, None, :]]
        if not ph["lite_memory"]:
            self.state += [torch.zeros_like(self.state[0]) for _ in range(3)]
        self.first = True

    def _rows(self, v):
        return torch.from_numpy(np.ascontiguousarray(v)).cuda()[:, None]

    def energy(self, k, src):
        t, ph, dt = self.t, self.ph, 0.5 * self.t.dt
        rho, dg, Ng = ph["energy_density"], t.dg, t.Ng
        sig, lo, hi = (np.maximum(x, 0.0) for x in (t.sigma, t.S[:-1], t.S[1:]))
        flatF, flatf = self.state[k].view(Ng, -1), self.state[k + 1].view(Ng, -1)
        T = np.maximum(t.Tc, 0.0) if ph["eq15_straggling"] else np.zeros(Ng)
        Thi, Tlo = np.append(T[1:], 0.0), np.insert(T[:-1], 0, 0.0)
        dg2 = max(dg * dg, EPS)
        lanes = flatF.shape[1]
        step = max(1, int(1.2e9 // (8 * Ng)))
        for b in range(0, lanes, step):
            F, f = flatF[:, b:b + step], flatf[:, b:b + step]
            s = src.view(Ng, -1)[:, b:b + step] if src is not None else 0.0
            up = torch.zeros_like(F)
            if ph["legacy_energy"]:
                den = np.maximum(1.0 / dt + rho * lo / dg + sig, EPS)
                A = F.clamp(min=0.0) / dt + s
                lap = torch.zeros_like(F)
                P = F.clamp(min=0.0)
                lap[:-1] += P[1:]
                lap[1:] += P[:-1]
                lap -= 2.0 * P
                lap *= self._rows(0.5 * dt * T / dg2)
                nF, nf = torch.zeros_like(F[0]), torch.zeros_like(F[0])
                for g in range(Ng - 1, -1, -1):
                    h = rho * hi[g] / dg
                    nF = ((A[g] + h * nF) / den[g] + lap[g]).clamp(min=0.0)
                    nf = ((f[g] / dt + h * nf) / den[g]).clamp(min=0.0)
                    F[g], f[g] = nF, nf
                continue
            iF = 1.0 / np.maximum(1.0 / dt + 0.5 * rho * lo / dg + 0.5 * sig, EPS)
            A, Ff, Fhi = 1.5 * rho * hi / dg * iF, 0.5 * rho * lo / dg * iF, 0.5 * rho * hi / dg * iF
            up[:-1] = F[1:] - f[1:]
            cur = F - f
            common = self._rows(0.5 * rho * hi / dg) * up - self._rows(0.5 * rho * lo / dg) * cur
            common += self._rows(1.0 / dt - 0.5 * sig - rho * T / dg2) * F + s
            if ph["eq15_straggling"]:
                common[:-1] += self._rows(0.5 * rho * Thi / dg2)[:-1] * F[1:]
                common[1:] += self._rows(0.5 * rho * Tlo / dg2)[1:] * F[:-1]
            coe = np.maximum(1.0 / dt + 0.5 * sig + 1.5 * rho * lo / dg + 0.5 * rho * (hi - lo) / dg
                             + A * 0.5 * rho * lo / dg, EPS)
            rhs = self._rows(1.0 / dt - 0.5 * sig - 0.5 * rho * (hi - lo) / dg) * f
            rhs += self._rows(1.5 * rho * hi / dg) * up
            rhs += self._rows(1.5 * rho * lo / dg) * cur
            rhs -= self._rows(1.5 * rho * (lo + hi) / dg) * F
            rhs -= self._rows(A) * common
            rhs /= self._rows(coe)
            common *= self._rows(iF)
            # new f = rhs + kd * delta, new F = Ff * f + common + Fhi * delta, delta = (F - f) of the group above
            kd = (1.5 * rho * hi / dg - A * 0.5 * rho * hi / dg) / coe
            beta = common + self._rows(Ff - 1.0) * rhs
            alpha = Fhi + (Ff - 1.0) * kd
            delta = up.zero_()
            for g in range(Ng - 2, -1, -1):
                torch.add(beta[g + 1], delta[g + 1], alpha=float(alpha[g + 1]), out=delta[g])
            rhs += self._rows(kd) * delta
            F[:] = self._rows(Ff) * rhs + common + self._rows(Fhi) * delta
            f[:] = rhs

    def _div(self, X):
        """Flux divergence of [g, z, y, ang]."""
        t, out = self.t, None
        for dim, w, h, n in ((2, t.oy, t.dy, t.Ny1), (1, t.oz, t.dz, t.Nz1)):
            idx = torch.arange(-2, n + 2, device="cuda").clamp(0, n - 1)
            G = X.index_select(dim, idx)                       # cells -2 .. n+1
            d = G.narrow(dim, 1, n + 3) - G.narrow(dim, 0, n + 3)
            back, fwd = d.narrow(dim, 0, n + 2), d.narrow(dim, 1, n + 2)
            small = fwd.abs() < EPS
            th = back / torch.where(small, torch.ones_like(fwd), fwd)
            s = torch.maximum((2.0 * th).clamp(max=1.0), th.clamp(max=2.0)).clamp(min=0.0) * fwd
            s[small] = 0.0                                     # cells -1 .. n
            c = G.narrow(dim, 1, n + 2)
            left = torch.where(w >= 0.0, w * (c + 0.5 * s).narrow(dim, 0, n + 1),
                               w * (c - 0.5 * s).narrow(dim, 1, n + 1))
            part = (left.narrow(dim, 1, n) - left.narrow(dim, 0, n)) / h
            out = part if out is None else out + part
        return out

    def transport(self, k, clip):
        t, dt = self.t, 0.5 * self.t.dt
        X = self.state[k].view(t.Ng, t.Nz1, t.Ny1, t.NA)
        step = max(1, int(6e8 // (8 * t.Nz1 * t.Ny1 * t.NA)))
        for b in range(0, t.Ng, step):
            F = X[b:b + step]
            d0 = self._div(F)
            P = F - dt * d0
            d0 += self._div(P.clamp_(min=0.0) if clip else P)
            F -= 0.5 * dt * d0
            if clip:
                F.clamp_(min=0.0)

    def angle(self, k):
        t = self.t
        X = self.state[k].view(t.Ng, -1, t.Nmu, t.Nom)
        step = max(1, int(1e9 // (8 * X[0].numel())))
        for b in range(0, t.Ng, step):
            Y = (t.sv @ (X[b:b + step] @ t.su)) * t.fac[b:b + step, None]
            X[b:b + step] = (t.sv @ Y) @ t.su

    def source(self):
        t = self.t
        out = torch.zeros_like(self.state[0])
        for e, P, c in ((t.e1, self.state[0].clamp(min=0.0), t.dg), (t.e2, self.state[1], t.dg / 3.0)):
            A = torch.bmm(P, t.kv)
            out.view(t.Ng, -1).addmm_(e, A.view(t.Ng, -1), alpha=c)
        return out

    def dose(self):
        t = self.t
        w = t.wyz.reshape(-1, 1)
        vol = t.du * t.dv * t.dy * t.dz
        m = [(a * w).sum((1, 2)) for a in self.state]
        if len(m) == 1:  # psi^1 only
            return float((m[0] * torch.from_numpy(t.w1).cuda()).sum()) * vol, 0.0
        total = (m[0] + m[2]) * torch.from_numpy(t.w1).cuda() + (m[1] + m[3]) * torch.from_numpy(t.w2).cuda()
        return float(total.sum()) * vol, float(self.state[1].sum()) * t.dg

    def lite_step(self):
        t = self.t
        F = self.state[0].view(t.Ng, -1)
        lo, hi = np.maximum(t.S[:-1], 0.0), np.maximum(t.S[1:], 0.0)
        den = np.maximum(1.0 / t.dt + lo / t.dg + np.maximum(t.sigma, 0.0), EPS)
        F.clamp_(min=0.0)
        F /= self._rows(den * t.dt)
        for g in range(t.Ng - 2, -1, -1):
            F[g].add_(F[g + 1], alpha=float(hi[g] / t.dg / den[g]))

    def step(self):
        if self.ph["lite_memory"]:
            self.lite_step()
            return self.dose()
        for k in (0,) if self.first else (0, 2):
            src = self.source() if k == 2 else None
            self.energy(k, src)
            for a, clip in ((k, True), (k + 1, False)):
                self.transport(a, clip)
                self.angle(a)
                self.transport(a, clip)
            self.energy(k, src)
        self.first = False
        return self.dose()

    def planes(self):
        t, s = self.t, self.state
        w1, w2 = self._rows(t.w1), self._rows(t.w2)
        plane = (w1 * (s[0] + s[2]).sum(2) + w2 * (s[1] + s[3]).sum(2)).sum(0) * (t.du * t.dv)
        vol = t.du * t.dv * t.dy * t.dz
        mom = torch.stack([(s[0] + s[2]).sum((1, 2)), (s[1] + s[3]).sum((1, 2))], 1) * vol
        return plane.cpu(), mom.reshape(-1).cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "dose":
        ph, w = _dose_weights(case, seed)
        F0, f0, F1, f1 = _dose_arrays(case, seed)
        wy, wz = np.ones(case["ny"] + 1), np.ones(case["nz"] + 1)
        if case["trapezoidal"]:
            wy[[0, -1]], wz[[0, -1]] = 0.5, 0.5
        pos = torch.from_numpy((wz[:, None] * wy[None, :]).reshape(1, -1, 1)).cuda()
        total = proxy = 0.0
        for g in range(case["ng"]):
            total += float(((F0[g].double() + F1[g]) * pos).sum() * w[2 * g]
                           + ((f0[g].double() + f1[g]) * pos).sum() * w[2 * g + 1])
            proxy += float(f0[g].double().sum())
        vol = (ph["ly"] / ph["ny"]) * (ph["lz"] / ph["nz"]) * (ph["lu"] / (ph["nom"] + 1)) * (ph["lv"] / (ph["nmu"] + 1))
        return torch.tensor([total * vol, proxy * ph["lg"] / ph["ng"]], dtype=torch.float64)
    if kind == "serve":
        out = []
        for ph in _uneven(case, seed):
            ph.update(lite_memory=False, legacy_energy=False, eq15_straggling=False)
            x = _Exact(ph, os.path.join(TABLES, ph["material_name"]))
            got = np.array([x.step() for _ in range(case["steps"])])
            out.append([got[:, 0], got[:, 1]])
        return out
    ph = _physical(case, seed)
    x = _Exact(ph, os.path.join(TABLES, case.get("tables", "water")))
    if kind == "resume":
        shape = x.state[0].shape
        x.state = [a.reshape(shape).clone() for a in _resume_state(case, seed)]
        x.first = False
    got = np.array([x.step() for _ in range(case["steps"])])
    out = [got[:, 0], got[:, 1]]
    if kind == "resume":
        out += [a.reshape(-1).cpu() for a in x.state]
    elif case["planes"]:
        out += list(x.planes())
    return out
