"""The work a user of this framework has it do, as cases that can be timed and compared.

Four families, each through the entry points a program calls:

  single    one FP64 solve of the Euler or Navier-Stokes equations: a state in, time steps, the
            state out (`gpu.Solver`), from the 65 x 65 vortex to the 1025 x 1025 Kelvin-Helmholtz mesh
  samples   plain Monte Carlo, one FP64 sample after the other on one handle: initial condition
            from the sample's random numbers, steps to the output time, moments
  ensemble  batched FP32 members advanced together (`batch.Batch`): Kelvin-Helmholtz levels with
            integrals and moments, the Navier-Stokes cylinder with the wall force at output times
  surrogate the control variate's network (`mlp.MLP`): training on solver runs, and evaluation

`exact` restates the numerical method in plain torch, FP64, from the triangulation alone.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tensum_b200 import abi, batch, cases, cylinder, gpu, mlp, preproc

PERIODIC = {t: ("periodic", {}) for t in (1, 2, 3, 4)}
FLUXES = ("kepes_tecno_roe", "kepes_tecno_rusanov", "kepec", "kep", "roe_ec")
EXTRAS = 7                                 # moment records: density, mach number and entropy too


# ------------------------------------------------------------------------ cases

def listed():
    return [
        # the accuracy run: a small mesh, thousands of short steps, so each step's latency is what counts
        dict(name="vortex65_tecno_roe", family="single", ic="vortex", n=65, flux="kepes_tecno_roe",
             recon="minmod", scheme="ssprk3", steps=200),
        # the shear layer at full resolution with the entropy-stable second-order flux
        dict(name="kh1025_tecno_rusanov", family="single", ic="kh", n=1025, flux="kepes_tecno_rusanov",
             recon="minmod", scheme="ssprk3", steps=40),
        # the same mesh with an entropy-conservative central flux: no gradients, bound by memory
        dict(name="kh1025_kepec", family="single", ic="kh", n=1025, flux="kepec", recon="first",
             scheme="ssprk3", steps=60),
        # a middle size that fills the last wave unevenly, the classical four-stage scheme
        dict(name="kh387_roe_ec_rk4", family="single", ic="kh", n=387, flux="roe_ec", recon="first",
             scheme="rk4", steps=60),
        # viscous flow with walls and far field, the wall force at every output time
        dict(name="cylinder128x256_fp64", family="single", ic="cylinder", n=128, nt=256,
             flux="kepes_tecno_roe", recon="minmod", scheme="ssprk3", steps=64, outputs=4),
        # plain Monte Carlo: samples one after the other on one handle
        dict(name="samples_kh257_fp64", family="samples", n=257, flux="kepes_tecno_rusanov", recon="minmod",
             samples=3, steps=24),
        # the ensemble of the Monte Carlo study: many members of one mesh, integrals and moments
        dict(name="ensemble_kh257x768", family="ensemble", ic="kh", n=257, flux="kepes_tecno_rusanov",
             recon="minmod", samples=768, steps=10, levels=1),
        # a pilot study: few members of a small mesh (their count an odd multiple of 32)
        dict(name="ensemble_kh65x96", family="ensemble", ic="kh", n=65, flux="kepes_tecno_rusanov",
             recon="minmod", samples=96, steps=32, levels=1),
        # three levels of a multilevel estimator in one batch: 129, 257 and 513 vertices a side
        dict(name="ensemble_multilevel", family="ensemble", ic="kh", n=129, flux="kepes_tecno_rusanov",
             recon="minmod", samples=512, steps=4, levels=3),
        # viscous members with per-sample Mach number, Reynolds number and inflow angle
        dict(name="ensemble_cylinder128x256x128", family="ensemble", ic="cylinder", n=128, nt=256,
             flux="kepes_tecno_roe", recon="minmod", samples=128, steps=24, outputs=2, levels=1),
        # the surrogate trained on the study's solver runs
        dict(name="surrogate_fit", family="fit", rows=256, din=3, batch=64, epochs=200),
        # the surrogate evaluated at the extra inputs of the control-variate estimator
        dict(name="surrogate_predict", family="predict", rows=1 << 20, din=3, precision=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["periodic", "periodic", "periodic", "cylinder", "samples", "ensemble", "ensemble",
                       "ensemble_cylinder", "fit", "predict"])
    if kind == "periodic":
        flux = rng.choice(FLUXES)
        tecno = flux.startswith("kepes")
        n = _log(rng, 21, 900)
        return dict(family="single", ic=rng.choice(["kh", "vortex"]), n=n, flux=flux,
                    recon=rng.choice(["minmod", "minmod", "van_albada", "first"]) if tecno else "first",
                    scheme=rng.choice(["ssprk3", "ssprk3", "rk4"]), steps=rng.randint(20, 40))
    if kind == "cylinder":
        return dict(family="single", ic="cylinder", n=_log(rng, 24, 180), nt=_log(rng, 48, 400),
                    flux=rng.choice(["kepes_tecno_roe", "kepes_tecno_rusanov"]), recon="minmod", scheme="ssprk3",
                    steps=rng.randint(20, 60), outputs=rng.randint(1, 4))
    if kind == "samples":
        return dict(family="samples", n=_log(rng, 33, 400), flux=rng.choice(FLUXES[:3]), recon="minmod",
                    samples=rng.randint(2, 3), steps=rng.randint(8, 24))
    if kind == "ensemble":
        n = _log(rng, 33, 257)
        levels = rng.choice([1, 1, 2])
        room = 40e6 / (n * n * (1 if levels == 1 else 2))
        return dict(family="ensemble", ic="kh", n=n, flux=rng.choice(FLUXES[:3]),
                    recon=rng.choice(["minmod", "minmod", "first"]),
                    samples=32 * max(levels, min(_log(rng, 1, 32), int(room / 32))), steps=rng.randint(4, 10),
                    levels=levels)
    if kind == "ensemble_cylinder":
        n, nt = _log(rng, 24, 128), _log(rng, 48, 256)
        room = 4e6 / (n * nt)
        return dict(family="ensemble", ic="cylinder", n=n, nt=nt, flux=rng.choice(FLUXES[:2]), recon="minmod",
                    samples=32 * max(1, min(_log(rng, 1, 8), int(room / 32))), steps=rng.randint(8, 24),
                    outputs=rng.randint(1, 2), levels=1)
    if kind == "fit":
        return dict(family="fit", rows=_log(rng, 64, 512), din=rng.choice([3, 20]), batch=rng.choice([32, 64, 100, 128]),
                    epochs=rng.randint(40, 160))
    return dict(family="predict", rows=_log(rng, 1, 1 << 20), din=rng.choice([3, 20]), precision=rng.choice([0, 1, 1]))


# ------------------------------------------------------------- meshes and inputs

@functools.lru_cache(maxsize=6)
def _mesh(ic, n, nt=0):
    """The triangulation a case runs on and its dual geometry, as a program reads them once."""
    m = cases.cylinder_mesh(n, nt) if ic == "cylinder" else cases.vortex_mesh(n) if ic == "vortex" else cases.kh_mesh(n)
    return m, preproc.preprocess(m)


def _rng(seed):
    return np.random.default_rng(seed)


def _dt(case, n):
    """About one time step of the mesh, to choose output times."""
    return {"kh": 0.0785, "vortex": 1.5}[case.get("ic", "kh")] / (n - 1)


def _vortex(coords, seed):
    """The isentropic vortex, its strength and centre drawn from the seed."""
    r = _rng(seed)
    beta, shift = r.uniform(4.0, 5.5), r.uniform(-1.0, 1.0, 2)
    return cases.vortex_ic(coords - shift, beta=beta)


def _inputs(case, seed):
    """(count, 3) Mach number, Reynolds number and inflow angle."""
    return cylinder.draw_inputs(case.get("samples", 1), seed)


CYL_DT = 1.8e-4                           # about one time step of the cylinder meshes


def _level_n(case):
    return [(case["n"] - 1) * 2 ** l + 1 for l in range(case["levels"])]


def _level_samples(case):
    return [max(32, case["samples"] // 4 ** l // 32 * 32) for l in range(case["levels"])]


def _surrogate_data(case, seed):
    """Inputs, a smooth three-component response with the solver's scales, and initial weights."""
    r = _rng(seed)
    d = case["din"]
    x = r.uniform(0.0, 1.0, (case["rows"], d)) if d != 3 else np.stack(
        [r.uniform(0.15, 0.25, case["rows"]), r.uniform(80.0, 120.0, case["rows"]),
         r.uniform(-2.0, 2.0, case["rows"])], axis=1)
    z = (x - x.mean(0)) / (x.std(0) + 1e-12)
    a = r.normal(size=(d, 3)) / math.sqrt(d)
    y = np.stack([1.3 + 0.1 * np.tanh(z @ a[:, 0]), 0.01 * np.exp(0.3 * (z @ a[:, 1])), 0.25 + 0.02 * np.sin(z @ a[:, 2])], 1)
    w = [r.uniform(-1.0, 1.0, (o, i)) * math.sqrt(6.0 / i) for o, i in ((64, d), (64, 64), (64, 64), (3, 64))]
    theta = np.concatenate([np.concatenate([m.ravel(), np.zeros(m.shape[0])]) for m in w]).astype(np.float32)
    return x, y, theta


def _config(case, final_time, stamps):
    return dict(flux=case["flux"], reconstruct=case["recon"], boundary=PERIODIC, final_time=final_time,
                time_stamps=stamps, cfl=0.8, time_scheme=case.get("scheme", "ssprk3"))


def _cyl_configs(case, seed):
    T = case["steps"] * CYL_DT
    return [cases.cylinder_config(m, re, a, T, case["outputs"], flux=case["flux"], recon=case["recon"])
            for m, re, a in _inputs(case, seed)]


def prepare(case, seed):
    f = case["family"]
    s = dict(case=case)
    if f in ("fit", "predict"):
        s["x"], s["y"], s["theta"] = _surrogate_data(case, seed)
        s["net"] = mlp.MLP(case["din"], 3, seed=1)
        s["net"].params = s["theta"]
        if f == "predict":                 # standardised as a fit on a study's runs leaves it
            s["net"].xm, s["net"].xs = s["x"].mean(0), s["x"].std(0) + 1e-12
            s["net"].ym, s["net"].ys = s["y"].mean(0), s["y"].std(0) + 1e-300
        return s
    if f == "ensemble":
        if case["ic"] == "cylinder":
            m, g = _mesh("cylinder", case["n"], case["nt"])
            cfgs = _cyl_configs(case, seed)
            s["b"] = batch.Batch([(abi.Problem(g, cfgs[0]), case["samples"])])
            s["mu"] = [c["mu_ref"] for c in cfgs]
            s["bv"] = np.stack([abi.bface_values(g, c["boundary"]) for c in cfgs])
            s["ic"] = np.stack([cases.cylinder_ic(m.coords[:1], q[0], q[2])[0] for q in _inputs(case, seed)])
            return s
        T = case["steps"] * _dt(case, _level_n(case)[-1])
        P = [abi.Problem(_mesh("kh", n)[1], _config(case, T, 1)) for n in _level_n(case)]
        s["b"] = batch.Batch(list(zip(P, _level_samples(case))))
        s["rows"] = [_rng([seed, l]).uniform(0.0, 1.0, (k, cases.KH_RND_PER_SAMPLE))
                     for l, k in enumerate(_level_samples(case))]
        return s
    if f == "samples":
        _, g = _mesh("kh", case["n"])
        s["solver"] = gpu.Solver(abi.Problem(g, _config(case, case["steps"] * _dt(case, case["n"]), 1)))
        s["fields"] = gpu.expr_fields(cases.kh_expressions())
        s["rows"] = _rng(seed).uniform(0.0, 1.0, (case["samples"], cases.KH_RND_PER_SAMPLE))
        s["solver"].moments_init(1, EXTRAS)
        return s
    if case["ic"] == "cylinder":
        m, g = _mesh("cylinder", case["n"], case["nt"])
        q = _inputs(case, seed)[0]
        s["problem"] = abi.Problem(g, _cyl_configs(case, seed)[0])
        prim = cases.cylinder_ic(m.coords, q[0], q[2])
    else:
        m, g = _mesh(case["ic"], case["n"])
        s["problem"] = abi.Problem(g, _config(case, 1.0e9, 1))
        prim = _vortex(m.coords, seed) if case["ic"] == "vortex" else cases.kh_ic(m.coords, *cases.kh_coefficients(seed))
    s["solver"] = gpu.Solver(s["problem"])
    s["in"], _ = s["solver"].output_buffers(with_gradients=False)    # pinned, as the bindings offer them
    s["out"], _ = s["solver"].output_buffers(with_gradients=False)
    s["in"][:] = prim
    return s


def run(s):
    case = s["case"]
    f = case["family"]
    if f == "fit":
        s["net"].params = s["theta"]       # a fresh network, its optimiser state reset
        losses = s["net"].fit(s["x"], s["y"], epochs=case["epochs"], batch=case["batch"], lr=2e-3)
        return dict(losses=losses, params=s["net"].params)
    if f == "predict":
        return s["net"].predict(s["x"], precision=case["precision"])
    if f == "ensemble":
        b, out = s["b"], {}
        if case["ic"] == "cylinder":
            b.set_parameters(0, mu_ref=s["mu"], bface_values=s["bv"])
            b.set_uniform(0, s["ic"])
            for i in range(1, case["outputs"] + 1):
                b.advance(i)
                out["forces%d" % i] = b.forces(0, cylinder.FORCES)
            out["first"] = b.get_state(0, 0)
            return out
        for l, rows in enumerate(s["rows"]):
            b.set_kh(l, rows)
        b.advance(1)
        for l in range(case["levels"]):
            out["integrals%d" % l] = b.integrals(l)
            out["moments%d" % l] = b.moments(l, EXTRAS)
            out["last%d" % l] = b.get_state(l, b.S[l] - 1)
        return out
    if f == "samples":
        v = s["solver"]
        for k in range(case["samples"]):
            v.set_state_expr(s["fields"], s["rows"][k])
            v.advance(1)
            v.moments_increment(0, k + 1)
        v.moments_finalize(0, case["samples"])
        return v.moments_get(0)
    v = s["solver"]
    if case["ic"] == "cylinder":
        v.update_parameters(s["problem"])
        v.set_state(s["in"])
        rows = [v.forces(cylinder.FORCES)]
        for i in range(1, case["outputs"] + 1):
            info = v.advance(i)
            rows.append(v.forces(cylinder.FORCES))
        return dict(state=v.get_state(s["out"]), forces=np.stack(rows), time=info[0])
    v.set_state(s["in"])
    info = v.step(case["steps"])
    return dict(state=v.get_state(s["out"]), clock=info[:2], residual=info[2])


def work(case):
    """Per stage and vertex: the state read and written once, U_old read in all but the first, and
    the mesh (a normal and two indices per edge, coordinates and areas per vertex) once per stage
    however many members share it; FP64 8 bytes, FP32 members 4.  Operations of the flux, the
    gradients and the update as written on paper."""
    f = case["family"]
    d = case.get("din", 0)
    if f == "fit":
        p = 64 * d + 2 * 64 * 64 + 3 * 64
        return dict(bytes=4 * (case["rows"] * (d + 3) + 2 * (p + 195)), flops=6.0 * p * case["rows"] * case["epochs"])
    if f == "predict":
        return dict(bytes=8 * case["rows"] * (d + 3), flops=2.0 * case["rows"] * (64 * d + 2 * 64 * 64 + 3 * 64))
    stages = 4 if case.get("scheme") == "rk4" else 3
    cyl = case.get("ic") == "cylinder"
    tecno = case["flux"].startswith("kepes")
    per_edge = (250 if tecno else 70) + (150 if cyl else 0)
    per_vertex = 120 + (72 if tecno and case["recon"] != "first" else 0)
    if f == "ensemble":
        levels = list(zip([(case["n"], case["nt"])] if cyl else [(n, n) for n in _level_n(case)], _level_samples(case)))
        word, count = 4, [k for _, k in levels]
    else:
        levels = [((case["n"], case.get("nt", case["n"])), 1)]
        word, count = 8, [case.get("samples", 1)]
    total = dict(bytes=0.0, flops=0.0)
    for ((a, b), members), k in zip(levels, count):
        v = a * b
        passes = case["steps"] * stages * (k if f == "samples" else 1)
        # finer levels take proportionally smaller steps to the common output time
        passes = passes * a / levels[-1][0][0]
        total["bytes"] += passes * v * (word * (4 + 4 + 4 * (stages - 1) / stages) * members + word * (3 * 2 + 3) + 24)
        total["flops"] += passes * v * members * (3.0 * per_edge + per_vertex)
    return total


# --------------------------------------------------------------- the method in 64 bits

GAM, PRANDTL = 1.4, 0.72


class _Method:
    """The vertex-centred scheme on one triangulation: `state` is (T, u, v, p), each (vertices, members)."""

    def __init__(self, mesh, flux, recon, scheme):
        self.flux, self.recon, self.scheme = flux, recon, scheme
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        xy, cells = t(np.asarray(mesh.coords, np.float64)), t(np.asarray(mesh.cells, np.int64))
        self.V, self.dev, self.cells, self.xy = xy.shape[0], dev, cells, xy
        x = xy[cells]                                             # (C, 3, 2)
        e1, e2 = x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]
        area = 0.5 * (e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0])
        cen = x.mean(1)
        opp = x[:, [1, 2, 0]] - x[:, [2, 0, 1]]                   # opposite edge of each vertex
        self.N = torch.stack([opp[..., 1], -opp[..., 0]], -1)     # P1 normals
        self.inv2a = 1.0 / (2.0 * area)
        A = torch.zeros(self.V, dtype=torch.float64, device=dev).index_add_(0, cells.reshape(-1), (area / 3.0).repeat_interleave(3))
        self.sets = [s for s in mesh.periodic_sets]
        if self.sets:                                             # member -> set number, and the members
            self.pm = t(np.concatenate([np.asarray(s) for s in self.sets]))
            self.ps = t(np.concatenate([np.full(len(s), i) for i, s in enumerate(self.sets)]))
        self.w = torch.ones(self.V, dtype=torch.float64, device=dev)
        if self.sets:
            size = torch.bincount(self.ps).double()
            self.w[self.pm] = 1.0 / size[self.ps]
        self.A = self.periodic(A[:, None])[:, 0]
        # dual normals: the segment from each half edge's midpoint to the centroid
        i, j = cells[:, [0, 1, 2]].reshape(-1), cells[:, [1, 2, 0]].reshape(-1)
        d = cen.repeat_interleave(3, 0) - 0.5 * (xy[i] + xy[j])
        n = torch.stack([d[:, 1], -d[:, 0]], 1)
        lo, hi = torch.minimum(i, j), torch.maximum(i, j)
        key, inv, cnt = torch.unique(lo * self.V + hi, return_inverse=True, return_counts=True)
        self.a, self.b = key // self.V, key % self.V
        self.n = torch.zeros(key.shape[0], 2, dtype=torch.float64, device=dev).index_add_(0, inv, torch.where((i == lo)[:, None], n, -n))
        self.d = xy[self.b] - xy[self.a]
        self.area = self.n.norm(dim=1)
        # boundary faces that are not periodic, in the orientation of their cell
        bf = np.asarray(mesh.bfaces, np.int64)
        bf = bf[bf[:, 3] == 0]
        self.nb = len(bf)
        if self.nb:
            at = torch.full((key.shape[0],), -1, dtype=torch.int64, device=dev)
            once = (cnt[inv] == 1).nonzero()[:, 0]
            at[inv[once]] = once
            v0, v1 = t(bf[:, 0]), t(bf[:, 1])
            half = at[torch.searchsorted(key, torch.minimum(v0, v1) * self.V + torch.maximum(v0, v1))]
            self.b0, self.b1, self.bc = i[half], j[half], half // 3
            e = xy[self.b1] - xy[self.b0]
            self.bn = torch.stack([e[:, 1], -e[:, 0]], 1)
            self.wall = t(bf[:, 2]) == 1
            self.inner = torch.ones(cells.shape[0], dtype=torch.bool, device=dev)
            self.inner[self.bc] = False

    def periodic(self, q):
        if self.sets:
            s = torch.zeros(len(self.sets), q.shape[1], dtype=q.dtype, device=q.device).index_add_(0, self.ps, q[self.pm])
            q = q.clone()
            q[self.pm] = s[self.ps]
        return q

    @staticmethod
    def entropy(T, u, v, p):
        rho, beta = p / T, 0.5 / T
        s = torch.log(p) - GAM * torch.log(rho)
        return [(GAM - s) / (GAM - 1.0) - beta * (u * u + v * v), 2 * beta * u, 2 * beta * v, -2 * beta]

    @staticmethod
    def log_mean(a, b):
        f = (b - a) / (b + a)
        u = f * f
        F = torch.where(u < 1e-2, 1.0 + u / 3.0 + u * u / 5.0 + u * u * u / 7.0, torch.log(b / a) / (2.0 * torch.where(f == 0, 1.0, f)))
        return 0.5 * (a + b) / F

    def limited(self, a, b):
        if self.recon == "van_albada":
            s = torch.clamp((2 * a * b + 1e-14) / (a * a + b * b + 1e-14), min=0.0)
            return 0.25 * s * ((1 - s / 3) * a + (1 + s / 3) * b)
        m = torch.minimum(a.abs(), b.abs())
        return 0.5 * torch.where((a > 0) & (b > 0), m, torch.where((a < 0) & (b < 0), -m, torch.zeros_like(m)))

    def num_flux(self, L, R, n, area, grads=None, d=None):
        Tl, ul, vl, pl = L
        Tr, ur, vr, pr = R
        nx, ny, ar = (n[:, :1] / area[:, None]), (n[:, 1:] / area[:, None]), area[:, None]
        rl, rr = pl / Tl, pr / Tr
        if self.flux == "kep":
            H = 0.5 * (GAM * Tl / (GAM - 1) + 0.5 * (ul * ul + vl * vl) + GAM * Tr / (GAM - 1) + 0.5 * (ur * ur + vr * vr))
            p, rho, ux, uy = 0.5 * (pl + pr), 0.5 * (rl + rr), 0.5 * (ul + ur), 0.5 * (vl + vr)
            m = rho * (ux * nx + uy * ny)
            return [ar * q for q in (m, nx * p + ux * m, ny * p + uy * m, H * m)]
        if self.flux == "roe_ec":
            bl, br = torch.sqrt(rl / pl), torch.sqrt(rr / pr)
            z1, zx, zy = 0.5 * (bl + br), 0.5 * (bl * ul + br * ur), 0.5 * (bl * vl + br * vr)
            z5, z1l, z5l = 0.5 * (bl * pl + br * pr), self.log_mean(bl, br), self.log_mean(bl * pl, br * pr)
            m = z5l * (zx * nx + zy * ny)
            fx, fy = nx * z5 / z1 + zx / z1 * m, ny * z5 / z1 + zy / z1 * m
            e = 0.5 / z1 * ((GAM + 1) / (GAM - 1) / z1l * m + zx * fx + zy * fy)
            return [ar * q for q in (m, fx, fy, e)]
        bl, br = 0.5 / Tl, 0.5 / Tr
        rho, beta = self.log_mean(rl, rr), self.log_mean(bl, br)
        p = 0.5 * (rl + rr) / (bl + br)
        ux, uy = 0.5 * (ul + ur), 0.5 * (vl + vr)
        vn = ux * nx + uy * ny
        m = rho * vn
        fx, fy = nx * p + ux * m, ny * p + uy * m
        k2 = 0.5 * (ul * ul + vl * vl + ur * ur + vr * vr)
        e = 0.5 * (1.0 / ((GAM - 1) * beta) - k2) * m + ux * fx + uy * fy
        if self.flux == "kepec":
            return [ar * q for q in (m, fx, fy, e)]
        a = torch.sqrt(0.5 * GAM / beta)
        k = 0.5 * (ux * ux + uy * uy)
        H, v1 = a * a / (GAM - 1) + k, ux * ny - uy * nx
        one, nil = torch.ones_like(a), torch.zeros_like(a)
        S = [torch.sqrt(0.5 * rho / GAM), torch.sqrt((GAM - 1) * rho / GAM), torch.sqrt(p), torch.sqrt(0.5 * rho / GAM)]
        col = [(one, ux - a * nx, uy - a * ny, H - a * vn), (one, ux, uy, k), (nil, ny + nil, -nx + nil, v1),
               (one, ux + a * nx, uy + a * ny, H + a * vn)]
        if self.flux == "kepes_tecno_roe":
            lam = [(vn - a).abs(), vn.abs(), vn.abs(), (vn + a).abs()]
        else:
            lam = [vn.abs() + a] * 4
        Vl, Vr = self.entropy(*L), self.entropy(*R)
        dV = [y - x for x, y in zip(Vl, Vr)]
        out = [nil, nil, nil, nil]
        for c, s, l in zip(col, S, lam):
            z = s * sum(x * y for x, y in zip(c, dV))
            if grads is not None:
                sl, sr = (s * sum(x * (g[2 * q] * d[:, :1] + g[2 * q + 1] * d[:, 1:]) for q, x in enumerate(c)) for g in grads)
                z = z - self.limited(2 * sr - z, z) - self.limited(2 * sl - z, z)
            out = [o + s * l * z * x for o, x in zip(out, c)]
        return [ar * (q - 0.5 * o) for q, o in zip((m, fx, fy, e), out)]

    def cell_sums(self, q):
        """Sum of N_k W_k over each cell's vertices with the walls' corrections: 8 x (cells, members)."""
        W = self.entropy(*q)
        out = []
        for w in W:
            c = w[self.cells]                                     # (C, 3, members)
            out += [(self.N[..., 0, None] * c).sum(1), (self.N[..., 1, None] * c).sum(1)]
        if self.nb:
            at = self.wall.nonzero()[:, 0]
            v0, v1, c, n = self.b0[at], self.b1[at], self.bc[at], self.bn[at]
            B0, B1 = (self.entropy(q[0][v], 0 * q[1][v], 0 * q[2][v], q[3][v]) for v in (v0, v1))
            for k in range(4):
                dW = 0.5 * (B0[k] + B1[k] - W[k][v0] - W[k][v1])
                out[2 * k].index_add_(0, c, n[:, :1] * dW)
                out[2 * k + 1].index_add_(0, c, n[:, 1:] * dW)
        return W, out

    def to_vertices(self, c):
        v = torch.zeros(self.V, c.shape[1], dtype=c.dtype, device=c.device)
        for k in range(3):
            v.index_add_(0, self.cells[:, k], c)
        return self.periodic(v)

    def gradients(self, cells):
        return [self.to_vertices(c) / (6.0 * self.A[:, None]) for c in cells]

    def residual(self, q, mu):
        R = [torch.zeros_like(q[0]) for _ in range(4)]
        grads = None
        need = self.flux.startswith("kepes") and self.recon != "first"
        if need or mu is not None:
            W, cell = self.cell_sums(q)
            if need:
                G = self.gradients(cell)
                grads = ([g[self.a] for g in G], [g[self.b] for g in G])
        F = self.num_flux([x[self.a] for x in q], [x[self.b] for x in q], self.n, self.area, grads, self.d)
        for r, f in zip(R, F):
            r.index_add_(0, self.a, f).index_add_(0, self.b, -f)
        if self.nb:
            for v in (self.b0, self.b1):
                w, f = self.wall, ~self.wall
                p = q[3][v[w]]
                R[1].index_add_(0, v[w], 0.5 * self.bn[w][:, :1] * p)
                R[2].index_add_(0, v[w], 0.5 * self.bn[w][:, 1:] * p)
                x = [c[v[f]] for c in q]
                F = self.num_flux(x, [far.expand_as(c) for far, c in zip(self.far, x)], self.bn[f], self.bn[f].norm(dim=1))
                for r, y in zip(R, F):
                    r.index_add_(0, v[f], 0.5 * y)
        if mu is not None:
            self.viscous(q, W, cell, mu, R)
        return [self.periodic(r) for r in R]

    def viscous(self, q, W, cell, mu, R):
        kk = mu * (GAM / (GAM - 1.0)) / PRANDTL
        dE = [c * self.inv2a[:, None] for c in cell]
        st = [w[self.cells].mean(1) for w in W]
        w = self.wall[:, None]
        ends = []
        for v in (self.b0, self.b1):
            x = [c[v] for c in q]
            ends.append(self.entropy(x[0], torch.where(w, 0.0, x[1]), torch.where(w, 0.0, x[2]), x[3]))
        for k in range(4):
            st[k][self.bc] = 0.5 * (ends[0][k] + ends[1][k])
        e1, e2, e4 = st[1] / st[3], st[2] / st[3], 1.0 / st[3]
        d1x, d1y, d2x, d2y, d4x, d4y = dE[2], dE[3], dE[4], dE[5], dE[6], dE[7]
        # du_i/dx_j = -(dV_i - e_i dV4) / V4 and so on: stresses and heat flux from the entropy variables
        ux, uy = (-(d1x - e1 * d4x) * e4, -(d1y - e1 * d4y) * e4)
        vx, vy = (-(d2x - e2 * d4x) * e4, -(d2y - e2 * d4y) * e4)
        sxx, syy, sxy = mu * (4 * ux - 2 * vy) / 3, mu * (4 * vy - 2 * ux) / 3, mu * (uy + vx)
        u, v = -e1, -e2
        hx, hy = kk * d4x * e4 * e4, kk * d4y * e4 * e4            # k grad T, T = -1 / V4
        fx = (-sxx, -sxy, -(u * sxx + v * sxy + hx))
        fy = (-sxy, -syy, -(u * sxy + v * syy + hy))
        flux = lambda n, c=slice(None): [-(a[c] * n[:, :1] + b[c] * n[:, 1:]) for a, b in zip(fx, fy)]  # noqa: E731
        for k in range(3):
            for r, f in zip(R[1:], flux(self.N[:, k])):
                r.index_add_(0, self.cells[:, k], 0.5 * f)
        fb = flux(self.bn, self.bc)
        normal = (hx[self.bc] * self.bn[:, :1] + hy[self.bc] * self.bn[:, 1:])
        fb[2] = torch.where(w, fb[2] - normal, fb[2])              # adiabatic wall
        for v in (self.b0, self.b1):
            for r, f in zip(R[1:], fb):
                r.index_add_(0, v, -0.5 * f)

    def time_step(self, q, mu):
        T, u, v, p = q
        c = torch.sqrt(GAM * T)
        lam = torch.zeros_like(T)
        for at in (self.a, self.b):
            lam.index_add_(0, at, (u[at] * self.n[:, :1] + v[at] * self.n[:, 1:]).abs() + c[at] * self.area[:, None])
            if mu is not None:
                lam.index_add_(0, at, mu * (self.area / self.d.norm(dim=1))[:, None] * (T / p)[at])
        if self.nb:
            for at in (self.b0, self.b1):
                lam.index_add_(0, at, 0.5 * ((u[at] * self.bn[:, :1] + v[at] * self.bn[:, 1:]).abs() + c[at] * self.bn.norm(dim=1)[:, None]))
        return (0.8 * self.A[:, None] / self.periodic(lam)).min(0).values

    @staticmethod
    def conserved(q):
        T, u, v, p = q
        rho = p / T
        return [rho, rho * u, rho * v, p / (GAM - 1) + 0.5 * rho * (u * u + v * v)]

    @staticmethod
    def primitive(U):
        r, x, y, E = U
        p = (GAM - 1) * (E - 0.5 * (x * x + y * y) / r)
        return [p / r, x / r, y / r, p]

    def step(self, q, dt, mu):
        U0 = U = self.conserved(q)
        f = dt[None, :] / self.A[:, None]
        if self.scheme == "rk4":
            acc = [torch.zeros_like(x) for x in U]
            for w, nxt in ((1, 0.5), (2, 0.5), (2, 1.0), (1, None)):
                R = self.residual(q, mu)
                acc = [a + w * r for a, r in zip(acc, R)]
                U = [u - f * (nxt * r if nxt else a / 6.0) for u, r, a in zip(U0, R, acc)]
                q = self.primitive(U)
            return q
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
            R = self.residual(q, mu)
            U = [a * u0 + b * (u - f * r) for u0, u, r in zip(U0, U, R)]
            q = self.primitive(U)
        return q

    def advance(self, q, t, end, mu=None):
        """Every member from its time to `end`, the last step shortened to meet it."""
        live = t < end
        while bool(live.any()):
            dt = self.time_step(q, mu)
            over = t + dt > end
            dt = torch.where(live, torch.where(over, end - t, dt), 0.0)
            q1 = self.step(q, dt, mu)
            q = [torch.where(live[None, :], y, x) for x, y in zip(q, q1)]
            t = torch.where(live, torch.where(over, torch.full_like(t, end), t + dt), t)
            live = t < end
        return q, t

    def forces(self, q, mu):
        """Pressure and viscous force on the wall, per member."""
        _, cell = self.cell_sums(q)
        G = self.gradients(cell)
        at = self.wall.nonzero()[:, 0]
        n = self.bn[at]
        grad, p, T = [], 0.0, 0.0
        for v in (self.b0[at], self.b1[at]):
            V5 = -1.0 / q[0][v]
            # on the wall u = v = 0, so grad u = -grad V2 / V5
            grad.append([-G[k][v] / V5 for k in (2, 3, 4, 5)])
            p, T = p + 0.5 * q[3][v], T + 0.5 * q[0][v]
        ux, uy, vx, vy = (0.5 * (x + y) for x, y in zip(*grad))
        div = (ux + vy) / 3.0
        sxx, syy, sxy = 2 * mu * (ux - div), 2 * mu * (vy - div), mu * (uy + vx)
        nx, ny = n[:, :1], n[:, 1:]
        return torch.stack([(nx * p).sum(0), (ny * p).sum(0), -(sxx * nx + sxy * ny).sum(0), -(sxy * nx + syy * ny).sum(0)], 1)


def _records(q, s=0):
    """PrimVar records (T, p, u, v, w) of member s."""
    T, u, v, p = (x[:, s] for x in q)
    return torch.stack([T, p, u, v, torch.zeros_like(T)], 1).cpu()


def _quantities(q):
    T, u, v, p = q
    rho = p / T
    return [T, p, u, v, torch.zeros_like(T), rho, torch.sqrt(u * u + v * v) / torch.sqrt(GAM * T),
            torch.log(p) - GAM * torch.log(rho)]


def _kh_states(m, rows):
    """The Kelvin-Helmholtz states (T, u, v, p) of random-number rows, one member a row."""
    x, r = m.xy[:, :1], torch.as_tensor(rows, device=m.dev)
    half = r.shape[1] // 2
    s = sum(r[None, :, k - 1] * torch.sin(2 * math.pi * k * x + 2 * math.pi * r[None, :, half + k - 1]) for k in range(1, half + 1))
    inside = ((m.xy[:, 1:] - 0.5).abs() < 0.25).expand_as(s)
    p = torch.full_like(s, 2.5)
    return [p / torch.where(inside, 2.0, 1.0), torch.where(inside, 0.5, -0.5).double(), 0.01 * s, p]


def _moments(x):
    """Mean, sum of squares and squared deviations over the members (last axis)."""
    mean, sq, dev = x.mean(-1), (x * x).sum(-1), ((x - x.mean(-1, keepdim=True)) ** 2).sum(-1)
    return [mean.cpu(), sq.cpu(), dev.cpu()]


def _exact_surrogate(case, seed):
    x, y, theta = _surrogate_data(case, seed)
    xm, xs, ym, ys = x.mean(0), x.std(0) + 1e-12, y.mean(0), y.std(0) + 1e-300
    X, Y = torch.as_tensor((x - xm) / xs), torch.as_tensor((y - ym) / ys)
    th, P = torch.as_tensor(theta.astype(np.float64)), []
    for o, i in ((64, case["din"]), (64, 64), (64, 64), (3, 64)):
        P += [th[:o * i].reshape(o, i).clone(), th[o * i:o * i + o].clone()]
        th = th[o * i + o:]
    gelu = lambda z: 0.5 * z * (1 + torch.erf(z / math.sqrt(2.0)))  # noqa: E731

    def forward(a):
        zs = []
        for k in range(3):
            zs.append(a @ P[2 * k].T + P[2 * k + 1])
            a = gelu(zs[-1])
        return a @ P[6].T + P[7], zs, a
    if case["family"] == "predict":
        return torch.cat([forward(X[i:i + 65536])[0] for i in range(0, X.shape[0], 65536)]).numpy() * ys + ym
    M, S, step, losses = [torch.zeros_like(p) for p in P], [torch.zeros_like(p) for p in P], 0, []
    for _ in range(case["epochs"]):
        for at in range(0, X.shape[0], case["batch"]):
            xb, tb = X[at:at + case["batch"]], Y[at:at + case["batch"]]
            out, zs, a = forward(xb)
            losses_now = ((out - tb) ** 2).mean()
            d, g = 2.0 * (out - tb) / tb.numel(), [None] * 8
            for k in (3, 2, 1, 0):
                prev = gelu(zs[k - 1]) if k else xb
                g[2 * k], g[2 * k + 1] = d.T @ prev, d.sum(0)
                if k:
                    z = zs[k - 1]
                    d = (d @ P[2 * k]) * (0.5 * (1 + torch.erf(z / math.sqrt(2.0))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi))
            step += 1
            for p, m, s, q in zip(P, M, S, g):
                m.mul_(0.9).add_(0.1 * q)
                s.mul_(0.999).add_(0.001 * q * q)
                p.sub_(2e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(s / (1 - 0.999 ** step)) + 1e-8))
        losses.append(losses_now)
    return dict(losses=torch.stack(losses), params=torch.cat([p.reshape(-1) for p in P]))


def exact(case, seed):
    f = case["family"]
    if f in ("fit", "predict"):
        return _exact_surrogate(case, seed)
    cyl = case.get("ic") == "cylinder"
    mesh = lambda n: _mesh("cylinder" if cyl else case.get("ic", "kh"), n, case.get("nt", 0))[0]  # noqa: E731
    new = lambda n: _Method(mesh(n), case["flux"], case["recon"], case.get("scheme", "ssprk3"))  # noqa: E731
    zeros = lambda m, k: torch.zeros(k, dtype=torch.float64, device=m.dev)  # noqa: E731
    if cyl:
        m = new(case["n"])
        inp = _inputs(case, seed)
        free = np.array([cases.cylinder_freestream(mach, angle) for mach, _, angle in inp])       # T, u, v, p
        mu = torch.as_tensor(np.array([cases.cylinder_viscosity(a, b) for a, b, _ in inp]), device=m.dev)
        m.far = [torch.as_tensor(np.ascontiguousarray(free[None, :, c]), device=m.dev) for c in range(4)]
        q, t = [x.expand(m.V, -1).clone() for x in m.far], zeros(m, len(inp))
        rows, T = [m.forces(q, mu)], case["steps"] * CYL_DT
        for i in range(1, case["outputs"] + 1):
            q, t = m.advance(q, t, i * (T / case["outputs"]), mu)
            rows.append(m.forces(q, mu))
        if f == "single":
            return dict(state=_records(q), forces=torch.stack(rows).cpu(), time=np.float64(t[0].item()))
        return dict({"forces%d" % i: r[:, None].cpu() for i, r in enumerate(rows) if i}, first=_records(q))
    if f == "single":
        m = new(case["n"])
        xy = np.asarray(mesh(case["n"]).coords)
        prim = _vortex(xy, seed) if case["ic"] == "vortex" else cases.kh_ic(xy, *cases.kh_coefficients(seed))
        q = [torch.as_tensor(np.ascontiguousarray(prim[:, c:c + 1]), device=m.dev) for c in (0, 2, 3, 1)]
        time = 0.0
        for _ in range(case["steps"]):
            dt = m.time_step(q, None).min().reshape(1)
            q, time = m.step(q, dt, None), time + float(dt)
        return dict(state=_records(q), clock=torch.tensor([time, float(dt)], dtype=torch.float64), residual=None)
    if f == "samples":
        m = new(case["n"])
        rows = _rng(seed).uniform(0.0, 1.0, (case["samples"], cases.KH_RND_PER_SAMPLE))
        q, _ = m.advance(_kh_states(m, rows), zeros(m, len(rows)), case["steps"] * _dt(case, case["n"]))
        mean, sq, dev = _moments(torch.stack(_quantities(q), 1))
        return [mean, sq / case["samples"], dev / (case["samples"] - 1.0)]
    out, T = {}, case["steps"] * _dt(case, _level_n(case)[-1])
    for l, (n, S) in enumerate(zip(_level_n(case), _level_samples(case))):
        m = new(n)
        rows, got, ints = _rng([seed, l]).uniform(0.0, 1.0, (S, cases.KH_RND_PER_SAMPLE)), [], []
        most = max(1, int(6e6 / (n * n)))
        for at in range(0, S, most):
            part = rows[at:at + most]
            q, _ = m.advance(_kh_states(m, part), zeros(m, len(part)), T)
            got.append([x for x in q])
            Tq, u, v, p = q
            rho, aw = p / Tq, (m.A * m.w)[:, None]
            ints.append(torch.stack([(0.5 * rho * v * v * aw).sum(0), (0.5 * rho * u * u * aw).sum(0),
                                     (-rho * (torch.log(p) - GAM * torch.log(rho)) / (GAM - 1) * aw).sum(0)], 1))
        out["integrals%d" % l] = torch.cat(ints).cpu()
        q = [torch.cat([g[c] for g in got], 1) for c in range(4)]
        cols = [_moments(x) for x in _quantities(q)]
        out["moments%d" % l] = [torch.stack([c[k] for c in cols], 1) for k in range(3)]
        out["last%d" % l] = _records(q, S - 1)
    return out
