"""Performance cases of the droplet step: what a flow solver has this library do.

A pass of a "step" case is a stretch of a flow solver's time loop with its
fields in device memory: every time step hands over new flow fields
(fill_ext), advances the droplets (particle_update_BE, or the three RK3
stages) and takes the six source arrays (particle_coupling_update); at the end
of the stretch the droplet state is read back in list order, as for output or
a restart.  A "job" is one request of the serving loop, from the payload in
pinned host memory to the result on the host.  A "batch" is an ensemble of
boxes that advances as one CUDA graph.

The fields are those of the benchmark configurations (generator.CONFIGS):
divergence-free k^-5/3 velocity, noisy T and q.  Where droplets could drift for
thousands of steps the velocity changes sign from pass to pass, so that they
stay spread over the box however often a pass is repeated.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ntlp_b200
from ntlp_b200 import abi, devgen
from ntlp_b200 import generator as gen

FIELDS = ("u", "v", "w", "T", "q")
STATE = ("xp", "vp", "uf", "Tp", "Tf", "radius", "qinf", "qstar")


def _case(kind, nnx, nny, nnz, n, steps, precision, air="c0", ilin=0, iexner=0, stretch=0.0, stats=False, **kw):
    return dict(kind=kind, nnx=nnx, nny=nny, nnz=nnz, n=n, steps=steps, precision=precision, air=air, ilin=ilin,
                iexner=iexner, stretch=stretch, stats=stats, **kw)


def listed():
    return [
        # the smallest box of the ensemble and serving ranges: launches and latency count
        dict(_case("step", 32, 32, 32, 10_000, 10, "mixed"), name="step_mixed_32"),
        # a small FP64 box with no size a multiple of anything
        dict(_case("step", 33, 29, 31, 12_345, 10, "fp64"), name="step_fp64_ragged"),
        # one request of the serving loop: context, upload, recorded steps, result
        dict(_case("job", 64, 64, 64, 100_000, 8, "mixed"), name="job_mixed_64"),
        # many droplets per cell (the ensemble draws up to 4e6 into a 32^3 box)
        dict(_case("step", 40, 40, 40, 2_000_000, 5, "mixed"), name="step_mixed_dense"),
        # the plain configuration: 1 M droplets on 128^3, FP64, with the
        # statistics that the time loop takes at every step
        dict(_case("step", 128, 128, 128, 1_000_000, 5, "fp64", stats=True), name="step_fp64_1m"),
        # the same box in mixed precision
        dict(_case("step", 128, 128, 128, 1_000_000, 10, "mixed"), name="step_mixed_1m"),
        # trilinear interpolation, a ragged grid, few droplets per cell
        dict(_case("step", 150, 100, 66, 700_001, 10, "mixed", ilin=1), name="linear_mixed_ragged"),
        # the explicit integrator, on droplets whose response time its step resolves
        dict(_case("rk3", 96, 96, 96, 600_000, 4, "fp64", median=5e-5, dt=2e-4), name="rk3_fp64"),
        # uneven boxes advancing together, one graph launch
        dict(_case("batch", 0, 0, 0, 0, 10, "mixed", boxes=16, edge_lo=32, edge_hi=96, n_lo=10_000, n_hi=1_000_000),
             name="ensemble_mixed"),
        # the precision study's box, both precisions
        dict(_case("step", 256, 256, 256, 16_777_216, 4, "mixed", air="c1"), name="step_mixed_16m"),
        dict(_case("step", 256, 256, 256, 16_777_216, 2, "fp64", air="c1"), name="step_fp64_16m"),
        # the spray configuration: stretched grid, wind, droplets near the surface
        dict(_case("step", 512, 512, 128, 67_108_864, 2, "mixed", air="c2", stretch=1.02), name="spray_mixed_67m"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["rk3", "job", "batch"])
    precision = "fp64" if kind == "rk3" else "mixed" if kind == "job" else rng.choice(["mixed", "mixed", "fp64"])
    ilin = rng.choice([0, 0, 0, 0, 1])
    iexner = rng.choice([0, 0, 0, 0, 0, 1])
    steps = rng.randint(2, 8)
    if kind == "batch":
        return _case("batch", 0, 0, 0, 0, steps, precision, ilin=ilin, iexner=iexner, boxes=rng.randint(2, 12),
                     edge_lo=32, edge_hi=rng.randint(48, 96), n_lo=10_000, n_hi=_log_int(rng, 30_000, 500_000))
    nnx, nny, nnz = (_log_int(rng, 24, 160) for _ in range(3))
    n = _log_int(rng, 1e4, min(4e6, 64 * nnx * nny * nnz))
    stretch = rng.choice([0.0, 0.0, 1.02])
    more = dict(median=5e-5, dt=2e-4) if kind == "rk3" else {}
    return _case(kind, nnx, nny, nnz, n, steps, precision, ilin=ilin, iexner=iexner, stretch=stretch,
                 stats=kind == "step" and rng.random() < 0.2, **more)


# ---- inputs -----------------------------------------------------------------
def _params(case):
    # droplets reflect at the floor (icase 0): a box keeps its droplets
    # however often a pass is repeated
    return gen.default_params(ilin=case["ilin"], iexner=case["iexner"], icase=0,
                              precision=1 if case["precision"] == "mixed" else 0)


def _dt(case):
    return case.get("dt", gen.CONFIGS[case["air"]]["dt"])


def _boxes(case, seed):
    """The case's boxes: dicts of grid, flow fields and droplets on the device."""
    dev = torch.device("cuda", torch.cuda.current_device())
    p = _params(case)
    if case["kind"] == "batch":
        specs = devgen.draw_ensemble(case["boxes"], (case["edge_lo"], case["edge_hi"]), (case["n_lo"], case["n_hi"]),
                                     seed=3)   # the sizes are the case's, the contents the seed's
        return [devgen.make_box(s["edge"], s["n"], s["seed"] + seed, p, dev, median=s["median"], T0=s["T0"])
                for s in specs]
    cfg = gen.CONFIGS[case["air"]]
    box = devgen.make_box((case["nnx"], case["nny"], case["nnz"]), case["n"], seed, p, dev, extent=cfg["grid"][3:6],
                          stretch=case["stretch"] or None, rms=cfg["rms"], T0=cfg["T0"], sigT=cfg["sigT"],
                          q0=cfg["q0"], sigq=cfg["sigq"], lapse_per_m=cfg.get("lapse", 0.0),
                          loglaw_top=cfg.get("loglaw"), median=case.get("median", cfg.get("median", 1e-6)),
                          sigma_g=cfg.get("sigma_g", 1.5), bimodal=cfg.get("bimodal"), zfrac=cfg.get("zfrac", 1.0))
    return [box]


def _pinned(t):
    return t.cpu().pin_memory()


def prepare(case, seed):
    boxes, p = _boxes(case, seed), _params(case)
    torch.cuda.synchronize()
    state = dict(case=case, params=p, dt=_dt(case), passes=0, it=2)
    if case["kind"] == "job":
        b = boxes[0]
        state.update(grid=b["grid"], flow={k: _pinned(v) for k, v in b["flow"].items()},
                     droplets={k: _pinned(v) for k, v in b["droplets"].items()})
        return state
    if case["kind"] == "batch":
        B = ntlp_b200.DropletBatch([b["grid"] for b in boxes], p, [int(b["droplets"]["radius"].shape[0]) for b in boxes])
        for i, b in enumerate(boxes):
            B.box_fill_ext(i, b["flow"])
            B.set_box_droplets(i, b["droplets"])
        B.sync()
        state.update(step=B, n=[int(b["droplets"]["radius"].shape[0]) for b in boxes],
                     nodes=[(b["grid"]["nnz"] + 2) * b["grid"]["nny"] * b["grid"]["nnx"] for b in boxes])
        return state
    b = boxes[0]
    S = ntlp_b200.DropletStep(b["grid"], p, case["n"])
    S.set_droplets(b["droplets"])
    flow = b["flow"]
    flows = [flow]
    if case["air"] != "c2":
        flows.append({k: (-v if k in "uvw" else v) for k, v in flow.items()})
    shape = (case["nnx"], case["nny"], case["nnz"] + 2)
    f64 = dict(device=flow["u"].device, dtype=torch.float64)
    state.update(step=S, flows=flows, out=[torch.empty((3,) + shape, **f64)] + [torch.empty(shape, **f64) for _ in range(3)])
    torch.cuda.synchronize()
    return state


# ---- a pass -----------------------------------------------------------------
def _run_job(s):
    n = int(s["droplets"]["radius"].shape[0])
    B = ntlp_b200.DropletBatch([s["grid"]], s["params"], [n])
    try:
        B.box_fill_ext(0, s["flow"], sync=False)
        B.set_box_droplets(0, s["droplets"])
        B.graph_build(s["dt"], 1)
        for it in range(s["case"]["steps"]):
            B.advance_graph(s["dt"], s["it"] + it, 1)
        d = B.get_box_droplets(0)
        return dict(droplets={k: d[k] for k in STATE + ("lid",)}, sources=B.box_sources(0),
                    counters=[v for _, v in sorted(B.box_counters(0).items())])
    finally:
        B.close()


def _run_batch(s):
    B, dev = s["step"], torch.device("cuda", torch.cuda.current_device())
    B.advance_graph(s["dt"], s["it"], s["case"]["steps"])
    s["it"] += s["case"]["steps"]
    out = dict(xp=[], vp=[], Tp=[], radius=[])
    total, nodes = sum(s["n"]), sum(s["nodes"])
    flat = {k: torch.zeros((3 if k in ("xp", "vp") else 1) * total, device=dev, dtype=torch.float64) for k in out}
    src = torch.empty(6 * nodes, device=dev, dtype=torch.float64)
    # the caller's arrays are zeroed on torch's stream, the library copies on its own
    torch.cuda.current_stream().synchronize()
    at, ns, numpart = 0, 0, []
    for i, n in enumerate(s["n"]):
        d = {k: flat[k][3 * at:3 * (at + n)].view(3, n) if k in ("xp", "vp") else flat[k][at:at + n] for k in out}
        view = abi.make_droplets_struct(d, n=n)
        B._check(B.L.ntlp_box_droplets_download(B.h, i, view), "ntlp_box_droplets_download")
        numpart.append(int(view.n))
        m = s["nodes"][i]
        b = src[6 * ns:6 * (ns + m)]
        B._check(B.L.ntlp_box_sources(B.h, i, abi.NTLP_LAYOUT_COLUMN, abi.as_dptr(b[:3 * m]), abi.as_dptr(b[3 * m:4 * m]),
                                      abi.as_dptr(b[4 * m:5 * m]), abi.as_dptr(b[5 * m:])), "ntlp_box_sources")
        at, ns = at + n, ns + m
    return dict(droplets=flat, sources=src, numpart=numpart)


def run(s):
    case = s["case"]
    if case["kind"] == "job":
        return _run_job(s)
    if case["kind"] == "batch":
        return _run_batch(s)
    S, dt, flow = s["step"], s["dt"], s["flows"][s["passes"] % len(s["flows"])]
    s["passes"] += 1
    stats = None
    for k in range(case["steps"]):
        last = k == case["steps"] - 1
        S.fill_ext(flow)
        if case["kind"] == "rk3":
            for stage in (1, 2, 3):
                c = S.particle_update_rk3(stage, dt, s["it"], counters=last and stage == 3)
        else:
            c = S.particle_update_BE(dt, s["it"], counters=last)
        src = S.particle_coupling_update(dt, out=s["out"])
        if case["stats"]:
            stats = S.particle_xy_stats()
        s["it"] += 1
    out = dict(droplets=S.get_droplets_device(keys=STATE + ("lid",)), sources=src, counters=[v for _, v in sorted(c.items())])
    if stats is not None:
        out["stats"] = dict(levels=stats[1], lwp=stats[2])
    return out


def work(case):
    if case["kind"] == "batch":
        specs = devgen.draw_ensemble(case["boxes"], (case["edge_lo"], case["edge_hi"]), (case["n_lo"], case["n_hi"]), seed=3)
        n, nodes = sum(s["n"] for s in specs), sum(s["edge"] ** 2 * (s["edge"] + 2) for s in specs)
    else:
        n, nodes = case["n"], case["nnx"] * case["nny"] * (case["nnz"] + 2)
    # per droplet and step: 14 inputs and 17 outputs of 8 bytes (mixed: the
    # six diagnostics in 4); per node: five fields in, six sources out
    per = 248 if case["precision"] == "fp64" else 224
    stages = 3 if case["kind"] == "rk3" else 1
    points = 216 if case["ilin"] == 0 else 8
    fields = 1 if case["kind"] in ("job", "batch") else case["steps"]
    return dict(bytes=case["steps"] * (stages * n * per + 48 * nodes) + fields * 40 * nodes + 8 * 14 * n,
                flops=case["steps"] * n * (stages * (2 * 5 * points + 300) + 2 * 8 * 6))


# ---- the same in plain torch, 64 bits ---------------------------------------
def _window(idx, x, levels, nnz, wlev):
    """Stencil levels and Lagrange weights of uf_interp's vertical windows
    (particles.f90:635-728), [6, m] each."""
    a = torch.arange(-2, 4, device=x.device)[:, None]
    lev = idx[None] + a
    slot = a + 3                                    # Fortran position 1..6
    k2 = idx[None]
    first, last = torch.full_like(k2, 1), torch.full_like(k2, 6)

    def rule(m, f, l):
        first[m], last[m] = f, l
    if not wlev:
        rule((k2 == 2) | (k2 == nnz - 2), 2, 5)
        rule((k2 == 1) | (k2 == nnz - 1), 3, 4)
        rule(k2 == 0, 4, 5)
        rule(k2 == nnz, 2, 3)
        rule((k2 < 0) | (k2 > nnz), 0, 0)
    else:
        rule((k2 == 1) | (k2 == nnz - 2), 2, 5)
        rule((k2 == 0) | (k2 == nnz - 1), 3, 4)
        rule((k2 < 0) | (k2 >= nnz), 0, 0)
    use = (slot >= first) & (slot <= last)
    z = levels[lev.clamp(0, levels.numel() - 1)]
    return lev.clamp(0, levels.numel() - 1), _lagrange(x, z, use)


def _lagrange(x, nodes, use):
    w = []
    for j in range(6):
        t = torch.ones_like(x)
        for k in range(6):
            if k != j:
                f = (x - nodes[k]) / torch.where(use[k] & use[j], nodes[j] - nodes[k], torch.ones_like(x))
                t = t * torch.where(use[k], f, torch.ones_like(x))
        w.append(torch.where(use[j], t, torch.zeros_like(x)))
    return w


class _Exact:
    def __init__(self, grid, p, flow):
        self.g, self.p, self.f = grid, p, flow
        dev = flow["u"].device
        self.z, self.zz, self.dzw, self.dzu = (torch.as_tensor(grid[k], device=dev) for k in ("z", "zz", "dzw", "dzu"))
        self.dx, self.dy = grid["xl"] / grid["nnx"], grid["yl"] / grid["nny"]

    def base(self, x):
        """ipt, jpt (floor(x/dx)+1) and the levels at or below the droplet on zz and z."""
        nnz = self.g["nnz"]
        return (torch.floor(x[0] / self.dx).long() + 1, torch.floor(x[1] / self.dy).long() + 1,
                (torch.searchsorted(self.zz, x[2], right=True) - 1).clamp(0, nnz),
                (torch.searchsorted(self.z, x[2], right=True) - 1).clamp(0, nnz))

    def col(self, ix, iy):
        nx, ny = self.g["nnx"], self.g["nny"]
        return ((iy - 1) % ny) * nx + (ix - 1) % nx

    def interp(self, x):
        g, nnz = self.g, self.g["nnz"]
        plane = g["nnx"] * g["nny"]
        i0, j0, ku, kw = self.base(x)
        f = {k: v.reshape(-1) for k, v in self.f.items()}
        out = {k: torch.zeros_like(x[0]) for k in FIELDS}
        if self.p["ilin"] == 1:
            for i in (0, 1):
                wx = 1 - (x[0] - self.dx * (i0 + i - 1).double()).abs() / self.dx
                for j in (0, 1):
                    wy = 1 - (x[1] - self.dy * (j0 + j - 1).double()).abs() / self.dy
                    c = self.col(i0 + i, j0 + j)
                    for k in (0, 1):
                        wz = 1 - (x[2] - self.zz[ku + k]).abs() / self.dzu[ku + 1]
                        ww = 1 - (x[2] - self.z[kw + k]).abs() / self.dzw[kw + 1]
                        for q in FIELDS:
                            lev, w = (kw + k, ww) if q == "w" else (ku + k, wz)
                            out[q] += f[q][lev * plane + c] * wx * wy * w
            edge, lev = (ku == 0) | (ku == nnz), torch.where(ku == 0, torch.ones_like(ku), ku)
            c = self.col(i0 + 1, j0 + 1)
            for q in ("u", "v", "T", "q"):
                out[q] = torch.where(edge, f[q][lev * plane + c], out[q])
        else:
            always = [torch.ones_like(x[0], dtype=torch.bool)] * 6
            wx = _lagrange(x[0], [self.dx * (i0 + a - 3).double() for a in range(6)], always)
            wy = _lagrange(x[1], [self.dy * (j0 + a - 3).double() for a in range(6)], always)
            lu, wu = _window(ku, x[2], self.zz, nnz, False)
            lw, ww = _window(kw, x[2], self.z, nnz, True)
            for i in range(6):
                for j in range(6):
                    c, wxy = self.col(i0 + i - 2, j0 + j - 2), wx[i] * wy[j]
                    for k in range(6):
                        a, w = lu[k] * plane + c, wxy * wu[k]
                        for q in ("u", "v", "T", "q"):
                            out[q] += f[q][a] * w
                        out["w"] += f["w"][lw[k] * plane + c] * (wxy * ww[k])
        return torch.stack([out["u"], out["v"], out["w"]]), out["T"], out["q"]

    def pressure(self, z):
        p = self.p
        return p["surf_p"] * (1 - z * p["grav"] / p["Cpa"] / p["tsfcc1"]) ** (p["Cpa"] / p["Rd"])

    def air(self, z, Tf):
        p = self.p
        if p["iexner"] == 1:
            Tf = Tf * (p["surf_p"] / self.pressure(z)) ** (-p["Rd"] / p["Cpa"])
            return Tf, self.pressure(z) / p["Rd"] / Tf
        return Tf, torch.full_like(Tf, p["surf_rho"])

    def magnus(self, T):
        return 610.94 * torch.exp(17.6257 * (T - 273.15) / (243.04 + T - 273.15))

    def guess(self, Tf, q, rhoa, m_s, kap, r, es):
        """Equilibrium radius (rad_solver2, particles.f90:4328) and where it exists."""
        p = self.p
        lg = torch.log(p["Ru"] * Tf * rhoa * q / (p["Mw"] * es))
        a = -2 * p["Mw"] * p["Gam"] / (p["Ru"] * p["rhow"] * Tf) / lg
        c = kap * m_s / (2 / 3 * p["pi2"] * p["rhos"]) / lg
        Q, R = a * a / 9, (2 * a ** 3 + 27 * c) / 54
        M = R * R - Q ** 3
        th = torch.acos((R / Q.clamp_min(0) ** 1.5).clamp(-1, 1))
        one = -2 * Q.clamp_min(0).sqrt() * torch.cos((th - p["pi2"]) / 3) - a / 3
        two = -2 * Q.clamp_min(0).sqrt() * torch.cos((th + p["pi2"]) / 3) - a / 3
        S = -torch.sign(R) * (R.abs() + M.clamp_min(0).sqrt()) ** (1 / 3)
        real = S + Q / S - a / 3
        three = torch.where(one < 0, two, one)
        g = torch.where(M < 0, three, real)
        return g, (M < 0) | (real >= 0)

    def newton(self, a, b, d):
        """Gauss-Newton (particles.f90:4071) on the residual of ie_vrt_nd with its exact derivatives."""
        p = self.p
        act = torch.ones_like(a, dtype=torch.bool)
        ok = torch.zeros_like(act)
        for _ in range(50):
            rn, Tn = a * d["R"], b * d["Tp"]
            sq = (2 * rn * d["diff"] / p["nuf"]).sqrt()
            sh, nu = 2 + 0.6 * sq * p["Sc"] ** (1 / 3), 2 + 0.6 * sq * p["Pra"] ** (1 / 3)
            k1 = 18 * d["rhoa"] * p["nuf"] / (36 * p["Sc"] * p["rhow"])
            k2 = -p["Cpa"] / p["Cpp"] * 18 * d["rhoa"] * p["nuf"] / (12 * p["Pra"] * p["rhow"])
            rp, tp = k1 * sh / rn, k2 * nu / rn ** 2
            rp_a = k1 * (0.3 * sq * p["Sc"] ** (1 / 3) - sh) / (rn * a)
            tp_a = k2 * (0.3 * sq * p["Pra"] ** (1 / 3) - 2 * nu) / (rn ** 2 * a)
            cl = 3 * p["Lv"] / p["Cpp"] / rn
            sol = d["kap"] * d["m_s"] / (p["rhos"] * (2 / 3) * p["pi2"] * rn ** 3)
            kel = 2 * p["Mw"] * p["Gam"] / (p["Ru"] * p["rhow"] * rn * Tn)
            e1 = p["Lv"] * p["Mw"] / p["Ru"]
            qs = p["Mw"] / (p["Ru"] * Tn * d["rhoa"]) * d["es"] * torch.exp(e1 * (1 / d["Tf"] - 1 / Tn) + kel - sol)
            qs_a, qs_b = qs * (-kel + 3 * sol) / a, qs * (e1 / Tn - kel - 1) / b
            R1 = rp * (d["q"] - qs) * d["t0"] / d["R"]
            R1a, R1b = (rp_a * (d["q"] - qs) - rp * qs_a) * d["t0"] / d["R"], -rp * qs_b * d["t0"] / d["R"]
            w = d["R"] / d["t0"]
            T1 = (tp * (Tn - d["Tf"]) + cl * R1 * w) * d["t0"] / d["Tp"]
            T1a = (tp_a * (Tn - d["Tf"]) + (-cl / a * R1 + cl * R1a) * w) * d["t0"] / d["Tp"]
            T1b = (tp * d["Tp"] + cl * R1b * w) * d["t0"] / d["Tp"]
            h = d["h"]
            f1, f2 = a - 1 - h * R1, b - 1 - h * T1
            J11, J21, J12, J22 = 1 - h * R1a, -h * T1a, -h * R1b, 1 - h * T1b
            det = J11 * J22 - J12 * J21
            c1, c2 = (J22 * f1 - J12 * f2) / det, (J11 * f2 - J21 * f1) / det
            relax = torch.ones_like(a)
            for _ in range(11):
                relax = torch.where((a - relax * c1 < 0) | (b - relax * c2 < 0), relax / 2, relax)
            na, nb = a - relax * c1, b - relax * c2
            bad = ~((na >= 0.01) & (nb >= 0.01))
            done = (c1 * c1 + c2 * c2).sqrt() < 1e-11
            a, b = torch.where(act & ~bad, na, a), torch.where(act & ~bad, nb, b)
            ok |= act & done & ~bad
            act = act & ~done & ~bad
            if not bool(act.any()):
                break
        return a, b, ok | act   # one that only jitters in the last digits is there

    def be(self, d, dt, it):
        p, g = self.p, self.g
        x, r, Tp, m_s, kap = d["xp"].clone(), d["radius"], d["Tp"], d["m_s"], d["kappa_s"]
        uf, Tf, q = self.interp(x)
        Tf, rhoa = self.air(x[2], Tf)
        d["vp_old"], d["Tp_old"], d["radius_old"] = d["vp"], Tp, r
        v = uf.clone() if it <= 1 else d["vp"]
        x = x + dt * v
        vol = 2 / 3 * p["pi2"] * r ** 3
        rhop = (m_s + vol * p["rhow"]) / vol
        ti = 18 * rhoa * p["nuf"] / rhop / (2 * r) ** 2
        gr = torch.tensor(p["part_grav"], device=r.device, dtype=torch.float64)[:, None]
        v = (v + ti * dt * uf + dt * gr) / (1 + dt * ti)
        t0 = (m_s / (2 / 3 * p["pi2"] * p["radius_init"] ** 3) + p["rhow"]) * (2 * p["radius_init"]) ** 2 / (18 * rhoa * p["nuf"])
        es = self.magnus(Tf)
        guess, real = self.guess(Tf, q, rhoa, m_s, kap, r, es)
        one = torch.ones_like(r)
        a, b, ok = self.newton(torch.where(real, guess / r, one), torch.where(real, Tf / Tp, one),
                               dict(R=r, Tp=Tp, Tf=Tf, q=q, m_s=m_s, kap=kap, rhoa=rhoa, t0=t0, h=dt / t0, es=es,
                                    diff=(uf - v).square().sum(0).sqrt()))
        a, b = torch.where(ok, a, one), torch.where(ok, b, Tf / Tp)
        d.update(xp=x, vp=v, uf=uf, Tf=Tf, qinf=q, Tp=b * Tp, radius=a * r)
        d["qstar"] = self.qstar(Tf, d["Tp"], d["radius"], rhoa, m_s, kap)
        return self.walls(d)

    def qstar(self, Tf, Tp, r, rhoa, m_s, kap):
        p = self.p
        return p["Mw"] / (p["Ru"] * Tp * rhoa) * self.magnus(Tf) * torch.exp(
            p["Mw"] * p["Lv"] / p["Ru"] * (1 / Tf - 1 / Tp) + 2 * p["Mw"] * p["Gam"] / (p["Ru"] * p["rhow"] * r * Tp)
            - kap * m_s / (p["rhos"] * (2 / 3) * p["pi2"] * r ** 3))

    def rk3(self, d, dt, it):
        p = self.p
        zeta, gama = (0.0, -17 / 60, -5 / 12), (8 / 15, 5 / 12, 3 / 4)
        gr = torch.tensor(p["part_grav"], device=d["radius"].device, dtype=torch.float64)[:, None]
        d["vp_old"], d["Tp_old"], d["radius_old"] = d["vp"], d["Tp"], d["radius"]
        xr, vr, sr, lr, rr = d["vp"] * 0, d["vp"] * 0, d["Tp"] * 0, d["Tp"] * 0, d["Tp"] * 0
        for s in range(3):
            x, v, r, Tp, m_s, kap = d["xp"], d["vp"], d["radius"], d["Tp"], d["m_s"], d["kappa_s"]
            uf, Tf, q = self.interp(x)
            Tf, rhoa = self.air(x[2], Tf)
            Rep = 2 * r * (v - uf).square().sum(0).sqrt() / p["nuf"]
            vol = 2 / 3 * p["pi2"] * r ** 3
            rhop = (m_s + vol * p["rhow"]) / vol
            ti = 18 * rhoa * p["nuf"] / rhop / (2 * r) ** 2
            nu, sh = 2 + 0.6 * Rep.sqrt() * p["Pra"] ** (1 / 3), 2 + 0.6 * Rep.sqrt() * p["Sc"] ** (1 / 3)
            qs = self.qstar(Tf, Tp, r, rhoa, m_s, kap)
            xt, vt, Tt, rt = x + dt * zeta[s] * xr, v + dt * zeta[s] * vr, Tp + dt * zeta[s] * (sr + lr), r + dt * zeta[s] * rr
            xr, vr = v, (1 + 0.15 * Rep ** 0.687) * ti * (uf - v) + gr
            rr = sh / 9 / p["Sc"] * rhop / p["rhow"] * r * ti * (q - qs)
            sr = -nu / 3 / p["Pra"] * p["Cpa"] / p["Cpp"] * rhop / p["rhow"] * ti * (Tp - Tf)
            lr = 3 * p["Lv"] / p["Cpp"] / r * rr
            c = dt * gama[s]
            d.update(xp=xt + c * xr, vp=vt + c * vr, Tp=Tt + c * (sr + lr), radius=rt + c * rr, uf=uf, Tf=Tf, qinf=q, qstar=qs)
            # no droplet may leave between the stages: the stage's own slopes travel with the list
            d.update(xr=xr, vr=vr, sr=sr, lr=lr, rr=rr)
            d = self.walls(d)
            xr, vr, sr, lr, rr = (d[k] for k in ("xr", "vr", "sr", "lr", "rr"))
        return d

    def walls(self, d):
        p, g = self.p, self.g
        x, v, r = d["xp"].clone(), d["vp"].clone(), d["radius"]
        top = (g["z"][g["nnz"] - 1] if p["icase"] == 4 else g["z"][g["nnz"]]) - r
        up, low = x[2] > top, x[2] < r
        x[2] = torch.where(up, 2 * top - x[2], x[2])
        v[2] = torch.where(up, -v[2], v[2])
        if p["icase"] == 0:
            x[2] = torch.where(low, 2 * r - x[2], x[2])
            v[2] = torch.where(low, -v[2], v[2])
        for a, length in ((0, g["xl"]), (1, g["yl"])):
            x[a] = torch.where(x[a] > length, x[a] - length, torch.where(x[a] < 0, x[a] + length, x[a]))
        d["xp"], d["vp"] = x, v
        if p["icase"] != 0 and bool(low.any()):
            d = {k: t[..., ~low].contiguous() for k, t in d.items()}
        return d

    def sources(self, d, dt):
        """(6, nnx, nny, nnz+2): particle_coupling_update, particles.f90:1151."""
        p, g = self.p, self.g
        nx, ny, nz2 = g["nnx"], g["nny"], g["nnz"] + 2
        x, v, r, Tp, Tf, m_s = d["xp"], d["vp"], d["radius"], d["Tp"], d["Tf"], d["m_s"]
        rhoa = self.pressure(x[2]) / p["Rd"] / Tf if p["iexner"] == 1 else torch.full_like(r, p["surf_rho"])
        rate = (r - d["radius_old"]) / dt
        lat = 3 * p["Lv"] / p["Cpp"] / r * rate
        sens = (Tp - d["Tp_old"]) / dt - lat
        vol = 2 / 3 * p["pi2"] * r ** 3
        rhop = (m_s + vol * p["rhow"]) / vol
        ti = 18 * rhoa * p["nuf"] / rhop / (2 * r) ** 2
        H0 = p["rhow"] / rhoa * p["pi2"] * 2 * r ** 2 * rate
        gr = torch.tensor(p["part_grav"], device=r.device, dtype=torch.float64)[:, None]
        mom = rhop * vol / rhoa * ((v - d["vp_old"]) / dt - gr) + H0 * v
        heat = sens * 6 * p["rhow"] / rhop * p["Cpp"] / p["Cpa"] / ti * (p["pi2"] / 2) * r * p["nuf"]
        vals = -torch.stack([mom[0], mom[1], mom[2], heat, H0, H0 * p["Cpv"] / p["Cpa"] * (Tp - Tf)])
        i0, j0, k0, _ = self.base(x)
        dz = self.dzu[k0 + 1]
        vals = vals * d["mult"].double() / (self.dx * self.dy * dz)
        out = torch.zeros(6, nx * ny * nz2, device=r.device, dtype=torch.float64)
        for i in (0, 1):
            wx = 1 - (x[0] - self.dx * (i0 + i - 1).double()).abs() / self.dx
            for j in (0, 1):
                wy = 1 - (x[1] - self.dy * (j0 + j - 1).double()).abs() / self.dy
                for k in (0, 1):
                    w = wx * wy * (1 - (x[2] - self.zz[k0 + k]).abs() / dz)
                    out.index_add_(1, ((i0 + i - 1) % nx * ny + (j0 + j - 1) % ny) * nz2 + k0 + k, vals * w)
        return out.view(6, nx, ny, nz2)


def _advance(case, p, box, dt, it):
    E = _Exact(box["grid"], p, box["flow"])
    parts, src, m = [], 0.0, 1 << 22
    n = int(box["droplets"]["radius"].shape[0])
    for at in range(0, n, m):       # droplets do not see one another: a chunk runs all its steps
        d = {k: t[..., at:at + m].contiguous() for k, t in box["droplets"].items()}
        for s in range(case["steps"]):
            d = E.rk3(d, dt, it + s) if case["kind"] == "rk3" else E.be(d, dt, it + s)
        src = src + E.sources(d, dt)
        parts.append({k: d[k] for k in STATE})
    return {k: torch.cat([q[k] for q in parts], dim=-1) for k in STATE}, src


def exact(case, seed):
    p, dt = _params(case), _dt(case)
    boxes = _boxes(case, seed)
    if case["kind"] == "batch":
        res = [_advance(case, p, b, dt, 2) for b in boxes]
        return dict(droplets={k: torch.cat([d[k].reshape(-1) for d, _ in res]) for k in ("xp", "vp", "Tp", "radius")},
                    sources=torch.cat([s.reshape(-1) for _, s in res]), numpart=None)
    d, src = _advance(case, p, boxes[0], dt, 2)
    # whole numbers have no 64-bit value; the statistics are sums of the state above
    out = dict(droplets=dict(d, lid=None), sources=[src[q] for q in range(6)], counters=None)
    if case["stats"]:
        out["stats"] = None
    return out
