"""Performance cases: the work a user of the framework has it do, through its public entry
points, with what each pass returns and how exact that is.

A pass is a run of time steps (`Simulation.run`, `Ensemble.run`, `LocalSlabs.run`) and the
read-out that a program makes after it: the eight on-fault output planes and, after several steps,
the split-node state and the wavefield (a checkpoint).  A state is a simulation that goes on from pass to
pass, as a job does.  Cases of kind "waves" have no fault: they start from a seeded
wavefield that fills the domain, and `exact` integrates them in 64 bits.
"""
import math
import random

import numpy as np
import torch

import dynfd3dcuda_b200 as dfd
from dynfd3dcuda_b200.decomp import LocalSlabs

# one-sided 5-point operator and the 3-point one below the free surface
C5 = (0.29164704779069994, 0.6667451421652, 1.2501177132452999, 0.33341180882999999, 0.0416862855406)
C3 = (7.0 / 6.0, 4.0 / 3.0, 1.0 / 6.0)
FLAGS = ((-1, -1, -1), (1, 1, -1), (1, 1, 1), (-1, -1, 1), (-1, 1, -1), (1, -1, -1), (1, -1, 1), (-1, 1, 1))
CHECKPOINT = 40  # steps between two reads of the whole wavefield, which take about 10 % of a pass


def grid(kind, nx, ny, nz, steps, **opt):
    """A case: grid nx (fault normal) x ny (strike) x nz (depth), steps per pass, options."""
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=steps, dh=100.0, law="sw", shape="flat", pml=12, sponge=0,
             layered=False, refine=False, surface=True, tp_n=0, parts=1)
    c.update(opt)
    return c


def listed():
    return [
        # one step of a small job with its per-step outputs: the latency of a step (test and
        # set-up runs, coupled codes that look at the fault after every step)
        dict(grid("rupture", 24, 76, 40, 1, pml=6, refine=True), name="step_small"),
        # the plain Cartesian slip-weakening job (TPV3 class)
        dict(grid("rupture", 100, 200, 100, CHECKPOINT), name="cartesian_sw"),
        # the curved-grid job: 60 degree dip, hills on the free surface, refined x grid
        dict(grid("rupture", 300, 400, 200, CHECKPOINT, shape="dip", refine=True), name="curved_sw"),
        # the large single domain: 1-D layered medium, curved fault, PML 20 with a sponge
        dict(grid("rupture", 600, 1000, 300, 30, dh=50.0, shape="bumps", pml=20, sponge=20, layered=True,
                  refine=True), name="large_sw"),
        # rate and state (slip law) on a rough fault, the grid of the learned-guess study
        dict(grid("rupture", 200, 300, 150, CHECKPOINT, law="slip", shape="rough"), name="rough_rs"),
        # thermal pressurisation with columns of 64 points
        dict(grid("rupture", 120, 201, 143, CHECKPOINT, law="tp", tp_n=64), name="thermal_rs"),
        # eight scenarios of mixed size and friction law stepped together
        dict(grid("ensemble", 100, 200, 150, 20, parts=8), name="ensemble"),
        # a domain in two slabs with the halo exchange between stages (stage by stage)
        dict(grid("slabs", 120, 256, 121, 10, parts=2), name="two_slabs"),
        # wave propagation without a fault: odd sizes, curved grid, PML, free surface
        dict(grid("waves", 131, 203, 117, 16, shape="dip", pml=13, refine=True), name="waves_curved"),
        # the same without a free surface, in a layered medium with a sponge beside the PML
        dict(grid("waves", 96, 150, 98, 16, pml=10, sponge=10, layered=True, surface=False), name="waves_layered"),
    ]


def draw(rng):
    """One more case of the same ranges: grids of 24 to 1000 nodes an axis, every friction
    law, shape and option, PML 5 to 24, one domain, ensembles and slabs."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rupture"] * 5 + ["ensemble", "slabs"] + ["waves"] * 2)
    shape = rng.choice(["flat", "dip", "rough", "bumps"])
    opt = dict(shape=shape, pml=rng.randint(5, 24), refine=rng.random() < 0.5, layered=rng.random() < 0.3,
               surface=kind != "waves" or rng.random() < 0.7)
    if rng.random() < 0.3:
        opt["sponge"] = rng.randint(5, 20)
    if kind == "waves":
        opt["pml"] = min(opt["pml"], 16)
        return grid(kind, size(40, 160), size(40, 240), size(40, 140), 8, **opt)
    opt["law"] = rng.choice(["sw", "sw", "aging", "slip", "tp"])
    if opt["law"] == "tp":
        opt["tp_n"] = rng.choice([20, 33, 64, 100])
    if kind == "ensemble":
        return grid(kind, size(60, 110), size(110, 220), size(80, 160), 10, parts=rng.randint(2, 8),
                    **dict(opt, pml=min(opt["pml"], 16), law="sw", tp_n=0))
    if kind == "slabs":
        parts = rng.choice([2, 3, 4])
        return grid(kind, size(50, 130), parts * size(40, 80), size(50, 130), 4, parts=parts, **opt)
    nx, ny, nz = size(50, 600), size(80, 1000), size(50, 300)
    nodes = nx * ny * nz
    return grid(kind, nx, ny, nz, 1 if rng.random() < 0.3 else 20 if nodes < 5e7 else 10, **opt)


# ---------------------------------------------------------------- inputs of a job

def smooth_field(shape, seed, cell=12):
    """Seeded smooth field of unit size on a (NZ, NY) plane: random values on a coarse mesh,
    interpolated."""
    g = torch.Generator().manual_seed(int(seed))
    coarse = torch.randn((1, 1, shape[0] // cell + 3, shape[1] // cell + 3), generator=g, dtype=torch.float64)
    return torch.nn.functional.interpolate(coarse, size=tuple(shape), mode="bicubic", align_corners=True)[0, 0].numpy()


def fault_surface(c, seed):
    """x, y, z (NZ, NY) of the fault surface, the Fault_geometry planes."""
    ny, nz, dh = c["ny"], c["nz"], c["dh"]
    j = np.arange(ny)[None, :] + np.zeros((nz, 1))
    k = np.arange(nz)[:, None] + np.zeros((1, ny))
    x, y, z = 0.0 * j, (j - ny / 2) * dh, (k + 1 - nz) * dh
    rng = np.random.default_rng([int(seed), 1])
    if c["shape"] == "dip":
        top = 0.0 * j
        for _ in range(2):
            amp, at = 0.025 * nz * dh * rng.uniform(0.5, 1.0), rng.uniform(-0.3, 0.3) * ny * dh
            top = top + amp * np.exp(-(y - at) ** 2 / (0.125 * max(ny, 2 * nz) * dh) ** 2)
        z = z + k / (nz - 1) * top
        x = np.maximum(-z, 0.0) / math.tan(math.radians(60.0))
    elif c["shape"] == "rough":
        x = 0.15 * dh * smooth_field((nz, ny), seed + 2, 10)
    elif c["shape"] == "bumps":
        x = 4.0 * dh * np.sin(2 * np.pi * j / 1000 * rng.uniform(1.0, 3.0))
    return np.stack([x, y, z]).astype(np.float32)


def fault_planes(c, fx, seed):
    """The Fault_init_stress planes: a stressed fault with a nucleation patch, seeded
    heterogeneity of the shear stress and of the friction parameter a."""
    ny, nz, dh = c["ny"], c["nz"], c["dh"]
    x, y, z = [v.astype(np.float64) for v in fx]
    ty = np.stack([np.gradient(v, axis=1) for v in (x, y, z)])
    tz = np.stack([np.gradient(v, axis=0) for v in (x, y, z)])
    n = np.cross(ty, tz, axis=0)
    n /= np.linalg.norm(n, axis=0, keepdims=True)
    n *= np.sign(n[0:1])
    s = ty / np.linalg.norm(ty, axis=0, keepdims=True)
    depth, radius = min(7.5e3, 0.4 * (nz - 31) * dh), max(5 * dh, min(1.5e3, 0.15 * (ny - 60) * dh))
    r = np.hypot(y, z + depth)
    het = 1.0 + 0.01 * smooth_field((nz, ny), seed + 3)
    out = np.zeros((15, nz, ny))
    tn = -120e6
    if c["law"] == "sw":
        ts = np.where(r < radius, -82.5e6, -70e6) * het
        out[6], out[7], out[8], out[9] = 0.677, 0.525, 0.4, 0.0
    else:
        ts = -40e6 * het
        rng = np.random.default_rng([int(seed), 4])
        a = np.exp(rng.uniform(math.log(0.01), math.log(0.02), (nz, ny)))
        out[10], out[11], out[12], out[13] = a, 0.014, 0.2, 0.1
        out[14] = a * np.log(2e-6 / 1e-16 * np.sinh(np.abs(ts) / 120e6 / a))
        bump = np.where(r < radius, np.exp(np.minimum(r ** 2 / np.minimum(r ** 2 - radius ** 2, -1e-30), 0.0)), 0.0)
        out[3:6] = -45e6 * bump * s
    out[0:3] = tn * n + ts * s
    return out.astype(np.float32)


def layers_of(c):
    """Media1D rows (depth, rho, vp, vs): vs 2000 to 3600 m/s over depth."""
    if not c["layered"]:
        return None
    vs = np.linspace(2000.0, 3600.0, 16)
    depth = np.linspace(0.0, (c["nz"] - 1) * c["dh"], 16) + 0.37 * c["dh"]
    depth[0] = -1e4
    return np.stack([depth, 2670.0 + 0 * vs, math.sqrt(3.0) * vs, vs], 1).astype(np.float32)


def job_of(c):
    """The job dictionary (params.json keys)."""
    nx, ny, nz, dh = c["nx"], c["ny"], c["nz"], c["dh"]
    # below the stability limit 1.3 hmin / vpmax of the case's grid
    dt = (8e-5 if c["shape"] == "flat" or dh < 100 else 6e-5) * dh
    p = dict(NX=nx, NY=ny, NZ=nz, DH=dh, DT=dt, TMAX=1e4 * dt, PML_N=c["pml"], PML_velocity=6236.0, PML_bmax=2.5,
             PML_fc=1.6, INPORT_GRID_TYPE=1, INPORT_STRESS_TYPE=1, FreeSurface=int(c["surface"]),
             NormalRefine=int(c["refine"]))
    if c["sponge"]:
        p.update(useCerjan=1, DAMP_N=c["sponge"])
    if c["kind"] == "waves":
        p["Rupture"] = 0
    elif c["law"] == "sw":
        p.update(Friction_type=0, mu_s=0.677, mu_d=0.525, Dc=0.4, C0=0.0)
    else:
        p.update(Friction_type={"aging": 1, "slip": 2, "tp": 3}[c["law"]], RS_V0=1e-6, RS_f0=0.6, RS_fw=0.2,
                 RS_Vini=1e-16, RS_L=0.2, smooth_load_T=0.1)
        if c["law"] == "tp":
            p["TP_n"] = c["tp_n"]
    if c["kind"] != "waves":
        p["Fault_grid"] = [31, ny - 30, 31, nz]
    return p


def inputs_of(c, seed):
    """(job, fault geometry, fault initial state or None, layers or None) of a case."""
    fx = fault_surface(c, seed)
    st = None
    if c["kind"] != "waves":
        st = fault_planes(c, fx, seed)
        if c["law"] == "tp":
            rng = np.random.default_rng([int(seed), 5])
            hy = np.exp(rng.uniform(math.log(2e-5), math.log(4e-4), st.shape[1:]))
            st = np.concatenate([st, hy[None].astype(np.float32)])
    return job_of(c), fx, st, layers_of(c)


def start_wave(c, seed):
    """Seeded wavefield that fills the domain, (9, nx, nz, ny) float32 with zero ghosts:
    smooth over about six nodes, velocities of 0.1 m/s and stresses of 1 MPa."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    shape = (c["nx"], c["nz"], c["ny"])
    g = torch.Generator().manual_seed(int(seed) + 6)
    coarse = torch.randn((1, 9) + tuple(n // 6 + 3 for n in shape), generator=g, dtype=torch.float32).to(dev)
    w = torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True)[0]
    w[:3] *= 0.1
    w[3:] *= 1e6
    return torch.nn.functional.pad(w, (3,) * 6).cpu().numpy()


def scenario(c, i):
    """Scenario i of an ensemble: sizes within a third of the case's, slip weakening and
    rate and state in turn."""
    rng = random.Random("%d %d %d %d" % (c["nx"], c["ny"], c["nz"], i))
    # the united border takes 30 nodes at each end along strike and below
    nx, ny, nz = (max(lo, int(c[n] * rng.uniform(0.67, 1.33))) for n, lo in (("nx", 50), ("ny", 80), ("nz", 50)))
    return dict(c, kind="rupture", parts=1, nx=nx, ny=ny, nz=nz, law="sw" if i % 2 == 0 else "slip")


# ---------------------------------------------------------------- the measured path

def prepare(case, seed):
    c = grid(**{k: v for k, v in case.items() if k != "name"})
    state = dict(case=c, it=0)
    if c["kind"] == "ensemble":
        sims = []
        for i in range(c["parts"]):
            s = scenario(c, i)
            sims.append(dfd.Simulation(*inputs_of(s, seed + 100 * i)))
        state.update(sims=sims, run=dfd.Ensemble(sims))
    elif c["kind"] == "slabs":
        slabs = LocalSlabs(*inputs_of(c, seed), c["parts"])
        state.update(sims=slabs.sims, run=slabs)
    else:
        sim = dfd.Simulation(*inputs_of(c, seed))
        if c["kind"] == "waves":
            sim.set_wave(start_wave(c, seed))
        state.update(sims=[sim], run=sim)
    if c["kind"] != "waves":
        state["planes"] = [torch.empty((8, s.NZ, s.NY), dtype=torch.float32, pin_memory=True) for s in state["sims"]]
    if c["steps"] > 1:
        state["waves"] = [torch.empty((9, s.nx, s.nz, s.ny), dtype=torch.float32, pin_memory=True) for s in state["sims"]]
    return state


def run(state):
    c, sims = state["case"], state["sims"]
    state["run"].run(state["it"], c["steps"])
    state["it"] += c["steps"]
    out = {}
    if c["kind"] == "ensemble":
        state["run"].synchronize()  # the ensemble has a stream of its own
    if c["kind"] != "waves":
        for i, (s, p) in enumerate(zip(sims, state["planes"])):
            s.fetch_outputs(p.data_ptr())
            out["fault%d" % i] = dict(slip_rate=p[0:2], traction=p[2:5], slip=p[5], state=p[6], time=p[7])
    for i, (s, w) in enumerate(zip(sims, state.get("waves", ()))):
        s._check(dfd.lib().dfd_get_wave(s.h, w.data_ptr()))
        out["wave%d" % i] = dict(velocity=w[:3], stress=w[3:])
    if c["kind"] == "rupture" and c["steps"] > 1:
        split = sims[0].fault("split")
        out["split"] = dict(velocity=split[:3], traction=split[3:])
    if c["law"] == "tp" and c["kind"] == "rupture":
        out["TP"] = [sims[0].fault("TP_T"), sims[0].fault("TP_P")]
    return out


def work(case):
    """Per step and node the nine fields are read and written once (72 bytes; the metric of
    the separable grid is a few planes), the ADE state likewise for each PML face a node
    lies in; four stages of 27 five-point derivatives (9 operations each), about 90
    operations of Hooke's and Newton's laws and 18 of the Runge-Kutta sums."""
    c = grid(**{k: v for k, v in case.items() if k != "name"})
    nodes = face = 0
    for s in [scenario(c, i) for i in range(c["parts"])] if c["kind"] == "ensemble" else [c]:
        nx, ny, nz = s["nx"], s["ny"], s["nz"]
        nodes += nx * ny * nz
        face += s["pml"] * (2 * ny * nz + 2 * nx * nz + (1 if s["surface"] else 2) * nx * ny)
    return {"bytes": 72.0 * (nodes + face) * c["steps"], "flops": 4.0 * (27 * 9 + 90 + 18) * nodes * c["steps"]}


def tolerance(case):
    # four to ten times what the plain kernels (other sums, through global memory) and the
    # tiled ones show against each other after a pass: without a fault 2e-7 (largest value
    # 2e-6), with slip weakening 9e-7 (1e-4, ahead of the rupture front, where the field is
    # small), with rate and state 2e-5 (2e-3, its slip rates depend exponentially on stress)
    if case["kind"] == "waves":
        return {"rel": 1e-6, "max": 1e-5}
    if case.get("law", "sw") == "sw" and case["kind"] != "ensemble":
        return {"rel": 1e-5, "max": 2e-3}
    return {"rel": 1e-4, "max": 1e-2}


# ---------------------------------------------------------------- the same in 64 bits

def x_line(c):
    """x of the nx + 6 nodes of the line, refined to half the spacing around the fault."""
    nx, dh = c["nx"] + 6, c["dh"]
    x = np.zeros(nx)
    if c["refine"]:
        ic = c["nx"] // 2 + 3
        for sign in (1, -1):
            i = ic + sign
            while 0 <= i < nx:
                d = abs(i - ic)
                t = 0.0 if d < 10 else 1.0 - math.cos(math.pi * (d - 10) / 45.0) if d < 55 else 2.0
                x[i] = x[i - sign] + sign * dh * (0.5 + 0.25 * t)
                i += sign
    else:
        x = (np.arange(nx) - 3 - c["nx"] // 2) * dh
    for n in range(1, 4):
        x[3 - n] = 2 * x[3] - x[3 + n]
        x[nx - 4 + n] = 2 * x[nx - 4] - x[nx - 4 - n]
    return x


def extend(a):
    """A (NZ, NY) plane with three ghost rows and columns, extrapolated linearly."""
    for axis in (1, 0):
        a = np.moveaxis(a, axis, 0)
        lo = [2 * a[0] - a[n] for n in (3, 2, 1)]
        hi = [2 * a[-1] - a[-1 - n] for n in (1, 2, 3)]
        a = np.moveaxis(np.concatenate([np.stack(lo), a, np.stack(hi)]), 0, axis)
    return a


def pml_profiles(c, n, lo, hi):
    """alpha, beta, d of the absorbing layer along an axis of n nodes."""
    p = job_of(c)
    N, dh = c["pml"], c["dh"]
    x = np.full(n, -1.0)
    if lo:
        x[:N] = (N - 1 - np.arange(N)) * dh
    if hi:
        x[n - N:] = np.arange(N) * dh
    L = dh * (N - 1)
    r = 10.0 ** -((math.log10(N) - 1.0) / math.log10(2.0) + 3.0)
    dmax = -p["PML_velocity"] / (2 * L) * math.log(r) * 3.0
    u = np.where(x >= 0, x / L, 0.0)
    alpha = np.where(x >= 0, math.pi * p["PML_fc"] * (1 - u), 0.0)
    return alpha, 1.0 + np.where(x >= 0, (p["PML_bmax"] - 1) * u * u, 0.0), dmax * u * u


def exact(case, seed):
    """The wavefield of a "waves" case after its steps, in 64 bits; None for the others
    (the split-node friction solve has no closed form to restate in a few lines; the FP64
    oracle of the tests covers it)."""
    c = grid(**{k: v for k, v in case.items() if k != "name"})
    if c["kind"] != "waves":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.float64)  # noqa: E731
    p = job_of(c)
    nx, ny, nz, N = c["nx"], c["ny"], c["nz"], c["pml"]
    dh, dt, free = c["dh"], float(np.float32(p["DT"])), c["surface"]
    box = (nx, nz, ny)
    # metric: central differences of the grid (x(i) + fx, fy, fz), media by depth
    xl, (fx, fy, fz) = x_line(c), [extend(a.astype(np.float64)) for a in fault_surface(c, seed)]
    a = T(0.5 / dh * (xl[4:nx + 4] - xl[2:nx + 2]))[:, None, None]
    y3 = [T(0.5 / dh * (f[3:-3, 4:-2] - f[3:-3, 2:-4]))[None] for f in (fx, fy, fz)]
    z3 = [T(0.5 / dh * (f[4:-2, 3:-3] - f[2:-4, 3:-3]))[None] for f in (fx, fy, fz)]
    det = y3[1] * z3[2] - y3[2] * z3[1]
    zero = torch.zeros_like(det)
    xi = (1.0 / a + 0 * det, (y3[2] * z3[0] - y3[0] * z3[2]) / det / a, (y3[0] * z3[1] - y3[1] * z3[0]) / det / a)
    et, zt = (zero, z3[2] / det, -z3[1] / det), (zero, -y3[2] / det, y3[1] / det)
    jac = a * det
    lay = layers_of(c)
    if lay is not None:
        depth = -fz[3:-3, 3:-3]
        at = np.full(depth.shape, len(lay) - 1)
        for i, row in enumerate(lay.astype(np.float64)):
            at = np.where(depth > row[0], i, at)
        rho, vp, vs = (T(lay.astype(np.float64)[at, m])[None] for m in (1, 2, 3))
    else:
        rho, vp, vs = (zero + v for v in (2670.0, 6000.0, 3464.0))
    mu, lam = rho * vs ** 2, rho * (vp ** 2 - 2 * vs ** 2)
    l2m = lam + 2 * mu

    def terms(d, e):
        """Velocity and stress rates of one axis from the derivatives d and metric row e."""
        div = d[0] * e[0] + d[1] * e[1] + d[2] * e[2]
        return torch.stack([(d[3] * e[0] + d[6] * e[1] + d[7] * e[2]) / rho,
                            (d[6] * e[0] + d[4] * e[1] + d[8] * e[2]) / rho,
                            (d[7] * e[0] + d[8] * e[1] + d[5] * e[2]) / rho,
                            lam * div + 2 * mu * d[0] * e[0], lam * div + 2 * mu * d[1] * e[1],
                            lam * div + 2 * mu * d[2] * e[2], mu * (d[0] * e[1] + d[1] * e[0]),
                            mu * (d[0] * e[2] + d[2] * e[0]), mu * (d[1] * e[2] + d[2] * e[1])])

    def part(u, dim, off, n):
        """Field(s) u with three ghosts, shifted by off along dim, n nodes from the first."""
        sel = [Ellipsis] + [slice(3, s - 3) for s in u.shape[-3:]]
        sel[1 + dim] = slice(3 + off, 3 + off + n)
        return u[tuple(sel)]

    def diff(u, dim, sign):
        n = box[dim]
        s = [part(u, dim, sign * m, n) for m in (-1, 0, 1, 2, 3)]
        return sign * (-C5[0] * s[0] - C5[1] * s[1] + C5[2] * s[2] - C5[3] * s[3] + C5[4] * s[4]) / dh

    def along(v, dim):
        return T(v).reshape([-1 if m == dim else 1 for m in range(3)])

    # the axes in memory order: x, z, y
    alpha, beta, damp_d = {}, {}, {}
    for dim, n, lo, hi in ((0, nx, True, True), (2, ny, True, True), (1, nz, True, not free)):
        alpha[dim], beta[dim], damp_d[dim] = (along(v, dim) for v in pml_profiles(c, n, lo, hi))
    rows = {0: xi, 2: et, 1: zt}
    damp = 1.0
    if c["sponge"]:
        al, nd = math.sqrt(-math.log(0.92)) / c["sponge"], c["sponge"]
        edge = np.exp(-(al * (nd - np.arange(nd))) ** 2)
        f = []
        for dim, n in ((0, nx), (1, nz), (2, ny)):
            v = np.ones(n)
            v[:nd] = edge
            if not (dim == 1 and free):
                v[n - nd:] = edge[::-1]
            f.append(along(v, dim))
        damp = torch.minimum(torch.minimum(f[0], f[1]), f[2])
    if free:
        # dV/dz on the surface row from dV/dx and dV/dy (no traction there)
        top = lambda e: [(v + 0 * jac)[:, -1, :] for v in e]  # noqa: E731
        tx, ty, tz = top(xi), top(et), top(zt)
        tl, tm = (lam + 0 * jac)[:, -1, :], (mu + 0 * jac)[:, -1, :]

        def outer(e, f, s):
            dot = sum(u * v for u, v in zip(e, f))
            m = [[s * (tl * e[r] * f[q] + tm * e[q] * f[r] + (tm * dot if r == q else 0)) for q in range(3)]
                 for r in range(3)]
            return torch.stack([torch.stack(r, -1) for r in m], -2)

        inv = torch.linalg.inv(outer(tz, tz, 1.0))
        from_x = inv @ outer(tz, tx, -1.0 / beta[0][:, 0, :])
        from_y = inv @ outer(tz, ty, -1.0 / beta[2][:, 0, :])
        full = [e + 0 * jac for e in xi], [e + 0 * jac for e in et], [e + 0 * jac for e in zt]

    def apply(m, d):
        return torch.einsum("xyrq,qxy->rxy", m, d[:3, :, -1, :])

    def surface_rows(w, h, sign):
        """The momentum equation of the three top rows from the traction image."""
        s = w[3:, 3:-3, 3:-3, 3:-3]
        s = ((s[0], s[3], s[4]), (s[3], s[1], s[5]), (s[4], s[5], s[2]))
        total = 0.0
        for dim, e in zip((0, 2, 1), full):
            t = torch.stack([jac * sum(e[q] * s[r][q] for q in range(3)) for r in range(3)])
            if dim == 1:
                t[:, :, -1] = 0.0
                t = torch.cat([t, -t[:, :, -4:-1].flip(2)], 2)
                t = torch.nn.functional.pad(t, (3, 3, 3, 0, 3, 3))
            else:
                t = torch.nn.functional.pad(t, (3,) * 6)
            total = total + (diff(t, dim, sign[dim]) / beta[dim])[:, :, -3:]
        h[:3, :, -3:] = total / (rho + 0 * jac)[:, -3:] / jac[:, -3:]

    def rates(w, ade, sign):
        h, ade_h = 0.0, {}
        D = {dim: diff(w, dim, sign[dim]) for dim in (0, 2, 1)}
        rate = {dim: terms(D[dim], rows[dim]) for dim in (0, 2, 1)}
        zrate = rate[1]
        if free:
            V = D[1].clone()
            u = w[:3]
            V[:3, :, -1] = apply(from_x, D[0]) + apply(from_y, D[2])
            at = lambda k: u[:, 3:-3, 3 + k, 3:-3]  # noqa: E731
            k2, k3 = nz - 2, nz - 3
            if sign[1] > 0:
                V[:3, :, k2] = (at(k2 + 1) - at(k2)) / dh
                V[:3, :, k3] = (-C3[0] * at(k3) + C3[1] * at(k3 + 1) - C3[2] * at(k3 + 2)) / dh
            else:
                V[:3, :, k2] = (at(k2) - at(k2 - 1)) / dh
                V[:3, :, k3] = (C3[2] * at(k3 - 2) - C3[1] * at(k3 - 1) + C3[0] * at(k3)) / dh
            zrate = torch.cat([rate[1][:3], terms(V, zt)[3:]])
        h = rate[0] / beta[0] + rate[2] / beta[2] + zrate / beta[1]
        if free:
            surface_rows(w, h, sign)
        for dim in (0, 2, 1):
            h = h - ade[dim] / beta[dim]
            g = -(alpha[dim] + damp_d[dim] / beta[dim]) * ade[dim] + damp_d[dim] / beta[dim] * rate[dim]
            if free and dim != 1:
                V = torch.zeros_like(rate[dim])
                V[:3, :, -1] = apply(from_x if dim == 0 else from_y, D[dim])
                g[3:] += damp_d[dim] * terms(V, zt)[3:]
            ade_h[dim] = g
        return h, ade_h

    w = T(start_wave(c, seed))
    ade = {dim: torch.zeros((9,) + box, dtype=torch.float64, device=dev) for dim in (0, 1, 2)}
    inner = (slice(None),) + (slice(3, -3),) * 3
    for it in range(c["steps"]):
        w0, ade0 = w[inner].clone(), {d: v.clone() for d, v in ade.items()}
        sum_w, sum_ade = w0.clone(), {d: v.clone() for d, v in ade.items()}
        for irk, (ra, rb) in enumerate(((0.5, 1 / 6), (0.5, 1 / 3), (1.0, 1 / 3), (0.0, 1 / 6))):
            s = [v * (-1 if irk % 2 else 1) for v in FLAGS[it % 8]]
            h, g = rates(w, ade, {0: s[0], 2: s[1], 1: s[2]})
            sum_w += rb * dt * h
            w = w.clone()
            w[inner] = (sum_w if irk == 3 else w0 + ra * dt * h) * damp
            for d in ade:
                sum_ade[d] += rb * dt * g[d]
                ade[d] = sum_ade[d].clone() if irk == 3 else ade0[d] + ra * dt * g[d]
    w = w.cpu()
    return {"wave0": {"velocity": w[:3], "stress": w[3:]}}
