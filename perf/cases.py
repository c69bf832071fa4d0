"""Performance cases of the forward dynamic-rupture step.

Each case is one call sequence that a program using the solver makes: advance
a problem some steps and read back what it needs.  The sizes are those of the
tests, the benchmark workloads and the ensemble generator; ``draw`` gives
further ones over the same ranges (36x56x32 to 300x600x240 points, odd sizes
included).

A case's keys: the grid (ni fault-normal, nj along strike, nk up), ``faults``
(0, 1 or 2 planes), ``method`` (dynamic_method), ``free`` (free surface),
``boundary`` and ``layers`` (CFS-PML, exponential sponge or none), ``topo``
(hills on an imported curvilinear grid, else the extruded fault-plane grid),
``dip`` (degrees; 0 = vertical), ``margin`` (welded margin), ``steps`` per
pass, ``members`` (ensemble size, 1 = a single solver) and ``call``:

* ``run``       Solver.run, then fault fields, stations and surface peaks
* ``noalloc``   the same through Solver.run_noalloc
* ``records``   Solver.run_fault_output: fault fields every ``every`` steps
* ``snapshot``  Solver.run, then all nine wavefield components
* ``ensemble``  Ensemble.run, then every member's fault fields
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-cgfd3d-dynamic_b200"))
from cgfd import (FAULT_FIELDS, GRID_FAULT_PLANE, GRID_IMPORT, WAVE_COMPONENTS, Ensemble, Problem,  # noqa: E402
                  Setup, Solver)
from inputs import von_karman  # noqa: E402

MPA = 1.0e6
VP, VS, RHO = 6000.0, 3464.0, 2670.0
SHARED = 3_000_000      # points from which one prepared problem serves all seeds
DEFAULTS = dict(faults=1, method=2, free=True, boundary="pml", layers=10, topo=False, dip=0.0, margin=20,
                call="run", every=1, members=1, sizes=0)


def listed():
    def case(name, ni, nj, nk, steps, **kw):
        return {"name": name, "ni": ni, "nj": nj, "nk": nk, "steps": steps, **{**DEFAULTS, **kw}}
    return [
        # the smallest problem (tests, smoke check): launches and latency
        case("tiny_36x56x32", 36, 56, 32, 16, layers=5, margin=10),
        # two faults, continuity matrices, direct launches without allocation
        case("two_faults_noalloc_44x64x32", 44, 64, 32, 16, faults=2, method=1, layers=5, margin=8, call="noalloc"),
        # plain wave propagation in a small ragged hilly box, whole wavefield read back
        case("waves_snapshot_61x75x53", 61, 75, 53, 12, faults=0, topo=True, layers=8, call="snapshot"),
        # a rupture whose whole wavefield is read back, as for a snapshot file
        case("planar_snapshot_60x120x64", 60, 120, 64, 24, call="snapshot"),
        # the tpv-like half space of the examples: planar vertical fault, flat surface
        case("planar_100x160x80", 100, 160, 80, 40, margin=40),
        # odd sizes, buried fault (PML on all faces), continuity matrices, records while stepping
        case("buried_records_101x163x77", 101, 163, 77, 40, method=1, free=False, topo=True, margin=22,
             call="records", every=10),
        # exponential sponge instead of PML
        case("sponge_120x180x90", 120, 180, 90, 30, boundary="sponge", margin=30),
        # a batch of uneven scenarios advanced together
        case("ensemble_6", 160, 256, 128, 12, members=6, sizes=1003, margin=10, call="ensemble"),
        # ordinary production size: hills, layers, fault record every step (the reference's io_time_skip = 1)
        case("hills_records_200x300x160", 200, 300, 160, 16, topo=True, layers=20, margin=20, call="records"),
        # dipping fault in a sheared grid
        case("dipping_240x400x133", 240, 400, 133, 12, topo=True, dip=60.0, layers=20, margin=30),
        # the benchmark workload
        case("hills_300x600x240", 300, 600, 240, 16, topo=True, layers=20, margin=40),
    ]


def draw(rng):
    """One more case: points spread over the logarithm of 64 thousand to 36 million."""
    pts = math.exp(rng.uniform(math.log(64e3), math.log(36e6)))
    scale = (pts / (100 * 160 * 80)) ** (1.0 / 3.0)
    ni, nj, nk = (max(lo, int(n * scale * rng.uniform(0.85, 1.15))) for n, lo in ((100, 36), (160, 56), (80, 32)))
    while ni * nj * nk > 43_000_000:
        nj -= 7
    small = ni * nj * nk < 3_000_000
    call = rng.choice(["run", "run", "records", "noalloc", "snapshot", "ensemble"] if small else ["run", "run", "records"])
    members, sizes = 1, 0
    if call == "ensemble":
        members, sizes = rng.randint(3, 7), rng.randrange(1 << 20)
        ni, nj, nk = 160, 256, 128
    faults = rng.randint(0, 1) if call == "snapshot" else (2 if small and call != "ensemble" and rng.random() < 0.25 else 1)
    boundary = "pml" if call == "ensemble" else rng.choice(["pml", "pml", "pml", "sponge"])
    topo = faults == 0 or (faults == 1 and rng.random() < 0.6)
    edge = min(ni, nj, nk)
    layers = 10 if call == "ensemble" else rng.randint(5, max(6, min(20, edge // 7)))
    if call == "snapshot":
        boundary = "pml"
    return {**DEFAULTS, "ni": ni, "nj": nj, "nk": nk, "faults": faults, "method": rng.choice([1, 2]),
            "free": call == "ensemble" or rng.random() < 0.75, "boundary": boundary, "layers": layers, "topo": topo,
            "dip": rng.choice([45.0, 60.0, 75.0]) if topo and faults == 1 and rng.random() < 0.3 else 0.0,
            "margin": 10 if call == "ensemble" else rng.randint(8, max(9, min(40, nk // 3))),
            "steps": 8 if ni * nj * nk > 8_000_000 else rng.randint(8, 24), "call": call,
            "every": rng.choice([1, 4, 10]), "members": members, "sizes": sizes}


# ---- problems -----------------------------------------------------------------

def _spacing(case):
    return 100.0 if case["topo"] else 200.0


@functools.lru_cache(maxsize=2)
def _coords(ni, nj, nk, h, dip):
    """Grid under Gaussian hills, stretched from a flat bottom and sheared for a
    dipping fault plane x index ni // 2; [nk, nj, ni] float32 each."""
    rng = random.Random(1001)
    dev = "cuda"
    x = (torch.arange(ni, device=dev, dtype=torch.float64) - ni // 2) * h
    y = (torch.arange(nj, device=dev, dtype=torch.float64) - nj / 2.0) * h
    topo = torch.zeros(nj, ni, device=dev, dtype=torch.float64)
    for _ in range(6):
        amp, sig = rng.uniform(0.5, 3.0) * h, rng.uniform(0.12, 0.25) * nj * h
        cx, cy = rng.uniform(-0.3, 0.3) * ni * h, rng.uniform(-0.4, 0.4) * nj * h
        topo += amp * torch.exp(-((x[None, :] - cx) ** 2 + (y[:, None] - cy) ** 2) / (2 * sig * sig))
    bottom = -(nk - 1) * h
    t = torch.arange(nk, device=dev, dtype=torch.float64) / (nk - 1.0)
    z = bottom + (topo[None] - bottom) * t[:, None, None]
    x3 = x.expand(nk, nj, ni)
    if dip:
        x3 = x3 + (topo[None] - z) / math.tan(math.radians(dip))
    y3 = y[:, None].expand(nk, nj, ni)
    return tuple(v.float().contiguous().cpu().numpy() for v in (x3, y3, z))


@functools.lru_cache(maxsize=2)
def _medium(ni, nj, nk, h, layered):
    """Homogeneous, or four layers with a smooth 3% perturbation; lambda, mu, rho."""
    if not layered:
        mu = np.float32(VS * VS * RHO)
        lam = np.float32(VP * VP * RHO - 2.0 * VS * VS * RHO)
        return tuple(np.full((nk, nj, ni), v, np.float32) for v in (lam, mu, np.float32(RHO))), VP
    dev, rng = "cuda", random.Random(1002)
    k, j, i = (torch.arange(n, device=dev, dtype=torch.float32).reshape(s)
               for n, s in ((nk, (-1, 1, 1)), (nj, (1, -1, 1)), (ni, (1, 1, -1))))
    depth = (nk - 1 - k) / (nk - 1.0)
    vs = torch.full((nk, 1, 1), 2000.0, device=dev)
    for frac, v in ((0.08, 2600.0), (0.25, 3100.0), (0.5, 3600.0)):
        vs = torch.where(depth >= frac, torch.full_like(vs, v), vs)
    pert = 0.0
    for _ in range(4):
        a, b, c, ph = (rng.uniform(0.05, 0.5) for _ in range(4))
        pert = pert + torch.sin(a * i + b * j + 6 * ph) * torch.cos(c * k + ph)
    vs = vs * (1.0 + 0.015 * pert)
    vp = 1.73 * vs
    rho = 310.0 * vp ** 0.25
    mu = vs * vs * rho
    out = tuple(v.expand(nk, nj, ni).contiguous().cpu().numpy() for v in (vp * vp * rho - 2.0 * mu, mu, rho))
    return out, float(vp.max())


def _problem(case, seed):
    ni, nj, nk, h, margin = case["ni"], case["nj"], case["nk"], _spacing(case), case["margin"]
    (lam, mu, rho), vp = _medium(ni, nj, nk, h, case["topo"])
    rng = np.random.default_rng(seed)
    nf, L, free, dip = case["faults"], case["layers"], case["free"], case["dip"]
    cot = 1.0 / math.tan(math.radians(dip)) if dip else 0.0
    dt = 0.5 * h / ((math.sqrt(2.0 + (1.0 + cot) ** 2) if dip else math.sqrt(3.0)) * vp)
    # one fault at the x centre, or two a third of the box apart
    planes = [ni // 2 + 1] if nf == 1 else [ni // 3 + 1, 2 * ni // 3 + 1][:nf]
    j1, j2, k1 = int(nj * 0.125) + 1, int(nj * 0.875) + 1, int(nk * 0.25) + 1
    shape = (nf, nk, nj)
    mu_s = np.full(shape, 1000.0, np.float32)
    mu_s[:, k1 - 1:nk, j1 - 1:j2] = 0.65
    # shear traction: a von Karman field below the static strength with a nucleation patch above it
    ts = np.empty(shape)
    for f in range(nf):
        ts[f] = np.minimum(60.0 + 8.0 * von_karman(nj, nk, h, rng=rng), 64.5)
        half = max(2, min(7, nk // 12))
        kt = nk - margin // 2 if free else nk - margin
        jc, kc = int(rng.integers(nj // 2 - 3, nj // 2 + 4)), (max(k1, margin) + kt) // 2
        ts[f, kc - half:kc + half + 1, jc - half:jc + half + 1] = 80.0 if dip else 70.0
    d = math.radians(dip) if dip else math.pi / 2
    full = lambda v: np.full(shape, v, np.float32)
    pml = L if case["boundary"] == "pml" else 0
    abl = L if case["boundary"] == "sponge" else 0
    faces = lambda n: ((n, n), (n, n), (n, 0 if free else n))
    if case["topo"] or nf == 0:
        x3, y3, z3 = _coords(ni, nj, nk, h, dip)
        geo = dict(grid_mode=GRID_IMPORT, x3d=x3, y3d=y3, z3d=z3)
    else:
        jj, kk = np.meshgrid(np.arange(1, nj + 1), np.arange(1, nk + 1))
        fx = np.stack([np.full((nk, nj), (p - planes[0]) * h) for p in planes])
        geo = dict(grid_mode=GRID_FAULT_PLANE, fault_interval=h, fault_x=fx.astype(np.float32),
                   fault_y=np.stack([(jj - nj / 2.0) * h] * nf).astype(np.float32),
                   fault_z=np.stack([(kk - nk) * h] * nf).astype(np.float32))
    sta = np.stack([rng.integers(L + 2, ni - L - 2, 16), rng.integers(L + 2, nj - L - 2, 16), np.full(16, nk - 1)], 1)
    fsta = np.array([[nj // 2, (margin + nk) // 2]] * nf, np.float32).reshape(nf, 2)
    return Problem(ni=ni, nj=nj, nk=nk, dt=float(np.float32(dt)), lam=lam, mu=mu, rho=rho, fault_x_index=planes,
                   fault_grid=[[j1, j2, k1, nk]] * nf, T0x=full(-100.0 * MPA * math.sin(d)),
                   T0y=(ts * MPA).astype(np.float32), T0z=full(-100.0 * MPA * math.cos(d) if dip else 0.0), mu_s=mu_s,
                   mu_d=full(0.5), Dc=full(0.3), C0=full(0.0), dynamic_method=case["method"], welded_margin=margin,
                   free_surface=int(free), pml_layers=faces(pml), pml_ref_vel=((vp, vp),) * 3,
                   ablexp_layers=faces(abl), ablexp_ref_vel=((vp, vp),) * 3, stations=sta.astype(np.float32),
                   fault_stations=fsta, fault_station_fault=np.arange(nf, dtype=np.int32), max_records=512,
                   name=case["call"], **geo)


@functools.lru_cache(maxsize=4)
def _shared_setup(items):
    case = dict(items)
    p = _problem(case, 0)
    return p, Setup(p)


def _waves(case, seed, n):
    """n smooth random fields [nk, nj, ni], values of order one: sums of plane waves 8 to 40 points long."""
    g = torch.Generator().manual_seed(seed)
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    k, j, i = (torch.arange(m, device="cuda", dtype=torch.float32).reshape(s)
               for m, s in ((nk, (-1, 1, 1)), (nj, (1, -1, 1)), (ni, (1, 1, -1))))
    out = []
    for _ in range(n):
        f = torch.zeros(nk, nj, ni, device="cuda")
        for _ in range(4):
            u = torch.randn(3, generator=g)
            u = u / u.norm() * 2 * math.pi / (8.0 + 32.0 * float(torch.rand(1, generator=g)))
            f += torch.sin(float(u[0]) * i + float(u[1]) * j + (float(u[2]) * k + 6.3 * float(torch.rand(1, generator=g))))
        out.append((0.5 * f).cpu().numpy())
    return out


def _member_cases(case):
    """An ensemble's members: uneven sizes in the generator's ranges, half of them under hills."""
    r = random.Random(case["sizes"])
    return [{**case, "ni": r.randint(64, 160), "nj": r.randint(96, 256), "nk": r.randint(64, 128),
             "topo": bool(q % 2), "members": 1} for q in range(case["members"])]


def _solver(case, seed):
    """A solver with a wavefield already in the box: waves that earlier slip and sources radiated."""
    if case["ni"] * case["nj"] * case["nk"] >= SHARED:
        prob, setup = _shared_setup(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
        s = Solver(prob, setup=setup)
    else:
        s = Solver(_problem(case, seed))
    if case["call"] == "snapshot":
        for c, f in zip(WAVE_COMPONENTS, _waves(case, seed, 9)):
            s.set_wavefield(c, f * (0.05 if c[0] == "V" else 0.5 * MPA))
    else:
        s.set_wavefield("Txy", _waves(case, seed, 1)[0] * (0.5 * MPA))
    return s


def prepare(case, seed):
    if case["call"] == "ensemble":
        solvers = [_solver(m, seed + 101 * q) for q, m in enumerate(_member_cases(case))]
        return {"case": case, "solvers": solvers, "ensemble": Ensemble(solvers)}
    st = {"case": case, "solver": _solver(case, seed)}
    if case["call"] == "records":
        n = -(-case["steps"] // case["every"])
        st["records"] = torch.empty((n, case["faults"], len(FAULT_FIELDS), case["nk"], case["nj"]),
                                    dtype=torch.float32, pin_memory=True)
    return st


def _fault(a):
    """The 11 fields by what they are: traction, slip rate, slip, peak rate, rupture time."""
    return {"traction": a[..., 0:3, :, :], "rate": a[..., 3:6, :, :], "slip": a[..., 6:9, :, :],
            "peak": a[..., 9, :, :], "time": a[..., 10, :, :]}


def run(state):
    case = state["case"]
    if case["call"] == "ensemble":
        state["ensemble"].run(case["steps"])
        return [_fault(s.fault_all(0)) for s in state["solvers"]]
    s = state["solver"]
    if case["call"] == "records":
        buf = state["records"]
        n = s.run_fault_output(case["steps"], case["every"], out_ptr=buf.data_ptr(), max_records=len(buf))
        return {"records": n, **_fault(buf[:n])}
    if case["call"] == "noalloc":
        s.run_noalloc(case["steps"])
    else:
        s.run(case["steps"])
    if case["call"] == "snapshot":
        return {c: s.wavefield(c) for c in WAVE_COMPONENTS}
    st = s.stations()
    out = {"faults": [_fault(s.fault_all(f)) for f in range(case["faults"])],
           "station_velocity": st[:, :3], "station_stress": st[:, 3:]}
    if case["free"]:
        p = s.surface_peaks()
        out.update(pgv=p[0:5], pga=p[5:10], pgd=p[10:15])
    return out


def work(case):
    """Per step and point: the nine components in and out and the twelve metric and medium values in; per point of
    a PML face its nine auxiliary values in and out; four stages of about 380 operations per point."""
    cases = _member_cases(case) if case["call"] == "ensemble" else [case]
    b = f = 0.0
    for c in cases:
        ni, nj, nk = c["ni"], c["nj"], c["nk"]
        pts, face = ni * nj * nk, 0
        if c["boundary"] == "pml":
            face = (c["layers"] + 1) * (2 * nj * nk + 2 * ni * nk + (1 if c["free"] else 2) * ni * nj)
        b += c["steps"] * 4.0 * (30 * pts + 18 * face)
        f += c["steps"] * 4 * 380.0 * pts
        if c["call"] == "snapshot":
            b += 72.0 * pts
    return {"bytes": b, "flops": f}


# ---- the step in 64 bits --------------------------------------------------------

C5 = (-0.291647047, -0.666745142, 1.250117713, -0.333411808, 0.041686285)
PAIRS = ((0, 0, 0), (1, 1, 0), (1, 1, 1), (0, 0, 1), (0, 1, 0), (1, 0, 0), (1, 0, 1), (0, 1, 1))
G = 3                                                   # ghost points


def _shift(a, dim, m):
    """a at the interior points moved m points along dim (2 x, 1 y, 0 z of the last three axes)."""
    ix = [slice(G, -G)] * 3
    n = a.shape[a.dim() - 3 + dim]
    ix[dim] = slice(G + m, n - G + m)
    return a[(Ellipsis, *ix)]


def _deriv(a, dim, forward):
    w = C5 if forward else tuple(-v for v in C5)
    return sum(v * _shift(a, dim, m if forward else -m) for v, m in zip(w, (-1, 0, 1, 2, 3)))


def _rhs(D, e, lam, mu, slw):
    """One direction's part of the right-hand side from the nine derivatives D along it and its metric row e."""
    vx, vy, vz, xx, yy, zz, yz, xz, xy = D
    div = e[0] * vx + e[1] * vy + e[2] * vz
    return torch.stack([slw * (e[0] * xx + e[1] * xy + e[2] * xz), slw * (e[0] * xy + e[1] * yy + e[2] * yz),
                        slw * (e[0] * xz + e[1] * yz + e[2] * zz),
                        lam * div + 2 * mu * e[0] * vx, lam * div + 2 * mu * e[1] * vy, lam * div + 2 * mu * e[2] * vz,
                        mu * (e[2] * vy + e[1] * vz), mu * (e[2] * vx + e[0] * vz), mu * (e[1] * vx + e[0] * vy)])


def _extend(a):
    """Linear extrapolation of a [nz, ny, nx] field into its ghost points, x then y then z."""
    for dim in (2, 1, 0):
        n = a.shape[dim]
        at = lambda q: a.select(dim, q)
        for q in range(G):
            at(q).copy_(2 * at(G) - at(2 * G - q))
            at(n - 1 - q).copy_(2 * at(n - 1 - G) - at(n - 1 - 2 * G + q))
    return a


def _pml_profiles(P, X, dim, side):
    """alpha + d / beta, 1 / beta and d / beta per layer of one CFS-PML face, from the interior edge outwards."""
    L = P.pml_layers[dim][side]
    ax = 2 - dim
    n = X[0].shape[ax]
    ext = [x.narrow(ax, 0 if side == 0 else n - L - 1, L + 1) for x in X]
    dh = float(torch.sqrt(sum((e.narrow(ax, 1, L) - e.narrow(ax, 0, L)) ** 2 for e in ext)).mean())
    rpp = 10.0 ** -((math.log10(L) - 1.0) / math.log10(2.0) + 4.0)
    dmax = -P.pml_ref_vel[dim][side] / (2.0 * dh * L) * math.log(rpp) * 3.0
    r = torch.arange(L + 1, dtype=torch.float64, device=X[0].device) / L
    if side == 0:
        r = r.flip(0)
    beta = 1.0 + (P.pml_beta_max[dim][side] - 1.0) * r * r
    dd = dmax * r * r / beta
    return P.pml_alpha_max[dim][side] * (1.0 - r) + dd, 1.0 / beta, dd


def _convert(b, q, e3, lam, mu):
    """b-derivatives of the velocity turned into the dz part that keeps the surface free of traction."""
    def block(a, c):
        ab = (a * c).sum(0)
        I = torch.eye(3, dtype=a.dtype, device=a.device)
        return (lam * torch.einsum("r...,c...->...rc", a, c).movedim((-2, -1), (0, 1)) +
                mu * torch.einsum("r...,c...->...rc", c, a).movedim((-2, -1), (0, 1)) +
                mu * ab * I[(...,) + (None,) * ab.dim()]).movedim((0, 1), (-2, -1))
    m = -torch.linalg.solve(block(e3, e3), block(e3, b))
    return torch.einsum("...rc,c...->r...", m, q)


def exact(case, seed):
    """Plain restatement of the faultless step (metric, stencils, CFS-PML, traction-image free surface, RK4) in
    64 bits.  None with a fault: the split-node law is nonlinear and its restatement as long as the solver."""
    if case["faults"] or case["call"] != "snapshot" or case["boundary"] != "pml" or \
            case["ni"] * case["nj"] * case["nk"] * case["steps"] > 40_000_000:
        return None
    P = _problem(case, seed)
    dev, f8 = "cuda", torch.float64
    ni, nj, nk = P.ni, P.nj, P.nk
    inner = (Ellipsis, slice(G, -G), slice(G, -G), slice(G, -G))
    pad = lambda a: torch.nn.functional.pad(torch.as_tensor(a, dtype=f8, device=dev), (G,) * 6)
    X0 = [torch.as_tensor(v, dtype=f8, device=dev) for v in (P.x3d, P.y3d, P.z3d)]
    X = [_extend(pad(x)) for x in X0]
    w6 = ((-3, -0.01666667), (-2, 0.15), (-1, -0.75), (1, 0.75), (2, -0.15), (3, 0.01666667))
    cov = [torch.stack([sum(w * _shift(x, 2 - d, m) for m, w in w6) for x in X]) for d in range(3)]
    cross = [torch.linalg.cross(cov[(d + 1) % 3], cov[(d + 2) % 3], dim=0) for d in range(3)]
    jac = (cross[2] * cov[2]).sum(0)
    E = [c / jac for c in cross]
    JE = [torch.stack([_extend(pad(jac)) * _extend(pad(c)) for c in e]) for e in E]
    lam, mu, rho = (torch.as_tensor(v, dtype=f8, device=dev) for v in (P.lam, P.mu, P.rho))
    slw = 1.0 / rho
    faces = []
    for d in range(3):
        for side in range(2):
            L = P.pml_layers[d][side]
            if L:
                ax, n = 2 - d, (ni, nj, nk)[d]
                shape = [1, 1, 1]
                shape[ax] = L + 1
                prof = [v.reshape(shape) for v in _pml_profiles(P, X0, d, side)]
                cut = lambda a, ax=ax, side=side, n=n, L=L: a.narrow(a.dim() - 3 + ax, 0 if side == 0 else n - L - 1, L + 1)
                faces.append((d, cut, prof))
    top = (Ellipsis, nk - 1, slice(None), slice(None))
    free = bool(P.free_surface)
    e3s, es = E[2][top], [E[0][top], E[1][top]]

    def rates(u, aux, dirs):
        """Right-hand sides of the wavefield u [9, ...] with ghosts and of the faces' auxiliary fields."""
        h, daux, dv = 0.0, [], []
        parts = []
        for d in range(3):
            D = _deriv(u, 2 - d, dirs[d])
            dv.append(D[:3])
            parts.append(_rhs(D, E[d], lam, mu, slw))
        h = parts[0] + parts[1] + parts[2]
        if free:
            # dz of the velocity at and just under the surface
            v = u[:3]
            sgn = 1 if dirs[2] else -1
            row = lambda m: v[:, G + nk - 1 + m, G:-G, G:-G]
            two = lambda k0: sgn * (row(k0 + sgn) - row(k0))
            four = lambda k0: sgn * (-7.0 * row(k0) + 8.0 * row(k0 + sgn) - row(k0 + 2 * sgn)) / 6.0
            surf = sum(_convert(es[d], dv[d][top], e3s, lam[top], mu[top]) for d in range(2))
            zero = torch.zeros_like(surf)
            for k0, dz in ((0, surf), (-1, two(-1)), (-2, four(-2))):
                at = (Ellipsis, nk - 1 + k0, slice(None), slice(None))
                new = _rhs(torch.cat([dz, zero, zero]), E[2][at], lam[at], mu[at], slw[at])
                h[3:, nk - 1 + k0] += new[3:] - parts[2][3:, nk - 1 + k0]
            # momentum with the traction's odd image about the surface
            xx, yy, zz, yz, xz, xy = u[3:]
            rows = ((xx, xy, xz), (xy, yy, yz), (xz, yz, zz))
            T = [torch.stack([sum(JE[d][q] * r[q] for q in range(3)) for r in rows]) for d in range(3)]
            kt = G + nk - 1
            T[2][:, kt] = 0.0
            for m in range(1, G + 1):
                T[2][:, kt + m] = -T[2][:, kt - m]
            m = 4 if dirs[2] else 2
            img = sum(_deriv(T[d], 2 - d, dirs[d]) for d in range(3)) * slw / jac
            h[:3, nk - m:] = img[:, nk - m:]
        for n, (d, cut, (cA, cB, cD)) in enumerate(faces):
            r, a = cut(parts[d]).clone(), aux[n]
            if free and d < 2:
                # the surface row's converted dz gradient belongs to this direction too
                z = _convert(cut_top(cut, es[d]), cut_top(cut, dv[d][top]), cut_top(cut, e3s), cut_top(cut, lam[top]), cut_top(cut, mu[top]))
                zero = torch.zeros_like(z)
                q = _rhs(torch.cat([z, zero, zero]), cut_top(cut, e3s), cut_top(cut, lam[top]), cut_top(cut, mu[top]), cut_top(cut, slw[top]))
                r[3:, -1] += q[3:]
            cut(h).add_((cB - 1.0) * r - cB * a)
            daux.append(cD * r - cA * a)
        return h, daux

    def cut_top(cut, a):
        """A face's part of a surface field [..., nj, ni]."""
        return cut(a.unsqueeze(-3).expand(*a.shape[:-2], nk, nj, ni))[..., -1, :, :]

    u = torch.stack([pad(f * np.float32(0.05 if c[0] == "V" else 0.5 * MPA))
                     for c, f in zip(WAVE_COMPONENTS, _waves(case, seed, 9))])
    aux = [torch.zeros_like(cut(u[inner])) for _, cut, _ in faces]
    dt = float(np.float32(P.dt))
    ka, kb = (0.5, 0.5, 1.0), (1 / 6, 1 / 3, 1 / 3, 1 / 6)
    for it in range(case["steps"]):
        cu, ca, nu, na = u, aux, u.clone(), [a.clone() for a in aux]
        for st in range(4):
            h, da = rates(cu, ca, [(p + st) % 2 for p in PAIRS[it % 8]])
            nu[inner] += kb[st] * dt * h
            na = [a + kb[st] * dt * x for a, x in zip(na, da)]
            if st < 3:
                cu = u.clone()
                cu[inner] += ka[st] * dt * h
                ca = [a + ka[st] * dt * x for a, x in zip(aux, da)]
        u, aux = nu, na
    return {c: u[q][inner].contiguous() for q, c in enumerate(WAVE_COMPONENTS)}
