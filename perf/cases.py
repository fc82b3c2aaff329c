"""The solve stage's work, as a driver has it do it: a case's state handed over, a number of time steps,
the state back. perf.cases says what is timed (listed, draw), how it is set up (prepare), called (run)
and what the answer is in plain float64 torch (exact).

A case is a box of nx x ny x nz equal cells, cut into bx x by x bz blocks at ragged planes (blocks meet at
matched connections, code 101), with one boundary code per axis (400 open, 300 wall, 201 periodic) and:

  families   closures advanced together, "MK+IG+AG"
  precision  "fp64" (plain form) or "fp32flux" (the form the benchmark runs)
  scheme, limiter, riemann ("" = the closure's default), sensor (Jameson sensor), steady (local steps)
  gas        one-way coupling to a frozen gas: drag, heat, radiation
  evap       the IG and AG families evaporate (CEM, Langmuir-Knudsen interface, Stefan blowing)
  cloud      the seeded droplet blobs over a nearly empty floor; otherwise a smooth stream
  steps      time steps of one pass
  call       "host": one step_host call takes the state in page-locked arrays in and out;
             "loop": upload, one step call of all the steps, download;
             "each": the same with one step call per time step, as a driver that looks at each report
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from ice_b200 import abi
from ice_b200.case import Case, Family, Numerics, box_bc, box_nodes, empty_state
from ice_b200.solver import Solver

NC = {"MK": 6, "IG": 7, "AG": 12}
NRK = {"euler": 1, "RK2": 2, "RK3": 3}
CELL = 1e-4                       # cell size of the 3-D and 2-D boxes [m]
RADIUS = {"MK": 10e-6, "IG": 30e-6, "AG": 60e-6}
GAS_R, GAS_GAMMA, GAS_K, GAS_MU = 287.05, 1.4, 0.026, 1.8e-5


def _case(**kw):
    c = dict(nx=1, ny=1, nz=1, bx=1, by=1, bz=1, bc=400, families="IG", precision="fp64", scheme="RK2",
             limiter="vanleer", riemann="", sensor=False, steady=False, gas=False, evap=False, cloud=False,
             steps=10, call="host")
    c.update(kw)
    return c


def listed():
    return [
        # A shock tube of the 1-D Riemann configuration (2,000 cells, HLLE, minmod): launches are all it costs.
        _case(name="tube1d_ig_fp64", nx=2000, scheme="RK3", limiter="minmod", riemann="HLLE", steps=100, call="loop"),
        # A validation-sized plane run with local steps, the driver reading every step's report.
        _case(name="plane_mk_steady_fp64", families="MK", nx=100, ny=100, steady=True, steps=50, call="each"),
        # The two-family plane jets' numerics (MK and IG together, frozen gas, Rusanov, RK2).
        _case(name="plane_mk_ig_fp32", families="MK+IG", nx=509, ny=512, precision="fp32flux", riemann="Rusanov",
              gas=True, steps=40),
        # The reference's published benchmark shape (one IG block, drag and heat, RK2), in both forms.
        _case(name="box_ig_fp32", nx=128, ny=126, nz=129, precision="fp32flux", gas=True, steps=20),
        _case(name="box_ig_fp64", nx=96, ny=95, nz=97, gas=True, steps=10),
        # The evaporating AG droplet cloud (RK3, sensor), in both forms.
        _case(name="cloud_ag_fp32", families="AG", nx=96, ny=96, nz=96, precision="fp32flux", scheme="RK3", sensor=True,
              gas=True, evap=True, cloud=True, steps=10),
        _case(name="cloud_ag_fp64", families="AG", nx=64, ny=61, nz=67, scheme="RK3", sensor=True, gas=True, evap=True,
              cloud=True, steps=10),
        # A small block of the same cloud: too few cells to fill the GPU.
        _case(name="cloud_ag_small_fp32", families="AG", nx=32, ny=29, nz=31, precision="fp32flux", scheme="RK3",
              sensor=True, gas=True, evap=True, cloud=True, steps=20, call="loop"),
        # The headline workload's recipe: three families over ragged joined blocks.
        _case(name="blocks_all_fp32", families="MK+IG+AG", nx=131, ny=109, nz=118, bx=2, by=2, bz=2,
              precision="fp32flux", scheme="RK3", sensor=True, gas=True, evap=True, cloud=True, steps=8),
        _case(name="blocks_all_fp64", families="MK+IG+AG", nx=77, ny=64, nz=71, bx=2, by=2, bz=1, scheme="RK3",
              sensor=True, gas=True, evap=True, cloud=True, steps=5),
        # The same, by a driver that keeps the state in its own arrays: one step a call.
        _case(name="blocks_all_step_fp32", families="MK+IG+AG", nx=101, ny=109, nz=97, bx=2, by=2, bz=2,
              precision="fp32flux", scheme="RK3", sensor=True, gas=True, evap=True, cloud=True, steps=1),
        # Free transport on a periodic box, an inert MK family with its default Saurel solver.
        _case(name="periodic_mk_fp64", families="MK", nx=95, ny=61, nz=83, bc=201, scheme="RK3", limiter="mc", steps=10),
    ]


def _cost(c):
    """Relative time of a pass: stage updates of variables, plain form at about four times the other's."""
    nc = sum(NC[f] for f in c["families"].split("+"))
    return c["nx"] * c["ny"] * c["nz"] * nc * NRK[c["scheme"]] * c["steps"] * (4 if c["precision"] == "fp64" else 1)


_MOST = 131 * 109 * 118 * 25 * 3 * 8


def draw(rng):
    logu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    ndir = rng.choice([1, 2, 3, 3, 3, 3])
    fams = rng.choice(["MK", "IG", "IG", "AG", "AG", "MK+IG", "MK+IG+AG", "MK+IG+AG"])
    if ndir == 1:
        n = (logu(200, 4000), 1, 1)
    elif ndir == 2:
        n = (logu(40, 600), logu(40, 600), 1)
    else:
        m = logu(20, 128)
        n = tuple(max(16, int(m * rng.uniform(0.75, 1.25))) for _ in range(3))
    cloud = ndir == 3 and rng.random() < 0.6
    gas = cloud or rng.random() < 0.5
    c = _case(families=fams, nx=n[0], ny=n[1], nz=n[2], precision=rng.choice(["fp64", "fp32flux"]),
              scheme=rng.choice(["RK2", "RK3", "RK3"]), limiter=rng.choice(["vanleer", "vanleer", "vanleer", "minmod", "mc"]),
              riemann=rng.choice(["", "", "Rusanov", "HLLE"]), gas=gas, cloud=cloud, sensor=cloud, evap=cloud,
              steady=ndir == 2 and rng.random() < 0.4, steps=rng.choice([5, 10, 20, 40]))
    if ndir == 3:
        c["bx"], c["by"], c["bz"] = rng.choice([(1, 1, 1), (1, 1, 1), (2, 1, 1), (2, 2, 1), (2, 2, 2), (3, 2, 1)])
    c["bc"] = 400 if cloud else rng.choice([400, 400, 300, 201])
    c["call"] = rng.choice(["host", "loop", "each"]) if ndir < 3 else rng.choice(["host", "host", "loop"])
    while _cost(c) > _MOST and c["steps"] > 1:
        c["steps"] = max(1, c["steps"] // 2)
    while _cost(c) > _MOST:
        c["nx"], c["ny"], c["nz"] = (max(16, int(v * 0.9)) for v in (c["nx"], c["ny"], c["nz"]))
    return c


# ----------------------------------------------------------------------------- set-up
def _cuts(n, b):
    """b ragged parts of n cells, each at least n / (2 b)."""
    at = [int(round(n * (q + 0.13 * math.sin(2.3 * q)) / b)) for q in range(1, b)]
    return [0] + at + [n]


def _h(c):
    return CELL if c["ny"] > 1 else 1.0 / c["nx"]


def _spans(c):
    """Per block, in block order, ((x0, x1), (y0, y1), (z0, z1)) of its cells in the box."""
    xs, ys, zs = _cuts(c["nx"], c["bx"]), _cuts(c["ny"], c["by"]), _cuts(c["nz"], c["bz"])
    return [((xs[a], xs[a + 1]), (ys[b], ys[b + 1]), (zs[d], zs[d + 1]))
            for d in range(c["bz"]) for b in range(c["by"]) for a in range(c["bx"])]


def _families(c):
    out = []
    for f in c["families"].split("+"):
        drop = dict(rho_al=1000.0, cs_al=4180.0, lv_al=2.26e6, emiss=0.9 if c["evap"] else 0.0, Mv=18.015, cpv=1996.0,
                    Le=1.0, Tboil=373.15)
        riemann = c["riemann"]
        if f == "MK":
            out.append(Family("MK", riemann=riemann, rho_al=2700.0, cs_al=900.0, emiss=0.8 if c["evap"] else 0.0))
        else:
            out.append(Family(f, riemann=riemann, evap="CEM" if c["evap"] else "none",
                              intf="LK" if c["evap"] else "VLE", **drop))
    return out


def _numerics(c):
    return Numerics(scheme=c["scheme"], time_accurate=not c["steady"], cfl=0.5, dt_max=1.0, limiter=c["limiter"],
                    shock_detector=c["sensor"], coupled=c["gas"], drag="Schiller-Naumann", heat="Ranz-Marshall",
                    blowing=c["evap"], precision=abi.PREC_FP64 if c["precision"] == "fp64" else abi.PREC_FP32FLUX)


@functools.lru_cache(maxsize=2)
def _mesh(nx, ny, nz, bx, by, bz, bc, fams):
    """The case without its state: nodes, boundary table, metrics and paired records. A driver keeps its
    mesh; only the state and the gas are new with a seed."""
    c = _case(nx=nx, ny=ny, nz=nz, bx=bx, by=by, bz=bz, bc=bc, families=fams)
    h, spans = _h(c), _spans(c)
    nodes = [box_nodes(*(s[1] - s[0] for s in sp), lo=tuple(s[0] * h for s in sp),
                       size=tuple((s[1] - s[0]) * h for s in sp)) for sp in spans]
    n, cuts = (nx, ny, nz), (bx, by, bz)
    at = {sp: b for b, sp in enumerate(spans)}
    starts = [{s[d][0]: s[d] for s in spans} for d in range(3)]
    ends = [{s[d][1]: s[d] for s in spans} for d in range(3)]
    rows = []
    for b, sp in enumerate(spans):
        dims = tuple(s[1] - s[0] for s in sp)
        codes, across = {}, {}
        for f in range(1, 7):
            d, up = (f - 1) // 2, f % 2 == 0
            edge = sp[d][1] if up else sp[d][0]
            inside = 0 < edge < n[d]
            codes[f] = 101 if inside else 0 if n[d] == 1 else bc
            if codes[f] in (101, 201):
                e = edge % n[d] if up else (edge or n[d])
                part = (starts if up else ends)[d][e]
                other = sp[:d] + (part,) + sp[d + 1:]
                across[f] = (at[other], 1 if up else part[1] - part[0], f - 1 if up else f + 1)
        for (bb, i, j, k, f, code, pay) in box_bc(b + 1, dims, codes):
            if f in across:
                ob, cell, of = across[f]
                src = [i, j, k]
                src[(f - 1) // 2] = cell
                pay = (ob + 1, *src, of)
            rows.append((bb, i, j, k, f, code, pay))
    case = Case("perf", nodes, _families(c), _numerics(c), rows)
    case.build_geometry()
    case.build_records(abi.load_gpu())
    return case


def _waves(g, xyz, L, count, rms):
    """A divergence-free sum of seeded Fourier modes, |k| in 1..8 units of 2 pi / L, with the given RMS."""
    u = [0.0, 0.0, 0.0]
    total = 0.0
    dims = [k for k, x in enumerate(xyz) if x.numel() > 1]
    for _ in range(count):
        k = np.zeros(3)
        while not 1.0 <= np.linalg.norm(k) <= 8.0:
            k[dims] = g.integers(-8, 9, size=len(dims))
        a = g.normal(size=3)
        a = a - k * (a @ k) / (k @ k)
        a = a / max(np.linalg.norm(a), 1e-30) / np.linalg.norm(k)
        cs = torch.cos(sum(float(2.0 * math.pi / L * kk) * x for kk, x in zip(k, xyz)) + float(g.uniform(0, 2 * math.pi)))
        u = [p + float(q) * cs for p, q in zip(u, a)]
        total += 0.5 * float(a @ a)
    return [p * (rms / math.sqrt(total)) for p in u]


def _blobs(centres, xyz, width):
    x, y, z = xyz
    return [torch.exp(-((x - float(a)) ** 2 + (y - float(b)) ** 2 + (z - float(d)) ** 2) / (2.0 * width ** 2))
            for a, b, d in centres]


def _fields(c, seed):
    """The seeded box: per family its primitives (nc, nz, ny, nx) and the gas (9, nz, ny, nx) or None, float64
    on the GPU."""
    g = np.random.default_rng(seed)
    h = _h(c)
    n = (c["nx"], c["ny"], c["nz"])
    L = max(n) * h
    ax = [(torch.arange(m, dtype=torch.float64, device="cuda") + 0.5) * h for m in n]
    xyz = (ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None])
    shape = (n[2], n[1], n[0])
    full = lambda v: v.expand(shape) if torch.is_tensor(v) else torch.full(shape, float(v), dtype=torch.float64, device="cuda")
    spots = lambda m: np.stack([g.uniform(0.15, 0.85, size=m) * q * h for q in n], axis=-1)
    gas = None
    if c["gas"]:
        vel = _waves(g, xyz, L, 32, 15.0 if c["cloud"] else 10.0)
        T = full(300.0)
        if c["cloud"]:
            T = 300.0 + 1200.0 * torch.clamp(sum(_blobs(spots(8), xyz, 0.15 * L)), max=1.0)
        gas = torch.stack([full(v) for v in (101325.0 / (GAS_R * T), *vel, T, GAS_R, GAS_GAMMA, GAS_K, GAS_MU)])
    states = []
    for f, fam in zip(c["families"].split("+"), _families(c)):
        if c["cloud"]:
            blobs = torch.stack(_blobs(spots(16), xyz, 0.08 * L))
            rho = torch.clamp(1e-4 * fam.rho_al * torch.clamp(blobs.sum(0), max=1.0), min=1e-12)
            radius = torch.as_tensor(RADIUS[f] * np.exp(0.4 * g.normal(size=16)), device="cuda")[blobs.argmax(0)]
            u, theta, T = [gas[1], gas[2], gas[3]], 1e-2, full(300.0)
        elif c["ny"] == 1:        # two streams meeting, a seeded wave on each
            left = (xyz[0] < 0.5).double()
            wave = 1.0 + 0.1 * torch.sin(2.0 * math.pi * (6.0 * xyz[0] + g.uniform()))
            rho = full((0.5 + 0.5 * left) * wave)
            u = [full(2.0 * left - 1.0), full(0.0), full(0.0)]
            radius, theta, T = 10e-6, full(0.05 + 0.05 * left), full(300.0)
        else:                     # a smooth stream of 1e-3 kg/m3
            ph = g.uniform(0, 2 * math.pi, size=3)
            k = 2.0 * math.pi / L
            wave = full(torch.cos(k * xyz[0] + ph[0]) * torch.cos(k * xyz[1] + ph[1]) * torch.cos(k * xyz[2] + ph[2]))
            rho = 1e-3 * (1.0 + 0.3 * wave)
            w = 4.0 if c["nz"] > 1 else 0.0
            u = [10.0 + 2.0 * wave, 7.0 - wave, full(w) + (0.5 * wave if c["nz"] > 1 else 0.0)]
            radius, theta, T = RADIUS[f], 1.0 / 3.0, 300.0 + 5.0 * wave
        mass = 4.0 / 3.0 * math.pi * radius ** 3 * fam.rho_al
        p = torch.zeros((NC[f], *shape), dtype=torch.float64, device="cuda")
        p[0], p[1], p[2], p[3] = rho, u[0], u[1], u[2]
        if f == "IG":
            p[4] = rho * theta
        elif f == "AG":
            p[4], p[7], p[9] = rho * theta, rho * theta, rho * theta
            p[5] = 0.1 * rho * theta
        p[-2], p[-1] = T, rho / mass
        states.append(p)
    return states, gas


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    """The set-up solver (mesh, boundary table and gas handed over) and the state in host arrays."""
    c = case
    mesh = _mesh(c["nx"], c["ny"], c["nz"], c["bx"], c["by"], c["bz"], c["bc"], c["families"])
    states, gas = _fields(c, seed)
    states = [p.permute(1, 2, 3, 0).cpu().numpy() for p in states]
    full = Case("perf", mesh.nodes, _families(c), _numerics(c), mesh.bc_rows, geoms=mesh.geoms, rec_int=mesh.rec_int,
                rec_real=mesh.rec_real)
    gas = gas.cpu().numpy() if gas is not None else None
    for (x0, x1), (y0, y1), (z0, z1) in _spans(c):
        cut = (slice(z0, z1), slice(y0, y1), slice(x0, x1))
        per = []
        for p in states:
            a = _pinned((z1 - z0 + 4, y1 - y0 + 4, x1 - x0 + 4, p.shape[-1]))
            a[...] = np.nan
            a[2:-2, 2:-2, 2:-2] = p[cut]
            per.append(a)
        full.state.append(per)
        if gas is not None:
            own = [np.ascontiguousarray(q[cut]) for q in gas]
            full.gas.append({"prim5": np.ascontiguousarray(np.stack(own[:5], axis=-1)), "R": own[5], "gam": own[6],
                             "k": own[7], "mu": own[8]})
    out = [[_pinned(a.shape) for a in per] for per in full.state] if c["call"] == "host" else None
    return {"solver": Solver(full), "state": full.state, "out": out, "steps": c["steps"], "call": c["call"]}


def run(state):
    """The state handed over, advanced by the case's steps, and back: the interior of every block of every family
    (a ghost cell holds scratch)."""
    s = state["solver"]
    if state["call"] == "host":
        s.step_host(state["state"], state["out"], state["steps"])
        out = state["out"]
    else:
        s.upload(state["state"])
        if state["call"] == "loop":
            s.step(state["steps"])
        else:
            for _ in range(state["steps"]):
                s.step(1)
        out = s.download_all()
    return [[a[2:-2, 2:-2, 2:-2] for a in per] for per in out]


def work(case):
    """Per cell, family and stage: the state read and the new one written (16 nc bytes; 24 nc from the second stage
    on, which reads the step's first state too), the face normals and areas and the lengths (40 bytes a direction
    in FP64, 20 in the FP32-flux form), the volume, the nine gas values of a coupled run; per pass the state
    handed over and back. The floating-point operations are of the reconstruction, flux and update formulas."""
    c = case
    cells = c["nx"] * c["ny"] * c["nz"]
    ndir = sum(c[k] > 1 for k in ("nx", "ny", "nz"))
    nrk, word = NRK[c["scheme"]], 8 if c["precision"] == "fp64" else 4
    nbytes = flops = 0.0
    for f in c["families"].split("+"):
        nc = NC[f]
        fixed = 5 * word * ndir + 8 + (9 * word if c["gas"] else 0)
        per_step = nrk * fixed + 16 * nc + (nrk - 1) * 24 * nc
        nbytes += cells * (c["steps"] * per_step + 32 * nc)
        flops += cells * c["steps"] * nrk * (ndir * (22 * nc + 60) + 16 * nc + (150 if c["gas"] else 0))
    return {"bytes": nbytes, "flops": flops}


# ----------------------------------------------------------------------------- the answer in 64 bits
EPS = float(np.float32(1e-25))
TOLL = float(np.float32(1e-20))
EMPTY = 1e-6


def _conservative(f, p, cp):
    r, u, v, w = p[0], p[1], p[2], p[3]
    n2 = u * u + v * v + w * w
    if f == "MK":
        rest = [r * cp * p[4] + 0.5 * r * n2, p[5]]
    elif f == "IG":
        e = r * n2 + 3.0 * p[4]
        rest = [e, r * cp * p[5] + 0.5 * e, p[6]]
    else:
        t = [r * u * u + p[4], r * u * v + p[5], r * u * w + p[6], r * v * v + p[7], r * v * w + p[8], r * w * w + p[9]]
        rest = t + [r * cp * p[10] + 0.5 * (t[0] + t[3] + t[5]), p[11]]
    return torch.stack([r, r * u, r * v, r * w] + rest)


def _primitive(f, c, cp):
    r = c[0]
    u, v, w = (c[q] / (r + EPS) for q in (1, 2, 3))
    n2 = u * u + v * v + w * w
    if f == "MK":
        p = [r, u, v, w, (c[4] - 0.5 * r * n2) / (cp * r + EPS), c[5]]
        floor = [4, 5]
    elif f == "IG":
        P = (c[4] - r * n2) / 3.0
        P = torch.where((r <= EMPTY) & (P > r), r, P)
        p = [r, u, v, w, P, (c[5] - 0.5 * c[4]) / (cp * r + EPS), c[6]]
        floor = [4, 5, 6]
    else:
        t = [c[4] - r * u * u, c[5] - r * u * v, c[6] - r * u * w, c[7] - r * v * v, c[8] - r * v * w, c[9] - r * w * w]
        T = (c[10] - 0.5 * (c[4] + c[7] + c[9])) / (cp * r + EPS)
        tr = t[0] + t[3] + t[5]
        s = torch.where((r <= EMPTY) & (tr > 3.0 * r), 3.0 * r / tr, torch.ones_like(r))
        p = [r, u, v, w] + [q * s for q in t] + [T, c[11]]
        floor = [4, 7, 9, 10, 11]
    gone = r < EPS
    p = [torch.where(gone, torch.full_like(r, EPS), q) for q in p]
    if f == "AG":
        for q in (5, 6, 8):
            p[q] = torch.where(gone | (p[q].abs() < EPS), torch.zeros_like(r), p[q])
    for q in floor:
        p[q] = torch.where(p[q] < EPS, torch.full_like(r, EPS), p[q])
    return torch.stack(p)


def _physical(f, p):
    ok = torch.isfinite(p).all(0) & (p[0] >= 0)
    for q in {"MK": (), "IG": (4,), "AG": (4, 7, 9)}[f]:
        ok = ok & (p[q] >= 0)
    return ok


def _pressure(f, p, d):
    """P . n of the velocity covariance for the axis d."""
    if f == "IG":
        z = torch.zeros_like(p[4])
        return [p[4] if q == d else z for q in range(3)]
    return [p[q] for q in ((4, 5, 6), (5, 7, 8), (6, 8, 9))[d]]


def _sound(f, p, d):
    if f == "MK":
        return torch.zeros_like(p[0])
    pn = _pressure(f, p, d)[d]
    return torch.sqrt(3.0 * torch.clamp(pn, min=0.0) / (p[0] + EPS))


def _flux(f, p, d, cp):
    r, U = p[0], [p[1], p[2], p[3]]
    un = U[d]
    n2 = U[0] ** 2 + U[1] ** 2 + U[2] ** 2
    m = r * un
    if f == "MK":
        return torch.stack([m, m * U[0], m * U[1], m * U[2], m * (0.5 * n2 + cp * p[4]), p[5] * un])
    pn = _pressure(f, p, d)
    mom = [m * U[q] + pn[q] for q in range(3)]
    if f == "IG":
        return torch.stack([m, *mom, m * n2 + 5.0 * p[4] * un, m * (0.5 * n2 + cp * p[5]) + 2.5 * p[4] * un, p[6] * un])
    t = []
    for q, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
        t.append(m * U[a] * U[b] + un * p[4 + q] + U[a] * pn[b] + U[b] * pn[a])
    e = m * (0.5 * n2 + 0.5 * (p[4] + p[7] + p[9]) / (r + EPS) + cp * p[10]) + U[0] * pn[0] + U[1] * pn[1] + U[2] * pn[2]
    return torch.stack([m, *mom, *t, e, p[11] * un])


def _riemann(f, kind, a, b, d, cp):
    if kind == "Saurel":
        vn = 0.5 * (a[1 + d] + b[1 + d])
        p = torch.where(vn > 0, a, b)
        m = p[0] * vn
        n2 = p[1] ** 2 + p[2] ** 2 + p[3] ** 2
        return torch.stack([m, m * p[1], m * p[2], m * p[3], m * (0.5 * n2 + cp * p[4]), p[5] * vn])
    fa, fb, ca, cb = _flux(f, a, d, cp), _flux(f, b, d, cp), _conservative(f, a, cp), _conservative(f, b, cp)
    va, vb, sa, sb = a[1 + d], b[1 + d], _sound(f, a, d), _sound(f, b, d)
    if kind == "Rusanov":
        top = torch.stack([(va - sa).abs(), (vb - sb).abs(), (va + sa).abs(), (vb + sb).abs()]).amax(0)
        return 0.5 * (fa + fb - top * (cb - ca))
    ra, rb = a[0].sqrt(), b[0].sqrt()
    vr, sr = (ra * va + rb * vb) / (ra + rb), (ra * sa + rb * sb) / (ra + rb)
    z = torch.zeros_like(va)
    lo = torch.minimum(torch.minimum(z, va - sa), vr - sr)
    hi = torch.maximum(torch.maximum(z, vb + sb), vr + sr)
    mixed = (hi * fa - lo * fb + lo * hi * (cb - ca)) / (hi - lo)
    at = torch.stack([-lo, lo * hi, hi]).argmin(0)
    return torch.where(at == 0, fa, torch.where(at == 2, fb, mixed))


def _limited(limiter, x, y):
    r = y / (x + 1e-30)
    if limiter == "minmod":
        return torch.clamp(torch.clamp(r, max=1.0), min=0.0) * x
    if limiter == "vanleer":
        phi = (r + r.abs()) / (1.0 + r.abs())
    else:
        phi = torch.clamp(torch.minimum(torch.clamp(2.0 * r, max=2.0), 0.5 * (1.0 + r)), min=0.0)
    return torch.where(r > 0, torch.minimum(torch.clamp(phi, max=2.0), 2.0 * r), phi) * x


def _ghosts(f, p, axis, code):
    """p with two ghost layers on either side of the axis."""
    n = p.shape[axis]
    at = lambda q: p.narrow(axis, q, 1)
    if code in (101, 201):
        return torch.cat([p.narrow(axis, n - 2, 2), p, p.narrow(axis, 0, 2)], axis)
    if code == 0:
        return torch.cat([at(0)] * 2 + [p] + [at(n - 1)] * 2, axis)
    if code == 400:                  # a copy, then 3 g - 3 m + p = p
        return torch.cat([at(1), at(0), p, at(n - 1), at(n - 2)], axis)
    d = 3 - axis                     # a wall mirrors what moves away from it and lets the rest through
    layers = []
    for low, (m, q) in ((True, (0, 1)), (False, (n - 1, n - 2))):
        mirrored = (at(m)[1 + d] >= 0 if low else at(m)[1 + d] <= 0) | (low and d == 1)
        pair = []
        for cell in (at(m), at(q)):
            flip = cell.clone()
            for v in [1 + d] + ([t for t, ab in zip(range(4, 10), ("00", "01", "02", "11", "12", "22")) if
                                 (str(d) in ab and ab != 2 * str(d))] if f == "AG" else []):
                flip[v] = -flip[v]
            pair.append(torch.where(mirrored, flip, cell))
        layers.append(pair)
    return torch.cat([layers[0][1], layers[0][0], p, layers[1][0], layers[1][1]], axis)


def _kind(f, c):
    return c["riemann"] or ("Saurel" if f == "MK" else "Rusanov")


def _residual(f, c, p, h, cp, codes):
    """The sum of the face fluxes into every cell over its volume."""
    r0 = p[0:1]
    beta = None
    if c["sensor"]:
        sw = torch.zeros_like(p[0])
        for d in range(3):
            g = _ghosts(f, p, 3 - d, codes[d])[0]
            n = p.shape[3 - d]
            lo, hi = g.narrow(2 - d, 1, n), g.narrow(2 - d, 3, n)
            sw = torch.maximum(sw, ((hi - 2 * r0[0] + lo) / (hi + 2 * r0[0] + lo + 1e-30)).abs())
        phi = torch.clamp(sw * 20.0, min=0.0)
        beta = torch.where(sw < 0.05, 1.0 - torch.tanh(10.0 * phi ** 3), torch.zeros_like(sw))
    total = torch.zeros_like(p)
    for d in range(3):
        axis, n = 3 - d, p.shape[3 - d]
        if n < 2:
            continue
        g = _ghosts(f, p, axis, codes[d])
        diff = g.narrow(axis, 1, n + 3) - g.narrow(axis, 0, n + 3)
        back, fwd = diff.narrow(axis, 0, n + 2) / h, diff.narrow(axis, 1, n + 2) / h
        slope = _limited(c["limiter"], fwd, back) * (0.5 * h)
        rho = g[0]
        low = rho <= EMPTY
        first = low.narrow(axis - 1, 0, n + 2) | low.narrow(axis - 1, 1, n + 2) | low.narrow(axis - 1, 2, n + 2)
        ql, qr = g.narrow(axis, 1, n + 1), g.narrow(axis, 2, n + 1)
        sl, sr = slope.narrow(axis, 0, n + 1), slope.narrow(axis, 1, n + 1)
        fl, fr = first.narrow(axis - 1, 0, n + 1), first.narrow(axis - 1, 1, n + 1)
        if beta is None:
            weight = torch.ones_like(ql[0])
        else:
            e = beta.narrow(axis - 1, n - 1, 1), beta.narrow(axis - 1, 0, 1)
            if codes[d] != 201:
                e = e[1], e[0]
            wide = torch.cat([e[0], beta, e[1]], axis - 1)
            weight = torch.minimum(wide.narrow(axis - 1, 0, n + 1), wide.narrow(axis - 1, 1, n + 1))
        sl, sr = torch.where(fl, torch.zeros_like(sl), sl), torch.where(fr, torch.zeros_like(sr), sr)
        for _ in range(64):          # the weight halves until both states of the face are physical
            a, b = ql + sl * weight, qr - sr * weight
            bad = ~((fl | _physical(f, a)) & (fr | _physical(f, b)))
            if not bool(bad.any()):
                break
            weight = torch.where(bad, torch.where(0.5 * weight < 1e-18, torch.zeros_like(weight), 0.5 * weight), weight)
        F = _riemann(f, _kind(f, c), a, b, d, cp)
        total = total + (F.narrow(axis, 0, n) - F.narrow(axis, 1, n)) / h
    return total


def _evaporation(fam, c, gas, T, dp, Re, cpg, Pr):
    """The CEM mass rate with the Langmuir-Knudsen interface."""
    rho, Tg, R, k, mu = gas[0], gas[4], gas[5], gas[7], gas[8]
    pres, Mg, Ru = rho * R * Tg, 8314.46 / gas[5], 8314.46
    psat = 101325.0 * torch.exp(-fam.lv_al * fam.Mv / Ru * (1.0 / T - 1.0 / fam.Tboil))
    Xs = torch.where(psat >= pres, torch.full_like(T, 1.0 - 1e-12), torch.clamp(psat / pres, max=1.0 - 1e-12))
    mass = lambda X: X * fam.Mv / (X * fam.Mv + (1.0 - X) * Mg)
    Sc = Pr * fam.Le
    Dv = k / (rho * cpg * fam.Le)
    Sh = 2.0 + 0.6 * torch.sqrt(torch.clamp(Re, min=0.0)) * Sc ** (1.0 / 3.0)
    Yinf = fam.Yinf

    def rate(Y):
        B = (Y - Yinf) / (1.0 - Y)
        return torch.where((Y > Yinf) & (B > 0), -math.pi * dp * rho * Dv * Sh * torch.log1p(torch.clamp(B, min=0.0)),
                           torch.zeros_like(B))
    Ys = mass(Xs)
    dry = Ys <= Yinf
    md = rate(Ys)
    K = 2.0 * mu * torch.sqrt(2.0 * math.pi * T * Ru / fam.Mv) / (fam.alphaE * Sc * pres) / dp
    before = torch.full_like(md, math.inf)
    done = torch.zeros_like(dry)
    out = md
    for _ in range(30):
        new = rate(mass(torch.clamp(Xs - K * (-md * Pr / (2.0 * math.pi * mu * dp)), min=0.0)))
        off = (new - md).abs()
        out = torch.where(done, out, new)
        done = done | (off <= 1e-12 * new.abs())
        md = torch.where(off < before, new, 0.5 * (md + new))
        before = off
        if bool(done.all()):
            break
    return torch.where(dry, torch.zeros_like(out), out)


def _source(f, fam, c, p, gas):
    """The cell source of a family and its relaxation time."""
    T, n, r = p[-2], p[-1], p[0]
    R = (0.75 * r / (n * math.pi * fam.rho_al)) ** (1.0 / 3.0)
    F = [gas[1 + q] - p[1 + q] for q in range(3)]
    du = torch.sqrt(F[0] ** 2 + F[1] ** 2 + F[2] ** 2)
    Re = 2.0 * gas[0] * R * du / gas[8]
    cpg = gas[6] * gas[5] / (gas[6] - 1.0)
    Pr = cpg * gas[8] / gas[7]
    Nu = 2.0 + 0.6 * Re ** 0.5 * Pr ** (1.0 / 3.0)
    Cd = 24.0 / (Re + TOLL) * (1.0 + 0.15 * Re ** 0.687)
    Q = 2.0 * Nu * gas[7] * math.pi * R * (gas[4] - T)
    md = torch.zeros_like(r)
    if fam.evap != "none":
        md = _evaporation(fam, c, gas, T, 2.0 * R, Re, cpg, Pr)
    if c["evap"]:                    # Stefan blowing
        mp, dp = 4.0 / 3.0 * math.pi * R ** 3 * fam.rho_al, 2.0 * R
        b = -1.5 * Pr * (fam.rho_al * dp * dp / (18.0 * gas[8])) * md / mp
        b = torch.where((md < 0) & (mp > 0) & (b > 1e-10), b, torch.zeros_like(b))
        Q = Q * torch.where(b > 500.0, torch.zeros_like(b), torch.where(b > 0, b / torch.expm1(torch.clamp(b, 1e-10, 600.0)), torch.ones_like(b)))
    m = -md * n
    q = Q * n + fam.emiss * 5.670374419e-8 * 4.0 * math.pi * R * R * n * (gas[4] ** 4 - T ** 4)
    tau = 8.0 * fam.rho_al * R / (3.0 * gas[0] * Cd * du + TOLL)
    it = 1.0 / (tau + EPS)
    U = [p[1], p[2], p[3]]
    work_ = F[0] * U[0] + F[1] * U[1] + F[2] * U[2]
    n2 = U[0] ** 2 + U[1] ** 2 + U[2] ** 2
    s = [-m] + [-m * U[k] + r * F[k] * it for k in range(3)]
    heat = -m * fam.cs_al * T - m * fam.lv_al + q
    if f == "MK":
        s += [-m * 0.5 * n2 + heat + r * work_ * it]
    elif f == "IG":
        e = -m * (n2 + 3.0 * p[4] / r) + 2.0 * r * work_ * it - 6.0 * p[4] * it
        s += [e, heat + 0.5 * e]
    else:
        t = [-m * (U[a] * U[b] + p[4 + k] / r) + r * (F[b] * U[a] + F[a] * U[b]) * it - 2.0 * p[4 + k] * it
             for k, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)))]
        s += t + [heat + 0.5 * (t[0] + t[3] + t[5])]
    return torch.stack(s + [torch.zeros_like(r)]), tau


def exact(case, seed):
    """The interior states after the case's steps, by the step's formulas over the whole box in float64."""
    c = case
    h = _h(c)
    names, fams = c["families"].split("+"), _families(c)
    states, gas = _fields(c, seed)
    codes = [0 if n == 1 else c["bc"] for n in (c["nx"], c["ny"], c["nz"])]
    ndir = sum(n > 1 for n in (c["nx"], c["ny"], c["nz"]))
    weights = {"RK2": (1.0, 0.5), "RK3": (1.0, 0.25, 2.0 / 3.0), "euler": (1.0,)}[c["scheme"]]
    taus = [torch.full_like(p[0], math.inf) for p in states]
    for _ in range(c["steps"]):
        dts = []
        for f, p, tau in zip(names, states, taus):
            rate = sum(((p[1 + d].abs() + _sound(f, p, d)) / h for d in range(ndir)))
            dt = 0.5 * torch.where(rate > 0, torch.clamp(1.0 / rate, max=1e5), torch.full_like(rate, 1e5))
            dt = torch.clamp(dt, max=1.0)
            if c["gas"]:
                dt = torch.where((p[0] > EMPTY) & torch.isfinite(tau) & (tau > 0), torch.minimum(dt, tau), dt)
            dts.append(dt)
        if not c["steady"]:
            least = torch.stack([dt.min() for dt in dts]).min()
            dts = [least for _ in dts]
        for k, (f, fam) in enumerate(zip(names, fams)):
            cp, old = fam.cs_al, _conservative(f, states[k], fam.cs_al)
            p = states[k]
            for w in weights:
                R = _residual(f, c, p, h, cp, codes)
                if c["gas"]:
                    s, taus[k] = _source(f, fam, c, p, gas)
                    R = R + s
                new = old + (_conservative(f, p, cp) - old + R * dts[k]) * w
                p = _primitive(f, new, cp)
            states[k] = p
    states = [p.permute(1, 2, 3, 0).cpu().numpy() for p in states]
    return [[p[z0:z1, y0:y1, x0:x1] for p in states] for (x0, x1), (y0, y1), (z0, z1) in _spans(c)]
