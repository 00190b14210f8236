"""The measured work of the DEM library: what its users have it do, through the
public host classes (`mfix_dem.GpuSystem`, `mfix_dem.GpuBatch`).

A case is one running simulation (or one batch of them) and a pass over it is
what its driver asks for between two looks at the state: a number of
DES_TIME_STEPs and a download.  The inputs come from a seed alone and are made
here; the workloads follow the repository's own configurations
(`mfix_dem/configs.py`): settling columns, polydisperse Hertzian beds, the
homogeneously cooling gas, CFD-DEM coupling, batches of columns and hopper
discharges.  `exact` restates the contact, wall, drag and integration laws in
64-bit torch operations and follows the same steps.
"""
import math
import os
import sys

import numpy as np
import torch

# the package folder of the tree that runs this file (its root is the working folder)
sys.path.insert(0, os.path.join(os.getcwd(), "mfix-cfd-dem_b200"))

from mfix_dem import GpuBatch, GpuSystem, abi, load_library  # noqa: E402
from mfix_dem import params as P  # noqa: E402

PI = math.pi


# ---------------------------------------------------------------------------
# The cases

def listed():
    return [
        # The small dry run (the 4,000-sphere settling box that also runs on
        # a CPU): a step is a few microseconds of work, launches count.
        {"name": "settle_4k", "kind": "settle", "n": 4000, "steps": 500, "nsn": 25, "prec": "fp64", "intg": "EULER"},
        # An ordinary settled bed in a closed box, Adams-Bashforth, numbered
        # as a long-mixed system is: neighbours in memory are not neighbours
        # in space.
        {"name": "bed_mixed_150k", "kind": "bed", "n": 150001, "steps": 200, "nsn": 25, "prec": "fp64",
         "intg": "AB2", "order": "mixed", "walls": "box"},
        # The headline bed: a million polydisperse Hertzian spheres, most of
        # them in contact, periodic sides, plain FP64.
        {"name": "bed_1m_fp64", "kind": "bed", "n": 1000000, "steps": 200, "nsn": 25, "prec": "fp64",
         "intg": "EULER", "order": "cell", "walls": "floor"},
        # The same bed in split precision, the production form.
        {"name": "bed_1m_split", "kind": "bed", "n": 1000000, "steps": 200, "nsn": 25, "prec": "split",
         "intg": "EULER", "order": "cell", "walls": "floor"},
        # A granular gas, periodic on all sides: fast spheres, few contacts,
        # the neighbour search every few steps.
        {"name": "gas_200k", "kind": "gas", "n": 200003, "steps": 100, "nsn": 5, "prec": "fp64", "intg": "EULER"},
        # CFD-DEM with a frozen gas field: drag interpolated to the spheres
        # and the void fraction deposited back on every DEM step.
        {"name": "coupled_500k", "kind": "coupled", "n": 500000, "steps": 50, "nsn": 25, "scheme": "GARG_2012"},
        # One fluid step of a coupled driver: new gas fields in, a few DEM
        # sub-steps, the gas-side drag out (no interpolation, the default).
        {"name": "fluid_step_60k", "kind": "fluid_step", "n": 60007, "steps": 10, "nsn": 25, "scheme": "NONE"},
        # A batch of independent settled columns of uneven size.
        {"name": "columns_16", "kind": "columns", "n": 600000, "systems": 16, "steps": 400, "nsn": 25, "prec": "split"},
        # A few hopper cases as the server runs them together.
        {"name": "hoppers_5", "kind": "hoppers", "n": 160000, "systems": 5, "steps": 400, "nsn": 25, "prec": "split"},
        # A driver that keeps the DES arrays on the host: motion in, one
        # step, state out.
        {"name": "round_trip_250k", "kind": "round_trip", "n": 250000, "steps": 1, "nsn": 25, "prec": "fp64"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["settle", "bed", "bed", "gas", "coupled", "fluid_step", "columns", "hoppers", "round_trip"])
    prec = rng.choice(["fp64", "split"])
    intg = rng.choice(["EULER", "EULER", "AB2"])
    if kind == "settle":
        return {"kind": kind, "n": size(1500, 60000), "steps": 250, "nsn": rng.choice([10, 25]), "prec": prec,
                "intg": intg}
    if kind == "bed":
        return {"kind": kind, "n": size(30000, 900000), "steps": 200, "nsn": rng.choice([20, 25]), "prec": prec,
                "intg": intg, "order": rng.choice(["cell", "mixed"]), "walls": rng.choice(["box", "floor"])}
    if kind == "gas":
        return {"kind": kind, "n": size(20000, 300000), "steps": 100, "nsn": rng.choice([4, 5, 10]), "prec": prec,
                "intg": intg}
    if kind == "coupled":
        return {"kind": kind, "n": size(20000, 450000), "steps": 25, "nsn": 25,
                "scheme": rng.choice(["GARG_2012", "NONE"])}
    if kind == "fluid_step":
        return {"kind": kind, "n": size(10000, 120000), "steps": rng.randint(4, 20), "nsn": 25,
                "scheme": rng.choice(["GARG_2012", "NONE"])}
    if kind == "columns":
        return {"kind": kind, "n": size(60000, 600000), "systems": rng.randint(3, 16), "steps": 200, "nsn": 25,
                "prec": prec}
    if kind == "hoppers":
        return {"kind": kind, "n": size(40000, 160000), "systems": rng.randint(2, 6), "steps": 200, "nsn": 25,
                "prec": prec}
    return {"kind": kind, "n": size(20000, 250000), "steps": 1, "nsn": 25, "prec": prec}


# ---------------------------------------------------------------------------
# Inputs

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _packed_tile(rng, m=2048, phi=0.60):
    """m spheres with lognormal diameters (median 1 mm, sigma 0.25, 0.5-2 mm)
    at solids fraction phi in a periodic cube, overlaps pushed apart until
    they are a small part of a diameter.  Returns (positions, radii, edge)."""
    r = 0.5 * np.clip(1e-3 * np.exp(rng.normal(0.0, 0.25, m)), 0.5e-3, 2.0e-3)
    edge = float((np.sum(4.0 / 3.0 * PI * r ** 3) / phi) ** (1.0 / 3.0))
    x = torch.from_numpy(rng.uniform(0.0, edge, (m, 3))).to(_device())
    rt = torch.from_numpy(r).to(_device())
    reach = rt[:, None] + rt[None, :]
    reach.fill_diagonal_(0.0)
    for _ in range(240):
        d = [x[:, a, None] - x[None, :, a] for a in range(3)]
        d = [c - edge * torch.round(c / edge) for c in d]
        dist = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).clamp_min(1e-12)
        push = 0.45 * (reach - dist).clamp_min(0.0) / dist
        x = x + torch.stack([(push * c).sum(1) for c in d], 1)
        x = x - edge * torch.floor(x / edge)
    return x.cpu().numpy(), r, edge


def _lattice(rng, nx, ny, nz, a, jitter):
    kk, ii, jj = np.meshgrid(np.arange(nz), np.arange(nx), np.arange(ny), indexing="ij")
    x = np.stack([(ii.ravel() + 0.5) * a, (jj.ravel() + 0.5) * a, (kk.ravel() + 0.5) * a], 1)
    return x + rng.uniform(-jitter, jitter, x.shape)


def _cell_order(pos, width):
    """Numbering by cells of `width`, y fastest: spatial neighbours lie close."""
    g = np.floor((pos - pos.min(0)) / width).astype(np.int64)
    g1, g2 = g[:, 1].max() + 1, g[:, 0].max() + 1
    return np.argsort((g[:, 2] * g2 + g[:, 0]) * g1 + g[:, 1], kind="stable")


def _box_facets(lo, hi, periodic=(False, False, False)):
    """A large triangle per wall of the box, normals inward: (F,3 vertices,3), (F,3)."""
    lo, hi = np.asarray(lo, float), np.asarray(hi, float)
    tri, nrm = [], []
    for ax in range(3):
        if periodic[ax]:
            continue
        b, c = [a for a in range(3) if a != ax]
        for side in range(2):
            v = np.zeros((3, 3))
            v[:, :] = lo
            v[:, ax] = (lo, hi)[side][ax]
            v[1, b] += 2.0 * (hi[b] - lo[b])
            v[2, c] += 2.0 * (hi[c] - lo[c])
            tri.append(v)
            n = np.zeros(3)
            n[ax] = 1.0 if side == 0 else -1.0
            nrm.append(n)
    return np.array(tri), np.array(nrm)


def _hopper_facets(box, y_out, r_out, half_angle, seg=64):
    """Box sides and top, and a cone from the outlet up to the circle inscribed
    in the box."""
    lo = np.zeros(3)
    hi = np.asarray(box, float)
    tri, nrm = _box_facets(lo, hi)
    keep = [f for f in range(6) if f != 2]          # no floor
    tri, nrm = [tri[f] for f in keep], [nrm[f] for f in keep]
    c = 0.5 * hi
    rim, t = min(c[0], c[2]), math.tan(half_angle)
    y_top = y_out + (rim - r_out) / t

    def at(k, r, y):
        return np.array([c[0] + r * math.cos(2 * PI * k / seg), y, c[2] + r * math.sin(2 * PI * k / seg)])

    for k in range(seg):
        b0, b1, t0, t1 = at(k, r_out, y_out), at(k + 1, r_out, y_out), at(k, rim, y_top), at(k + 1, rim, y_top)
        for v in ((b0, b1, t1), (b0, t1, t0)):
            n = np.cross(v[1] - v[0], v[2] - v[0])
            n = n / np.linalg.norm(n)
            tri.append(np.array(v))
            nrm.append(n if n[1] > 0.0 else -n)
    return np.array(tri), np.array(nrm), y_top


def _system(pos, vel, radius, rho, order, rng, spin=0.0, **kw):
    """One system's arrays, numbered as asked, with its keywords; spins are
    normal with a deviation of `spin` rad/s."""
    omega = rng.normal(0.0, spin, pos.shape) if spin > 0.0 else np.zeros(pos.shape)
    if order == "mixed":
        perm = rng.permutation(len(pos))
    elif order == "cell":
        perm = _cell_order(pos, 6.0 * radius.max())
    else:
        perm = np.arange(len(pos))
    return dict(pos=pos[perm], vel=vel[perm], omega=omega[perm], radius=radius[perm], rho=rho, **kw)


HERTZ = dict(coll="HERTZ", en=0.85, mew=0.3, mew_r=0.01)


def _bed(case, rng, n):
    """The lowest n spheres of a stack of packed tiles, at rest but for small
    motions, on a floor with periodic sides or in a box."""
    x0, r0, edge = _packed_tile(rng)
    m = len(r0)
    k = max(2, int(round((n / m / 2.0) ** (1.0 / 3.0))))
    ky = -(-n // (m * k * k)) + 1
    shift = np.stack(np.meshgrid(np.arange(k), np.arange(ky), np.arange(k), indexing="ij"), -1).reshape(-1, 3)
    pos = (x0[None] + edge * shift[:, None]).reshape(-1, 3)
    radius = np.tile(r0, len(shift))
    low = np.argsort(pos[:, 1], kind="stable")[:n]
    pos, radius = pos[low], radius[low]
    pos = pos + rng.uniform(-1e-6, 1e-6, pos.shape)
    vel = rng.normal(0.0, 0.02, pos.shape)
    rmax = radius.max()
    pos[:, 1] -= np.min(pos[:, 1] - radius)
    side, height = k * edge, float(pos[:, 1].max()) + 12.0 * rmax
    if case.get("walls", "floor") == "floor":
        pos[:, 0] %= side
        pos[:, 2] %= side
        lo, hi, per = (0.0, 0.0, 0.0), (side, height, side), (True, False, True)
    else:
        lo, hi, per = (-rmax, 0.0, -rmax), (side + rmax, height, side + rmax), (False, False, False)
    return _system(pos, vel, radius, 2500.0, case.get("order", "cell"), rng, lo=lo, hi=hi, per=per,
                   facets=_box_facets(lo, hi, per), spin=20.0, **HERTZ)


def _settle(case, rng, n, kn=1000.0, mew=0.1, spacing=1.1, jitter=0.04, vmax=0.1, cols=10):
    """Monodisperse 1 mm spheres on a jittered lattice in a closed column."""
    d = 1e-3
    ny = -(-n // (cols * cols))
    width = (cols + 2) * d
    pos = _lattice(rng, cols, ny, cols, spacing * d, jitter * d)
    pos = pos[np.argsort(pos[:, 1], kind="stable")[:n]]
    pos[:, [0, 2]] += 0.5 * (width - cols * spacing * d)
    hi = (width, max(1.5 * ny, 12.0) * d, width)
    vel = rng.uniform(-vmax, vmax, pos.shape)
    return _system(pos, vel, np.full(len(pos), 0.5 * d), 2500.0, "cell", rng, lo=(0.0, 0.0, 0.0), hi=hi,
                   per=(False, False, False), facets=_box_facets((0, 0, 0), hi), coll="LSD", kn=kn, en=0.9, mew=mew,
                   mew_r=0.0)


def _gas(case, rng, n):
    """Nearly elastic 1 mm spheres at 18 % solids in a periodic cube."""
    d = 1e-3
    k = int(math.ceil(n ** (1.0 / 3.0)))
    a = 1.425 * d
    pos = _lattice(rng, k, k, k, a, 0.2 * d)
    pos = pos[np.sort(rng.permutation(len(pos))[:n])]
    vel = rng.normal(0.0, 0.4, pos.shape)
    vel -= vel.mean(0)
    side = k * a
    pos %= side
    return _system(pos, vel, np.full(n, 0.5 * d), 2500.0, "cell", rng, lo=(0.0, 0.0, 0.0), hi=(side,) * 3,
                   per=(True, True, True), facets=(np.zeros((0, 3, 3)), np.zeros((0, 3))), coll="LSD", kn=1000.0,
                   en=0.97, mew=0.1, mew_r=0.0, grav=(0.0, 0.0, 0.0))


def _fluidized(case, rng, n):
    """0.5 mm spheres in the lower part of a fluid grid of 1 mm cells."""
    d, dx = 0.5e-3, 1e-3
    cx = max(12, int(round((n / 55.0) ** (1.0 / 3.0) * 3.0)))
    a = 1.06 * d
    m = int(cx * dx / a)
    ny = -(-n // (m * m))
    cy = max(24, int(5 * ny * a / dx))
    pos = _lattice(rng, m, ny, m, a, 0.04 * d)
    pos = pos[np.argsort(pos[:, 1], kind="stable")[:n]]
    pos[:, [0, 2]] += 0.5 * (cx * dx - m * a)
    vel = rng.normal(0.0, 0.05, pos.shape)
    hi = (cx * dx, cy * dx, cx * dx)
    s = _system(pos, vel, np.full(len(pos), 0.5 * d), 2600.0, "cell", rng, lo=(0.0, 0.0, 0.0), hi=hi,
                per=(False, False, False), facets=_box_facets((0, 0, 0), hi), coll="LSD", kn=500.0, en=0.9, mew=0.1,
                mew_r=0.0, cells=(cx, cy, cx), dx=dx)
    g = (cx + 2, cy + 2, cx + 2)

    def noise(std):   # smooth over a few cells: coarse values interpolated
        c = torch.from_numpy(rng.normal(0.0, std, [1, 1] + [max(2, v // 4) for v in g[::-1]]))
        return torch.nn.functional.interpolate(c, size=g[::-1], mode="trilinear", align_corners=True)[0, 0].numpy()

    vs = np.zeros(g[::-1])
    c = [np.clip((pos[:, k] / dx).astype(int) + 1, 1, s["cells"][k]) for k in range(3)]
    np.add.at(vs, (c[2], c[1], c[0]), PI / 6.0 * d ** 3)
    ep = np.maximum(1.0 - vs / dx ** 3, 0.35)
    s["gas"] = dict(ep=ep.ravel().copy(), u=(noise(0.1) / ep).ravel(), v=((1.0 + noise(0.1)) / ep).ravel(),
                    w=(noise(0.1) / ep).ravel(), ro=1.2, mu=1.8e-5)
    return s


def _counts(case, least, weights):
    """The sizes of a batch's systems: a draw of their own for each case."""
    w = weights(np.random.default_rng([case["n"], case["systems"]]), case["systems"])
    return np.maximum((case["n"] * w / w.sum()).astype(int), least)


def _columns(case, rng):
    counts = _counts(case, 1000, lambda g, k: np.exp(g.normal(0.0, 0.9, k)))
    return [_settle(case, rng, int(c), kn=float(rng.uniform(200.0, 2000.0)), mew=float(rng.uniform(0.1, 0.5)),
                    spacing=1.0, jitter=0.015, vmax=0.02) for c in counts]


def _hoppers(case, rng):
    """2 mm spheres filling a cone (half-angle 30 degrees) and the box over
    it, the outlet 6-10 diameters wide."""
    d, angle = 2e-3, math.radians(30.0)
    out = []
    for c in _counts(case, 3000, lambda g, k: np.exp(g.uniform(math.log(0.1), 0.0, k))):
        box = (0.12, 0.13 + float(c) * d ** 3 / (PI * 0.058 ** 2), 0.12)
        r_out = 0.5 * d * int(rng.integers(6, 11))
        y_out = 0.012
        tri, nrm, y_top = _hopper_facets(box, y_out, r_out, angle)
        m = int(box[0] / d)
        pos = _lattice(rng, m, int((box[1] - y_out) / d), m, d, 0.015 * d)
        pos[:, 1] += y_out + 0.6 * d
        pos[:, [0, 2]] += 0.5 * (box[0] - m * d)
        rr = np.hypot(pos[:, 0] - 0.06, pos[:, 2] - 0.06)
        # above the cone by the sphere's radius less a slight overlap, within the walls
        wall = (pos[:, 1] - y_out) * math.sin(angle) + (r_out - rr) * math.cos(angle)
        ok = (wall > 0.499 * d) & (rr < 0.06 - 0.52 * d)
        pos = pos[ok]
        pos = pos[np.argsort(pos[:, 1], kind="stable")[:c]]
        vel = rng.normal(0.0, 0.01, pos.shape)
        h = dict(HERTZ, mew=float(rng.uniform(0.2, 0.6)), mew_r=0.0)
        out.append(_system(pos, vel, np.full(len(pos), 0.5 * d), 2500.0, "cell", rng, lo=(0.0, 0.0, 0.0), hi=box,
                           per=(False, False, False), facets=(tri, nrm), **h))
    return out


def _inputs(case, seed):
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, case["n"]])
    kind = case["kind"]
    if kind == "settle":
        return [_settle(case, rng, case["n"])]
    if kind in ("bed", "round_trip"):
        return [_bed(case, rng, case["n"])]
    if kind == "gas":
        return [_gas(case, rng, case["n"])]
    if kind in ("coupled", "fluid_step"):
        return [_fluidized(case, rng, case["n"])]
    return _columns(case, rng) if kind == "columns" else _hoppers(case, rng)


# ---------------------------------------------------------------------------
# The framework's side

def _keywords(case, s):
    k = dict(d_p0=(2.0 * float(s["radius"].max()),), ro_s0=(s["rho"],), coll_model=s["coll"],
             intg_method="ADAMS_BASHFORTH" if case.get("intg") == "AB2" else "EULER",
             des_en_input=s["en"], des_en_wall_input=[s["en"]], mew=s["mew"], mew_w=s["mew"], mew_r=s["mew_r"],
             mew_rw=s["mew_r"], grav=s.get("grav", (0.0, -9.81, 0.0)), domain_lo=s["lo"], domain_hi=s["hi"],
             fluid_cells=s.get("cells", (1, 1, 1)), periodic=s["per"], neighbor_search_n=case["nsn"],
             force_precision=abi.DEM_PREC_SPLIT if case.get("prec") == "split" else abi.DEM_PREC_FP64)
    if s["coll"] == "LSD":
        k.update(kn=s["kn"], kn_w=s["kn"])
    else:
        k.update(des_et_input=s["en"], des_et_wall_input=[s["en"]], e_young=(1e7,), v_poisson=(0.3,), ew_young=1e7,
                 vw_poisson=0.3)
    return P.DemCase(**k)


def _arrays(s):
    n = len(s["radius"])
    _, mass, omoi = P.particle_props(s["radius"], np.full(n, s["rho"]))
    return dict(**{k: np.ascontiguousarray(s[k].T) for k in ("pos", "vel", "omega")}, radius=s["radius"], pmass=mass,
                omoi=omoi, state=np.full(n, abi.DEM_STATE_NORMAL, np.int8), phase=np.ones(n, np.int32))


def _set_up(case, s):
    arr = _arrays(s)
    prm, _ = P.build_params(_keywords(case, s), arr["radius"], arr["pmass"], arr["phase"], arr["state"])
    tri, nrm = s["facets"]
    return prm, arr, (np.ascontiguousarray(tri.transpose(0, 2, 1)), nrm)   # VERTEX is [facet][component][vertex]


def _pinned(n):
    """Host arrays for the state in page-locked memory, as a driver that
    exchanges it often keeps them."""
    f = {k: torch.empty((3, n), dtype=torch.float64, pin_memory=True).numpy() for k in ("pos", "vel", "omega")}
    f["state"] = torch.empty(n, dtype=torch.int8, pin_memory=True).numpy()
    return f


def _grid(case, s):
    g = abi.DemFluidGrid()
    g.imax, g.jmax, g.kmax = s["cells"]
    g.drag_model = 0
    g.interp_scheme = abi.DEM_INTERP_GARG if case["scheme"] == "GARG_2012" else abi.DEM_INTERP_NONE
    g.dx = g.dy = g.dz = s["dx"]
    g.ro_g, g.mu_g, g.ep_star, g.ur_f_gs = s["gas"]["ro"], s["gas"]["mu"], 0.42, 1.0
    g.ro_s[0] = s["rho"]
    return g


def prepare(case, seed):
    """A simulation that runs: state and walls uploaded, the first neighbour
    period (and with it the first search) behind it."""
    torch.zeros(1, device="cuda")
    systems = _inputs(case, seed)
    if case["kind"] in ("columns", "hoppers"):
        sets = [_set_up(case, s) for s in systems]
        lim = P.batch_limits(load_library(), [(prm, len(a["radius"]), len(w[0])) for prm, a, w in sets],
                             bins_per_cell=24)
        b = GpuBatch(sets[0][0], lim)
        ids = []
        for prm, a, w in sets:
            sid = b.add(prm, len(a["radius"]))
            b.set_walls(sid, *w)
            b.upload_state(sid, **a)
            ids.append(sid)
        b.start(ids)
        b.step(case["nsn"])
        return {"kind": case["kind"], "steps": case["steps"], "batch": b, "ids": ids}
    s = systems[0]
    prm, a, w = _set_up(case, s)
    d = GpuSystem(prm, len(a["radius"]))
    d.set_walls(*w)
    d.upload_state(**a)
    d.init_neighbors()
    st = {"kind": case["kind"], "steps": case["steps"], "sys": d, "out": _pinned(d.n)}
    if "gas" in s:
        g = s["gas"]
        st.update(grid=_grid(case, s), gas=(g["ep"], g["u"], g["v"], g["w"]), scheme=case["scheme"])
        d.set_gas_fields(st["grid"], *st["gas"])
        d.step_coupled(case["nsn"])
    else:
        d.step(case["nsn"])
    if case["kind"] == "round_trip":
        d.download_state(st["out"])
    return st


def run(state):
    kind = state["kind"]
    if kind in ("columns", "hoppers"):
        b = state["batch"]
        b.step(state["steps"])
        return [b.download_state(i) for i in state["ids"]]
    d = state["sys"]
    if kind == "round_trip":
        o = state["out"]
        d.upload_state(o["pos"], o["vel"], o["omega"])
        d.step(state["steps"])
        return d.download_state(o)
    if kind == "coupled":
        d.step_coupled(state["steps"])
        ep, rop = d.get_mean_fields()
        return dict(d.download_state(state["out"]), ep_g=ep, rop_s=rop)
    if kind == "fluid_step":
        d.set_gas_fields(state["grid"], *state["gas"])
        d.step_coupled(state["steps"])
        if state["scheme"] == "NONE":
            f_gds, bm, f_gp = d.drag_gs_gas1()
            gas = dict(f_gds=f_gds, drag_bm=bm, f_gp=f_gp)
        else:
            f_gds, am, bm, f_gp = d.drag_gs_gas0()
            gas = dict(f_gds=f_gds, drag_am=am, drag_bm=bm, f_gp=f_gp)
        return dict(d.download_state(state["out"]), **gas)
    d.step(state["steps"])
    return d.download_state(state["out"])


# contacts per particle of each kind, for the work a pass cannot do without
CONTACTS = {"settle": 0.1, "bed": 2.2, "round_trip": 2.2, "gas": 0.05, "coupled": 0.4, "fluid_step": 0.4,
            "columns": 1.4, "hoppers": 1.4}


def work(case):
    """Per step: positions and velocities (with radius and mass) read and
    written, spins of the spheres in contact read and written, the tangential
    history of each contact read and written, its partner's index read; then
    the state copied out.  Coupled: the gas fields of the cells with spheres
    once a step."""
    n, c = case["n"], CONTACTS[case["kind"]]
    step = n * (64 + 48) + n * min(1.0, 2.0 * c) * 56 + n * c * 52
    flops = n * (40 + 250 * c)
    once = n * 73
    if case["kind"] == "round_trip":
        once += n * 72
    if case["kind"] in ("coupled", "fluid_step"):
        step += n * 8 * (1 + 4.0 / 6.0)
        flops += n * 250
        once += n / 6.0 * 8 * (2 if case["kind"] == "coupled" else 8)
    return {"bytes": float(case["steps"] * step + once), "flops": float(case["steps"] * flops)}


# ---------------------------------------------------------------------------
# The same steps in 64-bit torch operations

def _constants(case, s):
    """The contact tables and the solids time step of one phase."""
    r, rho, e = float(s["radius"].min()), s["rho"], s["en"]
    m = min((PI / 6.0) * (2.0 * float(s["radius"].max())) ** 3 * rho, 4.0 / 3.0 * PI * r * (r * r) * rho)
    beta = abs(math.log(e)) / math.sqrt(PI * PI + math.log(e) ** 2)
    c = {}
    if s["coll"] == "LSD":
        third = float(np.float32(0.28571428571429))
        c.update(kn=s["kn"], kt=third * s["kn"], etan=2.0 * math.sqrt(s["kn"]) * beta)
        c["etat"] = 0.5 * c["etan"]
        c.update(kn_w=c["kn"], kt_w=c["kt"], etan_w=c["etan"], etat_w=c["etat"])
        k_m = s["kn"] / (0.5 * m)
    else:
        E, nu = 1e7, 0.3
        G = 0.5 * E / (1.0 + nu)
        eeff = E * E / (2.0 * E * (1.0 - nu * nu))
        geff = G * G / (2.0 * G * (2.0 - nu))
        c.update(kn=4.0 / 3.0 * eeff, kt=8.0 * geff, etan=math.sqrt(5.0) * beta,
                 etat=math.sqrt(5.0) * math.sqrt(2.0 / 7.0) * beta)
        c.update(kn_w=c["kn"], kt_w=c["kt"], etan_w=c["etan"], etat_w=c["etat"])
        k_m = c["kn"] * math.sqrt(0.5 * r) / (0.5 * m)
    c["dt"] = PI / math.sqrt(k_m * (1.0 - beta * beta)) / 50.0
    return c


def _dot(a, b):
    return (a * b).sum(-1)


def _pairs(x, r, s):
    """MFiX's neighbour list: pairs i < j within FACTOR_RLM (r_i + r_j) of the
    nearest image, j in one of the search cells that i looks at (of cells
    wider than the search diameter the nearer two on each axis)."""
    dev, n = x.device, len(r)
    lo = torch.tensor(s["lo"], dtype=torch.float64, device=dev)
    L = torch.tensor(s["hi"], dtype=torch.float64, device=dev) - lo
    per = torch.tensor(s["per"], device=dev)
    width = 2.4 * float(r.max()) * 1.0001
    dims = torch.clamp((L / width).floor(), min=1.0)
    g = ((x - lo) / L * dims).floor()
    g = torch.where(per, g % dims, g.clamp_min(0.0).minimum(dims - 1)).long()
    d = dims.long()
    cell = (g[:, 0] * d[1] + g[:, 1]) * d[2] + g[:, 2]
    order = torch.argsort(cell, stable=True)
    ncell = int(d.prod())
    count = torch.bincount(cell, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    got = []
    span = [range(-1, 2) if int(d[a]) >= 3 or not s["per"][a] else range(0, 1) for a in range(3)]
    me = torch.arange(n, device=dev)
    # the search cells: three largest diameters wide, no wider than a fluid cell
    factor, dgn = float(np.float32(1.2)), []
    for ax in range(3):
        length = s["hi"][ax] - s["lo"][ax]
        dgn.append(max(int(length / min(6.0 * float(r.max()), length / s.get("cells", (1, 1, 1))[ax])), 1))
    q = (x - lo) * (torch.tensor(dgn, dtype=torch.float64, device=dev) / L)
    dg, off = q.floor().long(), q - q.floor()
    wide = torch.tensor([1.0 > 2.0 * float(r.max()) * factor * dgn[a] / (s["hi"][a] - s["lo"][a]) for a in range(3)],
                        device=dev)
    lo_off, hi_off = 1 - (wide & (off >= 0.5)).long(), 1 - (wide & (off < 0.5)).long()
    for o0 in span[0]:
        for o1 in span[1]:
            for o2 in span[2]:
                h = g + torch.tensor([o0, o1, o2], device=dev)
                inside = ((h >= 0) & (h < d) | per).all(1)
                h = torch.where(per, h % d, h.clamp_min(0).minimum(d - 1))
                c = (h[:, 0] * d[1] + h[:, 1]) * d[2] + h[:, 2]
                k = torch.where(inside, count[c], torch.zeros_like(c))
                i = torch.repeat_interleave(me, k)
                first = torch.cumsum(k, 0) - k
                j = order[start[c][i] + torch.arange(len(i), device=dev) - first[i]]
                near = i < j
                i, j = i[near], j[near]
                e = x[j] - x[i]
                e = torch.where(per, e - L * torch.round(e / L), e)
                near = _dot(e, e) <= (factor * (r[i] + r[j])) ** 2
                for ax in range(3):
                    rel = dg[j, ax] - dg[i, ax]
                    if s["per"][ax]:
                        rel = (rel + dgn[ax] // 2) % dgn[ax] - dgn[ax] // 2
                    near &= (rel >= -lo_off[i, ax]) & (rel <= hi_off[i, ax])
                got.append(i[near] * n + j[near])
    return torch.sort(torch.cat(got))[0]


def _tangential(c, kt, etat, fn, vt, hist, mew, dt):
    """Spring-dashpot tangential force with the Coulomb limit, and the history."""
    ot = dt * vt + hist
    mag = torch.sqrt(_dot(ot, ot))
    ft = -kt * ot - etat * vt
    limit = mew * torch.sqrt(_dot(fn, fn))
    slip = torch.sqrt(_dot(ft, ft)) > limit
    tg = ot / mag.clamp_min(1e-300)[:, None]
    ft = torch.where(slip[:, None], -limit[:, None] * tg, ft)
    ot = torch.where(slip[:, None], (limit[:, None] / kt) * tg, ot)
    return torch.where((mag > 0.0)[:, None], ft, torch.zeros_like(ft)), ot


def _facet_data(tri, nrm, dev):
    """The facets and, per facet, whether its vertex/edge contacts on each of
    its three edges are left to a nearly coplanar neighbour."""
    F = len(tri)
    ignore = np.zeros((F, 4), bool)
    mid = np.stack([0.5 * (tri[:, 0] + tri[:, 1]), 0.5 * (tri[:, 0] + tri[:, 2]), 0.5 * (tri[:, 1] + tri[:, 2])], 1) \
        if F else np.zeros((0, 3, 3))
    flat = nrm @ nrm.T > math.cos(5.0 / 180.0 * PI) + 1e-6
    np.fill_diagonal(flat, False)
    for a in range(3):
        for b in range(3):
            d = mid[:, None, a] - mid[None, :, b]
            ignore[:, a + 1] |= (((d * d).sum(-1) < 1e-9) & flat).any(1)
    return torch.from_numpy(tri).to(dev), torch.from_numpy(ignore).to(dev)


def _closest(T, x):
    """Closest point of triangles T (k,3,3) to points x (k,3), and the edge
    (1: vertices 1-2, 2: 1-3, 3: 2-3) it lies on, 0 inside."""
    a, b, c = T[:, 0], T[:, 1], T[:, 2]
    ab, ac = b - a, c - a
    ap, bp, cp = x - a, x - b, x - c
    d1, d2, d3, d4, d5, d6 = (_dot(ab, ap), _dot(ac, ap), _dot(ab, bp), _dot(ac, bp), _dot(ab, cp), _dot(ac, cp))
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    den = 1.0 / (va + vb + vc)
    q = a + ab * (vb * den)[:, None] + ac * (vc * den)[:, None]
    edge = torch.zeros(len(x), dtype=torch.long, device=x.device)
    bc = (d4 - d3) / ((d4 - d3) + (d5 - d6))
    for cond, pt, e in (((va < 0) & (d4 - d3 > 0) & (d5 - d6 > 0), b + bc[:, None] * (c - b), 3),
                        ((vb < 0) & (d2 > 0) & (d6 < 0), a + (d2 / (d2 - d6))[:, None] * ac, 2),
                        ((d6 > 0) & (d5 < d6), c, 2),
                        ((vc < 0) & (d1 > 0) & (d3 < 0), a + (d1 / (d1 - d3))[:, None] * ab, 1),
                        ((d3 > 0) & (d4 < d3), b, 1),
                        ((d1 < 0) & (d2 < 0), a, 1)):
        q = torch.where(cond[:, None], pt, q)
        edge = torch.where(cond, torch.full_like(edge, e), edge)
    return q, edge


class _Exact:
    """One system followed in 64 bits."""

    def __init__(self, case, s):
        dev = _device()
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.case, self.s, self.c, self.dev = case, s, _constants(case, s), dev
        self.hertz, self.ab2 = s["coll"] == "HERTZ", case.get("intg") == "AB2"
        self.x, self.v, self.r = t(s["pos"]), t(s["vel"]), t(s["radius"])
        self.w = t(s["omega"])
        self.m = (4.0 / 3.0) * PI * self.r ** 3 * s["rho"]
        self.omoi = 2.5 / (self.m * self.r * self.r)
        self.n = len(self.r)
        self.g = torch.tensor(s.get("grav", (0.0, -9.81, 0.0)), dtype=torch.float64, device=dev)
        self.L = torch.tensor(s["hi"], dtype=torch.float64, device=dev) - torch.tensor(s["lo"], dtype=torch.float64,
                                                                                       device=dev)
        self.per = torch.tensor(s["per"], device=dev)
        self.tri, self.ignore = _facet_data(*s["facets"], dev)
        self.wall_key = torch.zeros(0, dtype=torch.long, device=dev)
        self.wall_hist = torch.zeros((0, 3), dtype=torch.float64, device=dev)
        self.key = torch.zeros(0, dtype=torch.long, device=dev)
        self.hist = torch.zeros((0, 3), dtype=torch.float64, device=dev)
        self.age, self.due, self.old = 0, 0, None

    @staticmethod
    def _carry(key, old_key, old_hist):
        hist = torch.zeros((len(key), 3), dtype=torch.float64, device=key.device)
        if len(old_key) and len(key):
            at = torch.searchsorted(old_key, key).clamp_max(len(old_key) - 1)
            hist = torch.where((old_key[at] == key)[:, None], old_hist[at], hist)
        return hist

    def _stiffness(self, ov, reff, meff, wall=""):
        c = self.c
        kn, kt, en, et = c["kn" + wall], c["kt" + wall], c["etan" + wall], c["etat" + wall]
        if not self.hertz:
            o = torch.ones_like(ov)
            q = torch.sqrt(meff)
            return kn * o, kt * o, en * q, et * q
        so, sr = torch.sqrt(ov), torch.sqrt(reff)
        q = torch.sqrt(so)
        return kn * so * sr, kt * so * sr, en * q * torch.sqrt(kn * sr * meff), et * q * torch.sqrt(kt * sr * meff)

    def forces(self):
        s, c = self.s, self.c
        x, v, w, r = self.x, self.v, self.w, self.r
        f, t = torch.zeros_like(x), torch.zeros_like(x)
        om = torch.sqrt(_dot(w, w))
        # walls
        for_key, for_hist = [], []
        for k in range(0, len(self.tri), 16):
            T = self.tri[k:k + 16]
            lo, hi = T.amin(1), T.amax(1)
            near = ((x[:, None] + r[:, None, None] >= lo) & (x[:, None] - r[:, None, None] <= hi)).all(-1)
            i, q = torch.nonzero(near, as_tuple=True)
            pt, edge = _closest(T[q], x[i])
            d = pt - x[i]
            d2 = _dot(d, d)
            hit = (d2 < r[i] * r[i] - 1e-15) & ~((edge > 0) & self.ignore[k + q, edge])
            i, q, d, dm = i[hit], q[hit] + k, d[hit], torch.sqrt(d2[hit])
            nr, ov = d / dm[:, None], r[i] - dm
            vr = v[i] + dm[:, None] * torch.linalg.cross(w[i], nr)
            vn = _dot(vr, nr)
            kn, kt, en, et = self._stiffness(ov, r[i], self.m[i], "_w")
            fn = -(kn * ov + en * vn)[:, None] * nr
            key = i * 4096 + q
            hist = self._carry(key, self.wall_key, self.wall_hist)
            ft, ot = _tangential(c, kt[:, None], et[:, None], fn, vr - vn[:, None] * nr, hist, s["mew"], c["dt"])
            f.index_add_(0, i, fn + ft)
            tq = dm[:, None] * torch.linalg.cross(nr, ft)
            if s["mew_r"] > 0.0:
                tq = tq - torch.where((om[i] > 0)[:, None], (s["mew_r"] * 2.0 * r[i] * kn * ov / om[i].clamp_min(
                    1e-300))[:, None] * w[i], torch.zeros_like(tq))
            t.index_add_(0, i, tq)
            for_key.append(key)
            for_hist.append(ot)
        if for_key:
            key, at = torch.sort(torch.cat(for_key))
            self.wall_key, self.wall_hist = key, torch.cat(for_hist)[at]
        # pairs
        if self.age == self.due:
            self.list = _pairs(x, r, s)
            # searches: at the start, after the first step, then every NEIGHBOR_SEARCH_N
            self.due = 1 if self.age == 0 else (self.age // self.case["nsn"] + 1) * self.case["nsn"]
        self.age += 1
        i, j = self.list // self.n, self.list % self.n
        d = x[j] - x[i]
        d = torch.where(self.per, d - self.L * torch.round(d / self.L), d)
        d2 = _dot(d, d)
        hit = d2 <= (r[i] + r[j] - 1e-15) ** 2
        key = self.list[hit]
        i, j, d, dm = i[hit], j[hit], d[hit], torch.sqrt(d2[hit])
        hist = self._carry(key, self.key, self.hist)
        nr, ov = d / dm[:, None], r[i] + r[j] - dm
        arm = (dm * dm + r[i] ** 2 - r[j] ** 2) / (2.0 * dm)
        arm2 = dm - arm
        vr = v[i] - v[j] + torch.linalg.cross(w[i] * arm[:, None] + w[j] * arm2[:, None], nr)
        vn = _dot(vr, nr)
        kn, kt, en, et = self._stiffness(ov, r[i] * r[j] / (r[i] + r[j]), self.m[i] * self.m[j] / (self.m[i] +
                                                                                               self.m[j]))
        fn = -(kn * ov + en * vn)[:, None] * nr
        ft, ot = _tangential(c, kt[:, None], et[:, None], fn, vr - vn[:, None] * nr, hist, s["mew"], c["dt"])
        self.key, self.hist = key, ot
        f.index_add_(0, i, fn + ft)
        f.index_add_(0, j, -(fn + ft))
        tq = torch.linalg.cross(nr, ft)
        for k, a in ((i, arm), (j, arm2)):
            u = a[:, None] * tq
            if s["mew_r"] > 0.0:
                u = u - torch.where((om[k] > 0)[:, None], (s["mew_r"] * 2.0 * r[k] * kn * ov / om[k].clamp_min(
                    1e-300))[:, None] * w[k], torch.zeros_like(u))
            t.index_add_(0, k, u)
        return f, t

    def step(self, steps=1):
        for _ in range(steps):
            f, t = self.forces()
            if "gas" in self.s:
                f = f + self.drag()
            self.integrate(f, t)
            if "gas" in self.s:
                self.mean_fields()

    def integrate(self, f, t):
        dt = self.c["dt"]
        a = f / self.m[:, None] + self.g
        u = t * self.omoi[:, None]
        if self.ab2:
            # the first step takes the torque itself for the old spin rate
            ao, uo = (a, t) if self.old is None else self.old
            vn = self.v + 0.5 * (3.0 * a - ao) * dt
            self.x = self.x + 0.5 * (self.v + vn) * dt
            self.w = self.w + 0.5 * (3.0 * u - uo) * dt
            self.old = (a, u)
        else:
            vn = self.v + dt * a
            self.x = self.x + vn * dt
            self.w = self.w + u * dt
        self.v = vn
        lo = torch.tensor(self.s["lo"], dtype=torch.float64, device=self.dev)
        k = torch.where(self.per, torch.floor((self.x - lo) / self.L), torch.zeros_like(self.x))
        self.x = self.x - k * self.L

    # ---- gas ----
    def set_gas(self):
        s, g = self.s, self.s["gas"]
        cx, cy, cz = s["cells"]
        self.shape = (cz + 2, cy + 2, cx + 2)
        self.ep, self.ug, self.vg, self.wg = (torch.from_numpy(np.asarray(g[k])).to(self.dev).reshape(self.shape).clone()
                                              for k in ("ep", "u", "v", "w"))
        fl = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
        fl[1:-1, 1:-1, 1:-1] = 1.0
        self.fluid = fl
        p = torch.nn.functional.pad(fl, (0, 1, 0, 1, 0, 1))
        self.node_vol = s["dx"] ** 3 * sum(p[a:a + self.shape[0], b:b + self.shape[1], c:c + self.shape[2]]
                                           for a in (0, 1) for b in (0, 1) for c in (0, 1))

    def _where(self):
        """Fluid cell of every sphere and its place in it."""
        q = self.x / self.s["dx"]
        c = q.floor()
        return (c.long() + 1).unbind(1), (q - c).unbind(1)

    @staticmethod
    def _w(z, o):
        return z if o else 1.0 - z

    def _corners(self):
        (ci, cj, ck), z = self._where()
        for a in (0, 1):
            for b in (0, 1):
                for c in (0, 1):
                    yield ci - 1 + a, cj - 1 + b, ck - 1 + c, self._w(z[0], a) * self._w(z[1], b) * self._w(z[2], c)

    def fgp(self):
        """Gas velocity at the spheres, their drag coefficient times volume."""
        ug, vg, wg, g = self.ug, self.vg, self.wg, self.s["gas"]
        (ci, cj, ck), _ = self._where()
        if self.case["scheme"] == "NONE":
            u = torch.stack([0.5 * (ug[ck, cj, ci - 1] + ug[ck, cj, ci]), 0.5 * (vg[ck, cj - 1, ci] + vg[ck, cj, ci]),
                             0.5 * (wg[ck - 1, cj, ci] + wg[ck, cj, ci])], 1)
        else:
            u = torch.zeros_like(self.x)
            for i, j, k, wt in self._corners():
                u = u + wt[:, None] * 0.25 * torch.stack(
                    [ug[k, j, i] + ug[k, j + 1, i] + ug[k + 1, j, i] + ug[k + 1, j + 1, i],
                     vg[k, j, i] + vg[k, j, i + 1] + vg[k + 1, j, i] + vg[k + 1, j, i + 1],
                     wg[k, j, i] + wg[k, j + 1, i] + wg[k, j, i + 1] + wg[k, j + 1, i + 1]], 1)
        ep, mu, ro = self.ep[ck, cj, ci], g["mu"], g["ro"]
        vr = torch.sqrt(_dot(u - self.v, u - self.v))
        dp = 2.0 * self.r
        re = dp * vr * ro * ep / mu
        dense = 150.0 * (1.0 - ep) * mu / (ep * dp * dp) + 1.75 * ro * vr / dp
        cd = torch.where(re <= 1000.0, 24.0 * (1.0 + 0.15 * re ** 0.687) / (re + 1e-15), torch.full_like(re, 0.44))
        k = torch.where(ep <= 0.8, dense, 0.75 * cd * vr * ro * ep * ep ** -2.65 / dp)
        return u, torch.where(re == 0.0, torch.zeros_like(k), k) * (4.0 / 3.0) * PI * self.r ** 3

    def drag(self):
        u, k = self.fgp()
        return k[:, None] * (u - self.v)

    def _scatter(self, i, j, k, val):
        out = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
        nz, ny, nx = self.shape
        return out.view(-1).index_add_(0, (k * ny + j) * nx + i, val).view(self.shape)

    def mean_fields(self):
        s = self.s
        vol = s["dx"] ** 3
        if self.case["scheme"] == "NONE":
            (ci, cj, ck), _ = self._where()
            self.rop = self._scatter(ci, cj, ck, s["rho"] * (4.0 / 3.0) * PI * self.r ** 3) / vol
        else:
            node = sum(self._scatter(i, j, k, wt * self.m) for i, j, k, wt in self._corners())
            dens = torch.where(self.node_vol > 0, node / self.node_vol.clamp_min(1e-300), torch.zeros_like(node))
            p = torch.nn.functional.pad(dens, (1, 0, 1, 0, 1, 0))
            nz, ny, nx = self.shape
            acc = sum(p[a:a + nz, b:b + ny, c:c + nx] for a in (0, 1) for b in (0, 1) for c in (0, 1))
            # cells outside the fluid keep the sum times the cell volume
            self.rop = torch.where(self.fluid > 0, acc, acc * vol)
        ep = 1.0 - (self.rop / s["rho"]).clamp_max(1.0)
        self.ep = torch.where(self.fluid > 0, ep, self.ep)

    def gas_side(self):
        _, k = self.fgp()
        vol = self.s["dx"] ** 3
        (ci, cj, ck), _ = self._where()
        np_ = lambda a: a.reshape(-1).cpu().numpy()  # noqa: E731
        if self.case["scheme"] == "NONE":
            f = self._scatter(ci, cj, ck, k / vol)
            bm = [self._scatter(ci, cj, ck, k * self.v[:, a] / vol) for a in range(3)]
            return dict(f_gds=np_(f), drag_bm=np.stack([np_(b) for b in bm]), f_gp=np_(k))
        nv = (self.node_vol / 8.0).clamp_min(1e-300)
        am = sum(self._scatter(i, j, q, k * wt) for i, j, q, wt in self._corners()) / nv
        bm = [sum(self._scatter(i, j, q, k * wt * self.v[:, a]) for i, j, q, wt in self._corners()) / nv
              for a in range(3)]
        p = torch.nn.functional.pad(am, (1, 0, 1, 0, 1, 0))
        nz, ny, nx = self.shape
        f = 0.125 * self.fluid * sum(p[a:a + nz, b:b + ny, c:c + nx] for a in (0, 1) for b in (0, 1) for c in (0, 1))
        return dict(f_gds=np_(f), drag_am=np_(am), drag_bm=np.stack([np_(b) for b in bm]), f_gp=np_(k))

    def state(self):
        return dict(pos=self.x.T.cpu().numpy(), vel=self.v.T.cpu().numpy(), omega=self.w.T.cpu().numpy(), state=None)


def exact(case, seed):
    """What `run` returns on a fresh state, followed in 64 bits."""
    got = []
    for s in _inputs(case, seed):
        e = _Exact(case, s)
        if "gas" in s:
            e.set_gas()
        e.step(case["nsn"])
        if case["kind"] == "fluid_step":
            e.set_gas()
        e.step(case["steps"])
        got.append(e.state())
        if case["kind"] == "coupled":
            got[-1].update(ep_g=e.ep.reshape(-1).cpu().numpy(), rop_s=e.rop.reshape(-1).cpu().numpy())
        if case["kind"] == "fluid_step":
            got[-1].update(e.gas_side())
    return got if case["kind"] in ("columns", "hoppers") else got[0]
