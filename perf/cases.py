"""The calls that a user of this framework makes, as cases that can be timed.

Each case is one pass through the public entry points on inputs made from a
seed: flow maps (FP64, the drop-in default, and mixed precision) of the
analytic and the spline flows, the FTLE and Cauchy-Green fields, ridge points
and labelled ridges, flow-map composition, the spline build and a batch of
fields.  ``listed()`` holds the ordinary ones; ``draw(rng)`` takes others of
the same ranges; ``exact(case, seed)`` gives what a case computes in plain
64-bit torch / numpy.
"""
import math

import numpy as np
import torch

import numbacs_gb300 as nb
from numbacs_gb300 import workloads
from numbacs_gb300.batch import TILES, Field, FTLEBatch
from numbacs_gb300.extraction import ftle_ridge_pts, ftle_ridges
from numbacs_gb300.flows import eval_rhs

DEG = 180.0 / math.pi
R_EARTH = 6371.0
NT, NLON, NLAT = 121, 217, 101  # the geophysical velocity grid of workloads.geo_grid


def listed():
    return [
        # a first try: the 21 x 11 double gyre of the reference's own fixtures
        {"name": "dg_tiny_fp64", "op": "flowmap", "flow": "double_gyre", "precision": "fp64",
         "nx": 21, "ny": 11, "T": 8.0, "rtol": 1e-6, "atol": 1e-8, "arrays": "torch"},
        # the reference's double-gyre example as a drop-in user calls it: numpy
        # arrays, default precision and tolerances
        {"name": "dg_fp64", "op": "flowmap", "flow": "double_gyre", "precision": "fp64",
         "nx": 401, "ny": 201, "T": -10.0, "rtol": 1e-6, "atol": 1e-8, "arrays": "numpy"},
        # the geophysical flow (spline, spherical) at 0.4 degrees, default precision
        {"name": "geo_fp64", "op": "flowmap", "flow": "geo", "precision": "fp64",
         "nx": 338, "ny": 126, "T": -72.0, "rtol": 1e-6, "atol": 1e-8, "arrays": "torch"},
        # the benchmark's flow map: 0.2 degrees, mixed precision, its tolerance
        {"name": "geo_mixed", "op": "flowmap", "flow": "geo", "precision": "mixed",
         "nx": 676, "ny": 251, "T": -72.0, "rtol": 3e-9, "atol": 3e-8, "arrays": "torch"},
        # a time series in one batch: spline fields of mixed sizes and lengths
        # and a Bickley jet field, flow maps and FTLE of all of them
        {"name": "batch", "op": "batch", "nfields": 6, "jet_nx": 1001, "jet_ny": 301,
         "jet_T": 20.0, "rtol": 1e-7, "atol": 1e-6},
        # the FTLE of the double-gyre example's grid: one short call
        {"name": "ftle_small", "op": "ftle", "nx": 401, "ny": 201, "T": -10.0, "mask": False},
        # FTLE and ridge direction of a large grid
        {"name": "ftle_evec_large", "op": "evec", "nx": 4001, "ny": 4001, "T": -10.0,
         "mask": False},
        # the reference's idiom C_eig_2D -> ftle_from_eig on a 0.1 degree grid
        {"name": "ceig", "op": "ceig", "nx": 1351, "ny": 501, "T": -72.0, "mask": True},
        # ridge points of the benchmark's grid
        {"name": "ridge_pts", "op": "ridge_pts", "nx": 676, "ny": 251, "percentile": 90},
        # labelled ridges of a 0.05 degree grid
        {"name": "ridges", "op": "ridges", "nx": 2701, "ny": 1001, "percentile": 90},
        # a 72 h flow map composed of hourly ones
        {"name": "compose", "op": "compose", "nx": 676, "ny": 251, "maps": 72},
        # new velocity data made into a flow, and its velocity at the particles
        {"name": "spline", "op": "spline", "nt": NT, "nx": NLON, "ny": NLAT, "points": 169676},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["flowmap", "flowmap", "flowmap", "batch", "ftle", "evec", "ceig", "ridge_pts",
                     "ridges", "compose", "spline"])
    if op == "flowmap":
        flow = rng.choice(["double_gyre", "bickley_jet", "geo"])
        precision = rng.choice(["fp64", "mixed"])
        # FP64 particles cost about 40 times the mixed ones
        side = (338, 126) if precision == "fp64" else (676, 251)
        length = {"double_gyre": (4.0, 15.0), "bickley_jet": (4.0, 20.0), "geo": (24.0, 72.0)}[flow]
        rtol = rng.choice([1e-6, 1e-7] if precision == "fp64" or flow != "geo"
                          else [1e-6, 1e-7, 3e-9])
        T = round(rng.uniform(*length), 2)
        return {"op": op, "flow": flow, "precision": precision, "nx": _log(rng, 16, side[0]),
                "ny": _log(rng, 9, side[1]), "T": -T if flow == "geo" or rng.random() < 0.5 else T,
                "rtol": rtol, "atol": rtol * (10.0 if precision == "mixed" else 0.01),
                "arrays": rng.choice(["torch", "numpy"])}
    if op == "batch":
        return {"op": op, "nfields": rng.randint(2, 6), "jet_nx": _log(rng, 64, 1001),
                "jet_ny": _log(rng, 32, 301), "jet_T": round(rng.uniform(5.0, 20.0), 2),
                "rtol": 1e-7, "atol": 1e-6}
    if op in ("ftle", "evec", "ceig"):
        most = 4001 if op == "evec" else 2001
        return {"op": op, "nx": _log(rng, 21, most), "ny": _log(rng, 11, most),
                "T": round(rng.uniform(4.0, 72.0), 2), "mask": rng.random() < 0.3}
    if op in ("ridge_pts", "ridges"):
        return {"op": op, "nx": _log(rng, 64, 2701), "ny": _log(rng, 48, 1001),
                "percentile": rng.choice([0, 50, 80, 90, 95])}
    if op == "compose":
        return {"op": op, "nx": _log(rng, 64, 676), "ny": _log(rng, 48, 251),
                "maps": rng.randint(2, 72)}
    return {"op": op, "nt": _log(rng, 9, NT), "nx": _log(rng, 24, NLON), "ny": _log(rng, 16, NLAT),
            "points": _log(rng, 231, 169676)}


# ---------------------------------------------------------------- inputs

def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _linspace(a, b, n):
    return torch.from_numpy(np.linspace(a, b, n)).to(_dev())


def _velocity(seed, nt=NT, nx=NLON, ny=NLAT):
    """The synthetic geophysical velocity of `seed` on an nt x nx x ny grid."""
    t = 3.0 * np.arange(nt, dtype=np.float64)
    lon, lat = np.linspace(-100.0, 35.0, nx), np.linspace(-5.0, 45.0, ny)
    _, _, _, U, V = workloads.geo_velocity(seed, t=t, lon=lon, lat=lat)
    return t, lon, lat, torch.from_numpy(U).to(_dev()), torch.from_numpy(V).to(_dev())


def _flow(case, seed):
    """(params, t0, x, y) of a flow-map case, numpy; the flow's own values vary
    with the seed, within what its users set."""
    rng = np.random.default_rng(seed)
    if case["flow"] == "double_gyre":
        p = [math.copysign(1.0, case["T"]), rng.uniform(0.09, 0.11), rng.uniform(0.2, 0.3), 0.0,
             0.2 * math.pi, 0.0]
        return np.array(p), rng.uniform(0.0, 10.0), np.linspace(0.0, 2.0, case["nx"]), \
            np.linspace(0.0, 1.0, case["ny"])
    if case["flow"] == "bickley_jet":
        p = nb.get_predefined_flow("bickley_jet")[1].copy()
        p[0] = math.copysign(1.0, case["T"])
        p[3:6] *= rng.uniform(0.9, 1.1, 3)
        return p, rng.uniform(0.0, 10.0), np.linspace(0.0, 6.371 * math.pi, case["nx"]), \
            np.linspace(-3.0, 3.0, case["ny"])
    return np.array([-1.0]), 180.0, np.linspace(-100.0, 35.0, case["nx"]), \
        np.linspace(-5.0, 45.0, case["ny"])


def _batch_specs(case, seed):
    """[(t0, T, spacing)] of the batch's spline fields: hourly start times,
    lengths and grid spacings as the time series of the benchmark has them."""
    rng = np.random.default_rng(seed)
    spacing = [0.4, 0.2, 0.4, 0.1, 0.4, 0.2]
    return [(168.0 + k, float(rng.uniform(-120.0, -24.0)), spacing[k])
            for k in range(case["nfields"])]


def _shears(seed, nx, ny):
    """An area-preserving map of the (nx, ny) grid over [0, 2] x [0, 1], four
    sine shears: smooth, stretching and folding, as a flow map is."""
    rng = np.random.default_rng(seed)
    x, y = _linspace(0.0, 2.0, nx), _linspace(0.0, 1.0, ny)
    X, Y = x[:, None].expand(nx, ny).clone(), y[None, :].expand(nx, ny).clone()
    for _ in range(4):
        a, b, c, d = rng.uniform(0.15, 0.3), rng.uniform(0.1, 0.2), *rng.uniform(0.0, 2 * math.pi, 2)
        X = X + a * torch.sin(math.pi * Y + c)
        Y = Y + b * torch.sin(math.pi * X + d)
    return torch.stack([X, Y], dim=2).contiguous(), x, y


def _mask(case, seed):
    if not case.get("mask"):
        return None
    g = torch.Generator(device=_dev()).manual_seed(seed)
    return torch.rand((case["nx"], case["ny"]), generator=g, device=_dev()) < 0.2


def _tensor(F, dx, dy):
    """Cauchy-Green tensor (a, b, d) of the interior points, plain torch."""
    gx = (F[2:, 1:-1] - F[:-2, 1:-1]) / (2.0 * dx)
    gy = (F[1:-1, 2:] - F[1:-1, :-2]) / (2.0 * dy)
    return (gx * gx).sum(2), (gx * gy).sum(2), (gy * gy).sum(2)


def _eig(a, b, d):
    """(smaller, larger, unit eigenvector of the larger with x >= 0)."""
    l1 = 0.5 * ((a + d) + torch.sqrt((a - d) ** 2 + 4.0 * b * b))
    l0 = torch.where(l1 > 0, (a * d - b * b) / l1, 0.5 * (a + d))
    big = a >= d
    ex, ey = torch.where(big, l1 - d, b), torch.where(big, b, l1 - a)
    zero = b == 0
    ex = torch.where(zero, big.double(), ex)
    ey = torch.where(zero, 1.0 - big.double(), ey)
    n = torch.sqrt(ex * ex + ey * ey)
    s = torch.where((ex < 0) | ((ex == 0) & (ey < 0)), -1.0, 1.0) / n
    return l0, l1, torch.stack([ex * s, ey * s], dim=2)


def _inside(v, nx, ny):
    out = torch.zeros((nx, ny) + tuple(v.shape[2:]), dtype=v.dtype, device=v.device)
    out[1:-1, 1:-1] = v
    return out


def _ridge_field(case, seed):
    """FTLE field and ridge direction of one shear map, mirrored, scaled and
    moved by the seed: the fields of all seeds have equally many ridge points,
    so that their times compare.  The spacing and the moves are dyadic: no seed
    changes the spacing by a rounding."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    F, _, _ = _shears(7, nx, ny)
    a, b, d = _tensor(F, 2.0 / (nx - 1), 1.0 / (ny - 1))
    _, l1, ev = _eig(a, b, d)
    f = torch.where(l1 > 1.0, torch.log(l1.clamp_min(1.0)) / 20.0, torch.zeros_like(l1))
    f, ev = _inside(f * rng.uniform(0.5, 2.0), nx, ny), _inside(ev, nx, ny)
    for axis in (0, 1):
        if rng.random() < 0.5:
            f, ev = f.flip(axis), ev.flip(axis)
            ev = ev * torch.tensor([-1.0, 1.0] if axis == 0 else [1.0, -1.0], dtype=ev.dtype,
                                   device=ev.device)
    ev = torch.where(ev[..., :1] < 0, -ev, ev)
    hx, hy = 2.0 ** -round(math.log2((nx - 1) / 2.0)), 2.0 ** -round(math.log2(ny - 1.0))
    x = hx * (torch.arange(nx, dtype=torch.float64, device=_dev()) + rng.integers(-4000, 4000))
    y = hy * (torch.arange(ny, dtype=torch.float64, device=_dev()) + rng.integers(-4000, 4000))
    return f.contiguous(), ev.contiguous(), x, y


def _maps(case, seed):
    """Hourly flow maps of the grid: each point moved by a smooth displacement
    of up to about half a degree."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    x, y = _linspace(-100.0, 35.0, nx), _linspace(-5.0, 45.0, ny)
    out = torch.empty((case["maps"], nx, ny, 2), dtype=torch.float64, device=_dev())
    for k in range(case["maps"]):
        a, b, c, d = *rng.uniform(0.05, 0.15, 2), *rng.uniform(0.0, 2 * math.pi, 2)
        sx, sy = torch.sin(a * x + c), torch.sin(b * y + d)
        cx, cy = torch.cos(a * x + c), torch.cos(b * y + d)
        out[k, :, :, 0] = x[:, None] + 0.4 * sx[:, None] * cy[None, :]
        out[k, :, :, 1] = y[None, :] - 0.3 * cx[:, None] * sy[None, :]
    return out, nb.UCGrid((-100.0, 35.0, nx), (-5.0, 45.0, ny))


def _points(case, seed, t):
    g = torch.Generator(device=_dev()).manual_seed(seed)
    r = torch.rand((case["points"], 3), generator=g, device=_dev(), dtype=torch.float64)
    lo = torch.tensor([0.0, -100.0, -5.0], dtype=torch.float64, device=_dev())
    hi = torch.tensor([float(t[-1]), 35.0, 45.0], dtype=torch.float64, device=_dev())
    return lo + r * (hi - lo)


# ------------------------------------------------------------- the calls

def prepare(case, seed):
    op = case["op"]
    if op == "flowmap":
        p, t0, x, y = _flow(case, seed)
        if case["flow"] == "geo":
            t, lon, lat, U, V = _velocity(seed)
            flow = nb.get_flow_2D(*nb.get_interp_arrays_2D(t, lon, lat, U, V), spherical=1)
        else:
            flow = nb.get_predefined_flow(case["flow"])[0]
        if case["arrays"] == "torch":
            x, y = torch.from_numpy(x).to(_dev()), torch.from_numpy(y).to(_dev())
        return {"case": case, "flow": flow, "p": p, "t0": t0, "x": x, "y": y}
    if op == "batch":
        t, lon, lat, U, V = _velocity(seed)
        flow = nb.get_flow_2D(*nb.get_interp_arrays_2D(t, lon, lat, U, V), spherical=1)
        fields = []
        for t0, T, h in _batch_specs(case, seed):
            x, y = workloads.geo_ftle_grid(h)
            fields.append(Field(flow, t0, T, x, y, np.array([-1.0]), case["rtol"], case["atol"]))
        jet, p, _ = nb.get_predefined_flow("bickley_jet")
        fields.append(Field(jet, 0.1 * (seed % 97), case["jet_T"],
                            *workloads.bickley_batch_grid(case["jet_nx"], case["jet_ny"]), p))
        return {"case": case, "batch": FTLEBatch(fields, precision="mixed", blocks_per_sm=TILES)}
    if op in ("ftle", "evec", "ceig"):
        F, x, y = _shears(seed, case["nx"], case["ny"])
        return {"case": case, "F": F, "dx": float(x[1] - x[0]), "dy": float(y[1] - y[0]),
                "mask": _mask(case, seed)}
    if op in ("ridge_pts", "ridges"):
        f, ev, x, y = _ridge_field(case, seed)
        return {"case": case, "f": f, "ev": ev, "x": x, "y": y}
    if op == "compose":
        maps, grid = _maps(case, seed)
        return {"case": case, "maps": maps, "grid": grid}
    t, lon, lat, U, V = _velocity(seed, case["nt"], case["nx"], case["ny"])
    return {"case": case, "t": t, "lon": lon, "lat": lat, "U": U, "V": V,
            "pts": _points(case, seed, t)}


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "flowmap":
        fm = nb.flowmap_grid_2D(state["flow"], state["t0"], case["T"], state["x"], state["y"],
                                state["p"], rtol=case["rtol"], atol=case["atol"],
                                precision=case["precision"])
        return {"flowmap": fm}
    if op == "batch":
        state["batch"].run()
        return [{"flowmap": fm, "ftle": f, "evec": ev, "status": st}
                for fm, f, ev, st in state["batch"].results()]
    if op == "ftle":
        return {"ftle": nb.ftle_grid_2D(state["F"], case["T"], state["dx"], state["dy"],
                                        mask=state["mask"])}
    if op == "evec":
        f, ev = nb.ftle_evec_2D(state["F"], case["T"], state["dx"], state["dy"],
                                mask=state["mask"])
        return {"ftle": f, "evec": ev}
    if op == "ceig":
        vals, vecs = nb.C_eig_2D(state["F"], state["dx"], state["dy"], mask=state["mask"])
        return {"vals": vals, "vecs": vecs, "ftle": nb.ftle_from_eig(vals[..., 1], case["T"])}
    if op == "ridge_pts":
        return {"points": ftle_ridge_pts(state["f"], state["ev"], state["x"], state["y"],
                                         percentile=case["percentile"])}
    if op == "ridges":
        rs = ftle_ridges(state["f"], state["ev"], state["x"], state["y"],
                         percentile=case["percentile"])
        return {"points": torch.cat(rs) if rs else torch.zeros((0, 2), dtype=torch.float64),
                "lengths": np.array([r.shape[0] for r in rs], np.int64)}
    if op == "compose":
        return {"flowmap": nb.flowmap_composition(state["maps"], state["grid"], case["maps"])}
    grid, cu, cv = nb.get_interp_arrays_2D(state["t"], state["lon"], state["lat"], state["U"],
                                           state["V"])
    flow = nb.get_flow_2D(grid, cu, cv, spherical=1)
    return {"cu": cu, "cv": cv,
            "velocity": eval_rhs(flow, 0.0, state["pts"], np.array([1.0]))}


# ------------------------------------------------------------------ work

def _steps(flow, T, rtol):
    """Attempted DOP853 steps of a trajectory, about: the order-8 step grows
    as rtol^(1/8); per unit of time as measured on each flow."""
    per = {"double_gyre": 0.28, "bickley_jet": 0.5, "geo": 0.12}[flow]
    return max(2.0, per * abs(T) * rtol ** -0.125)


_RHS = {"double_gyre": 60.0, "bickley_jet": 110.0, "geo": 330.0}


def _flowmap_work(flow, precision, n, T, rtol):
    node = 16.0 if precision == "fp64" else 8.0
    coef = (NT + 2) * (NLON + 2) * (NLAT + 2) * node * min(1.0, (abs(T) / 3.0 + 4) / (NT + 2)) \
        if flow == "geo" else 0.0
    return {"bytes": 20.0 * n + coef, "flops": n * _steps(flow, T, rtol) * (438.0 + 12 * _RHS[flow])}


def work(case):
    op = case["op"]
    n = float(case.get("nx", 0) * case.get("ny", 0))
    if op == "flowmap":
        return _flowmap_work(case["flow"], case["precision"], n, case["T"], case["rtol"])
    if op == "batch":
        w = _flowmap_work("bickley_jet", "mixed", case["jet_nx"] * case["jet_ny"], case["jet_T"], 1e-6)
        particles = case["jet_nx"] * case["jet_ny"]
        for _, _, h in _batch_specs(case, 0):
            x, y = workloads.geo_ftle_grid(h)
            m = len(x) * len(y)
            particles += m
            g = _flowmap_work("geo", "mixed", m, 72.0, case["rtol"])
            w = {"bytes": w["bytes"] + 20.0 * m, "flops": w["flops"] + g["flops"]}
        return {"bytes": w["bytes"] + 24.0 * particles, "flops": w["flops"] + 50.0 * particles}
    if op == "ftle":
        return {"bytes": 24.0 * n, "flops": 50.0 * n}
    if op == "evec":
        return {"bytes": 40.0 * n, "flops": 60.0 * n}
    if op == "ceig":
        return {"bytes": 72.0 * n, "flops": 90.0 * n}
    if op == "ridge_pts":
        return {"bytes": 8.0 * n, "flops": 5.0 * n}
    if op == "ridges":
        return {"bytes": 9.0 * n, "flops": 5.0 * n}
    if op == "compose":
        return {"bytes": 16.0 * n * (case["maps"] + 1), "flops": 26.0 * n * case["maps"]}
    m = float((case["nt"] + 2) * (case["nx"] + 2) * (case["ny"] + 2))
    return {"bytes": 2 * 8.0 * n * case["nt"] + 2 * 8.0 * m + 2 * 16.0 * m + 40.0 * case["points"],
            "flops": 2 * 3 * 8.0 * m + 330.0 * case["points"]}


# ----------------------------------------------------------------- exact

def _prefilter(f):
    """Natural cubic B-spline coefficients of f along its three axes."""
    for axis in range(3):
        n = f.shape[axis]
        A = np.zeros((n + 2, n + 2))
        A[0, :3] = A[-1, -3:] = (1.0, -2.0, 1.0)
        for k in range(n):
            A[k + 1, k:k + 3] = (1.0 / 6.0, 4.0 / 6.0, 1.0 / 6.0)
        S = torch.from_numpy(np.ascontiguousarray(np.linalg.inv(A)[:, 1:-1])).to(f.device)
        f = torch.movedim(torch.tensordot(S, f, dims=([1], [axis])), 0, axis)
    return f.contiguous()


def _spline(C, lo, hi, n, pts):
    """(u, v) of the spline with coefficients C (nt+2, nx+2, ny+2, 2) at pts
    (k, 3); zero outside the grid box."""
    out = torch.zeros(pts.shape[0], dtype=torch.bool, device=pts.device)
    idx, wgt = [], []
    for d in range(3):
        u = (pts[:, d] - lo[d]) * ((n[d] - 1) / (hi[d] - lo[d]))
        out |= (pts[:, d] < lo[d]) | (pts[:, d] > hi[d])
        i = torch.floor(u).clamp(0, n[d] - 2)
        t = u - i
        s = 1.0 - t
        wgt.append(torch.stack([s ** 3, 3 * t ** 3 - 6 * t ** 2 + 4,
                                -3 * t ** 3 + 3 * t ** 2 + 3 * t + 1, t ** 3], 1) / 6.0)
        idx.append(i.long())
    NX, NY = n[1] + 2, n[2] + 2
    base = (idx[0] * NX + idx[1]) * NY + idx[2]
    flat = C.view(-1, 2)
    q = torch.arange(4, device=pts.device)
    uv = torch.zeros((pts.shape[0], 2), dtype=torch.float64, device=pts.device)
    for a in range(4):
        for b in range(4):
            rows = flat[(base + (a * NX + b) * NY)[:, None] + q]
            w = wgt[0][:, a] * wgt[1][:, b]
            uv += w[:, None] * (wgt[2][:, :, None] * rows).sum(1)
    uv[out] = 0.0
    return uv


def _rhs(case, p, C):
    if case["flow"] == "double_gyre":
        _, A, eps, alpha, om, psi = p

        def f(t, q):
            x, y = q[:, 0], q[:, 1]
            a = eps * math.sin(om * t + psi)
            b = 1.0 - 2.0 * a
            g, dg = a * x * x + b * x, 2.0 * a * x + b
            return torch.stack([
                -math.pi * A * torch.sin(math.pi * g) * torch.cos(math.pi * y) - alpha * x,
                math.pi * A * torch.cos(math.pi * g) * torch.sin(math.pi * y) * dg - alpha * y], 1)
        return f
    if case["flow"] == "bickley_jet":
        _, U0, L, A1, A2, A3, k1, k2, k3, c1, c2, c3 = p
        terms = ((A1, k1, c1), (A2, k2, c2), (A3, k3, c3))

        def f(t, q):
            x, y = q[:, 0], q[:, 1] / L
            s2 = 1.0 / torch.cosh(y) ** 2
            cs = sum(A * torch.cos(k * (x - c * t)) for A, k, c in terms)
            sn = sum(A * k * torch.sin(k * (x - c * t)) for A, k, c in terms)
            return torch.stack([U0 * s2 * (1.0 + 2.0 * torch.tanh(y) * cs), -U0 * L * s2 * sn], 1)
        return f

    def f(t, q):
        pts = torch.cat([torch.full_like(q[:, :1], t), q], 1)
        uv = _spline(C, (0.0, -100.0, -5.0), (3.0 * (NT - 1), 35.0, 45.0), (NT, NLON, NLAT), pts)
        uv = uv * (DEG / R_EARTH)
        uv[:, 0] /= torch.cos(q[:, 1] / DEG)
        return uv
    return f


def exact(case, seed):
    op = case["op"]
    if op == "flowmap":
        p, t0, x, y = _flow(case, seed)
        x, y = torch.from_numpy(x).to(_dev()), torch.from_numpy(y).to(_dev())
        nx, ny = len(x), len(y)
        q = torch.stack([x[:, None].expand(nx, ny), y[None, :].expand(nx, ny)], 2).reshape(-1, 2)
        C = None
        if case["flow"] == "geo":
            _, _, _, U, V = _velocity(seed)
            C = torch.stack([_prefilter(U), _prefilter(V)], 3).contiguous()
        f = _rhs(case, p, C)
        # classical Runge-Kutta at a fixed fine step
        steps = int(math.ceil(abs(case["T"]) * {"double_gyre": 100, "bickley_jet": 60, "geo": 8}[case["flow"]]))
        h, t = case["T"] / steps, t0
        for k in range(steps):
            t = t0 + k * h
            k1 = f(t, q)
            k2 = f(t + 0.5 * h, q + 0.5 * h * k1)
            k3 = f(t + 0.5 * h, q + 0.5 * h * k2)
            k4 = f(t + h, q + h * k3)
            q = q + (h / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        q = q.reshape(nx, ny, 2)
        return {"flowmap": q if case["arrays"] == "torch" else q.cpu().numpy()}
    if op == "batch":
        return None  # over a million trajectories: minutes in plain torch
    if op in ("ftle", "evec", "ceig"):
        nx, ny = case["nx"], case["ny"]
        F, x, y = _shears(seed, nx, ny)
        l0, l1, ev = _eig(*_tensor(F, float(x[1] - x[0]), float(y[1] - y[0])))
        f = torch.where(l1 > 1.0, torch.log(l1.clamp_min(1.0)), torch.zeros_like(l1)) \
            / (2.0 * abs(case["T"]))
        vals = torch.stack([l0, l1], 2)
        vecs = torch.stack([torch.stack([-ev[..., 1], ev[..., 0]], 2), ev], 2)
        out = {"ftle": f, "evec": ev, "vals": vals, "vecs": vecs}
        mask = _mask(case, seed)
        for key in out:
            v = _inside(out[key], nx, ny)
            if mask is not None:
                v[mask] = 0.0
            out[key] = v
        return {k: out[k] for k in {"ftle": ("ftle",), "evec": ("ftle", "evec"),
                                    "ceig": ("vals", "vecs", "ftle")}[op]}
    if op in ("ridge_pts", "ridges"):
        return _exact_ridges(case, seed)
    if op == "compose":
        maps, grid = _maps(case, seed)
        (x0, x1, nx), (y0, y1, ny) = grid
        pt = maps[0].reshape(-1, 2)
        for k in range(1, case["maps"]):
            m = maps[k].reshape(-1, 2)
            u, v = (pt[:, 0] - x0) * ((nx - 1) / (x1 - x0)), (pt[:, 1] - y0) * ((ny - 1) / (y1 - y0))
            i, j = torch.floor(u).clamp(0, nx - 2), torch.floor(v).clamp(0, ny - 2)
            a, b = (u - i)[:, None], (v - j)[:, None]
            e = (i * ny + j).long()
            new = (1 - a) * ((1 - b) * m[e] + b * m[e + 1]) + a * ((1 - b) * m[e + ny] + b * m[e + ny + 1])
            out = (pt[:, 0] < x0) | (pt[:, 0] > x1) | (pt[:, 1] < y0) | (pt[:, 1] > y1)
            new[out] = 0.0
            pt = new
        return {"flowmap": pt.reshape(nx, ny, 2)}
    t, _, _, U, V = _velocity(seed, case["nt"], case["nx"], case["ny"])
    pts = _points(case, seed, t)
    cu, cv = _prefilter(U), _prefilter(V)
    uv = _spline(torch.stack([cu, cv], 3).contiguous(), (0.0, -100.0, -5.0), (float(t[-1]), 35.0, 45.0),
                 (case["nt"], case["nx"], case["ny"]), pts) * (DEG / R_EARTH)
    uv[:, 0] /= torch.cos(pts[:, 2] / DEG)
    return {"cu": cu, "cv": cv, "velocity": uv}


def _exact_ridges(case, seed):
    f, ev, x, y = (v.cpu().numpy() for v in _ridge_field(case, seed))
    dx, dy = x[1] - x[0], y[1] - y[0]
    low = np.percentile(f, case["percentile"]) if case["percentile"] else 0.0
    c = f[2:-2, 2:-2]
    xp, xm, yp, ym = f[3:-1, 2:-2], f[1:-3, 2:-2], f[2:-2, 3:-1], f[2:-2, 1:-3]
    fx, fy = (xp - xm) / (2 * dx), (yp - ym) / (2 * dy)
    fxx, fyy = (xp - 2 * c + xm) / dx ** 2, (yp - 2 * c + ym) / dy ** 2
    fxy = (f[3:-1, 3:-1] - f[3:-1, 1:-3] - f[1:-3, 3:-1] + f[1:-3, 1:-3]) / (4 * dx * dy)
    ex, ey = ev[2:-2, 2:-2, 0], ev[2:-2, 2:-2, 1]
    c2 = ex * (fxx * ex + fxy * ey) + ey * (fxy * ex + fyy * ey)
    with np.errstate(divide="ignore", invalid="ignore"):
        t = -(fx * ex + fy * ey) / c2
    on = (c > low) & (c2 < 0) & (np.abs(t * ex) <= dx / 2) & (np.abs(t * ey) <= dy / 2)
    i, j = np.nonzero(on)
    pts = np.stack([x[i + 2] + (t * ex)[on], y[j + 2] + (t * ey)[on]], 1)
    if case["op"] == "ridge_pts":
        return {"points": torch.from_numpy(pts).to(_dev())}
    # 8-connected components, ordered by their first point in row-major order
    at = {k: q for q, k in enumerate(zip(i.tolist(), j.tolist()))}
    root = list(range(len(pts)))

    def find(a):
        while root[a] != a:
            root[a] = root[root[a]]
            a = root[a]
        return a

    for (a, b), q in at.items():
        for other in ((a - 1, b - 1), (a - 1, b), (a - 1, b + 1), (a, b - 1)):
            if other in at:
                r, s = find(q), find(at[other])
                root[max(r, s)] = min(r, s)
    lab = np.array([find(q) for q in range(len(pts))], np.int64)
    order = np.argsort(lab, kind="stable")
    n = np.bincount(lab, minlength=max(1, len(pts)))
    keep = n[lab[order]] >= 3
    return {"points": torch.from_numpy(pts[order][keep]).to(_dev()), "lengths": n[n >= 3]}
