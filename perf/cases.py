"""What a user of this framework has it do, as timed cases: one pass through the public entry
points on plates of the sizes the configurations, tests and examples of this repository use.

  * assemble: one residual (+ tangent) assembly of a plate with one elastic hinge, as a Newton
    iteration or a line-search trial calls it: host arrays in and out (the drivers' call) or
    device buffers (a caller that keeps K on the GPU);
  * batch: independent plates of uneven size as one problem, one CUDA-graph launch per pass;
  * shape: shape functions of scattered points over a node grid with one cut;
  * rebuild: every shape set of a plate recomputed for a moved cut (one step of progressive
    creasing);
  * post: what is written after an accepted step: strain energies and the point states.

A mixed-precision K holds FP32 sums widened to FP64, and the device KKT solve factors it in
FP32, so a mixed pass ends with K in FP32 (the conversion is exact).

`exact` restates the method in plain torch, FP64, from the geometry alone."""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "curvami-official_gb300"))

H = 0.5                      # node spacing of every plate
E_MOD, NU, THICK = 1.0, 0.3, 0.05
DOUBLE = torch.float64


# ---- the cases -----------------------------------------------------------------------------

def _assemble(name, n_side, **kw):
    c = {"kind": "assemble", "n_side": n_side, "rule": 3, "order": 2, "rho": 3.0, "window": 0, "crease": "line",
         "layup": "isotropic", "mode": "fp64", "want_K": True, "hinge_exact": False, "io": "host"}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A Newton iteration on the smallest plates the tests solve: launches and latency count.
        _assemble("newton_small", 15),
        # A Newton iteration of the plain FP64 method on the 41 x 41 plate (4x4 rule, cubic
        # B-spline window, rho = 3.5h), host arrays in and out.
        _assemble("newton_41", 41, rule=4, rho=3.5, window=1),
        # The square-twist example's class: cubic basis at rho = 6h, over 100 neighbours, exact
        # hinge tangent, 3x3 rule, host arrays in and out.
        _assemble("twist_61", 61, order=3, rho=6.0, hinge_exact=True),
        # A line-search trial (residual only) of a mid-size plate, device buffers.
        _assemble("trial_121", 121, rule=4, rho=3.5, crease="arc", want_K=False, io="device"),
        # FP64 residual and tangent of an odd-sized plate, device buffers.
        _assemble("plate_97_fp64", 97, rule=4, rho=3.5, crease="arc", io="device"),
        # The single-plate assembly at scale (201 x 201 nodes, 640,000 Gauss points), mixed.
        _assemble("plate_201_mixed", 201, rule=4, crease="arc", mode="mixed", io="device"),
        # An unsymmetric laminate (B != 0), mixed precision with the deterministic scatter.
        _assemble("laminate_87_det", 87, rule=3, layup="unsymmetric", mode="mixed_det", io="device"),
        # Uneven plates as one problem, one graph launch.
        {"name": "batch_12", "kind": "batch", "plates": 12, "side_min": 21, "side_max": 101, "rule": 4},
        # Shape functions of a new point set: scattered points, per-node radius, one cut.
        {"name": "shape_fp64", "kind": "shape", "points": 300000, "n_side": 301, "order": 2, "rho": 3.0, "window": 1,
         "per_node": True, "precision": "fp64"},
        # The same at a million points in mixed precision.
        {"name": "shape_mixed", "kind": "shape", "points": 1000000, "n_side": 401, "order": 2, "rho": 3.0, "window": 1,
         "per_node": True, "precision": "mixed"},
        # One tip move of progressive creasing on a sheet with cubic basis at rho = 6h.
        {"name": "rebuild_61", "kind": "rebuild", "n_side": 61, "rule": 3, "order": 3, "rho": 6.0, "window": 0},
        # After an accepted step of that sheet: energies and the exporter's point states.
        {"name": "post_81", "kind": "post", "n_side": 81, "rule": 3, "order": 2, "rho": 3.0, "window": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["newton", "newton", "cubic", "trial", "fp64", "mixed", "mixed", "laminate", "batch", "shape",
                       "shape", "rebuild", "post"])
    rule, crease = rng.choice([3, 4]), rng.choice(["line", "arc", "none"])
    # A support that an arc cuts wherever it falls needs the wide radius to be well conditioned.
    rho = 3.5 if crease == "arc" else rng.choice([3.0, 3.25, 3.5])
    quad = {"rule": rule, "crease": crease, "rho": rho, "window": rng.choice([0, 1])}
    if what == "newton":
        return _assemble(None, _log(rng, 15, 61), **quad)
    if what == "cubic":
        return _assemble(None, _log(rng, 21, 55), order=3, rho=rng.choice([5.0, 6.0]), hinge_exact=True,
                         crease=rng.choice(["line", "arc"]))
    if what == "trial":
        return _assemble(None, _log(rng, 15, 161), want_K=False, io=rng.choice(["host", "device"]), **quad)
    if what == "fp64":
        return _assemble(None, _log(rng, 31, 121), io="device", **quad)
    if what == "mixed":
        return _assemble(None, _log(rng, 21, 201), mode="mixed", io=rng.choice(["host", "device"]), **quad)
    if what == "laminate":
        return _assemble(None, _log(rng, 21, 111), layup="unsymmetric", mode=rng.choice(["mixed", "mixed_det"]),
                         io="device", **quad)
    if what == "batch":
        return {"kind": "batch", "plates": rng.randint(3, 12), "side_min": rng.randint(21, 41),
                "side_max": rng.randint(42, 101), "rule": rule}
    if what == "shape":
        return {"kind": "shape", "points": _log(rng, 3000, 300000), "n_side": rng.randint(61, 301),
                "order": rng.choice([1, 2, 2, 2]), "rho": 3.0, "window": rng.choice([0, 1]),
                "per_node": rng.choice([True, False]), "precision": rng.choice(["fp64", "mixed"])}
    n_side, order = _log(rng, 21, 61), rng.choice([2, 3])
    return {"kind": "rebuild" if what == "rebuild" else "post", "n_side": n_side, "rule": 3, "order": order,
            "rho": 3.25 if order == 2 else 6.0, "window": 0}


# ---- geometry (numpy, from the seed alone) ---------------------------------------------------

_GAUSS = {r: np.polynomial.legendre.leggauss(r) for r in (3, 4)}


def _nodes(n, rng, jitter):
    Y, X = np.meshgrid(np.arange(n) * H, np.arange(n) * H, indexing="ij")
    jx, jy = (rng.uniform(-jitter, jitter, (n, n)) for _ in range(2))
    jx[:, [0, -1]] = 0.0
    jy[[0, -1], :] = 0.0
    return np.stack([(X + jx).ravel(), (Y + jy).ravel()], 1)


def _cells(nodes, n, rule):
    """Tensor Gauss points of every grid cell: the bilinear map and its |det J| weights."""
    q, w = _GAUSS[rule]
    P = nodes.reshape(n, n, 2)
    c = np.stack([P[:-1, :-1], P[:-1, 1:], P[1:, 1:], P[1:, :-1]], 2).reshape(-1, 4, 2)
    xi, eta = (a.ravel() for a in np.meshgrid(q, q, indexing="ij"))
    N = 0.25 * np.stack([(1 - xi) * (1 - eta), (1 + xi) * (1 - eta), (1 + xi) * (1 + eta), (1 - xi) * (1 + eta)])
    Nx = 0.25 * np.stack([-(1 - eta), 1 - eta, 1 + eta, -(1 + eta)])
    Ny = 0.25 * np.stack([-(1 - xi), -(1 + xi), 1 + xi, 1 - xi])
    xy, gx, gy = (np.einsum("kg,ckd->cgd", M, c) for M in (N, Nx, Ny))
    det = np.abs(gx[..., 0] * gy[..., 1] - gx[..., 1] * gy[..., 0])
    return xy.reshape(-1, 2).copy(), (det * np.outer(w, w).ravel()).ravel()


def _crease(kind, n, lo=0.0, hi=1.0):
    """Vertices of a straight crease half-way between two node columns (from lo to hi of the
    side) or of an arc about the origin that crosses the node layout freely."""
    side = (n - 1) * H
    if kind == "line":
        y = np.linspace(lo * side, hi * side, max(4, int(math.ceil((hi - lo) * side / H))) + 1)
        return np.stack([np.full(len(y), ((n - 1) // 2 + 0.5) * H), y], 1)
    R = 0.6 * side
    a = np.linspace(0.0, math.pi / 2, max(8, int(math.ceil(R * math.pi / H))) + 1)
    v = np.stack([R * np.cos(a), R * np.sin(a)], 1)
    v[0, 1] = v[-1, 0] = 0.0
    return v


def _cut(v, extend=True):
    return {"vertices": v, "extend_start": extend, "extend_end": extend, "is_closed": False}


def _sides(v):
    """Crease Gauss points: one per segment, both sides 1e-7 off the crease."""
    t = v[1:] - v[:-1]
    L = np.linalg.norm(t, axis=1)
    t = t / L[:, None]
    X, nrm = 0.5 * v[:-1] + 0.5 * v[1:], np.stack([-t[:, 1], t[:, 0]], 1)
    return X + 1e-7 * nrm, X - 1e-7 * nrm, L, t


def _field(nodes, side, rng, slope=math.tan(math.radians(60.0))):
    """A smooth displacement, eight plane waves per component: slopes of w up to 60 degrees."""
    out = []
    for c in range(3):
        th, ph, a = rng.uniform(0, 2 * math.pi, 8), rng.uniform(0, 2 * math.pi, 8), rng.normal(size=8)
        k = 2 * math.pi / rng.uniform(0.2 * side + 1.0, 2.0 * side + 1.0, 8)
        arg = np.outer(nodes[:, 0], k * np.cos(th)) + np.outer(nodes[:, 1], k * np.sin(th)) + ph
        g = np.hypot(np.cos(arg) @ (a * k * np.cos(th)), np.cos(arg) @ (a * k * np.sin(th))).max()
        out.append(np.sin(arg) @ a * (slope if c == 2 else 0.1 * slope) / g)
    return np.stack(out, 1).ravel()


def _layup(kind):
    """A, B, D: one isotropic ply, or two orthotropic plies at 20 and 70 degrees (B != 0)."""
    if kind == "isotropic":
        plies = [(E_MOD, E_MOD, NU, E_MOD / (2 * (1 + NU)), 0.0, THICK)]
    else:
        plies = [(1.0, 0.3, 0.3, 0.2, 20.0, 0.6 * THICK), (1.0, 0.3, 0.3, 0.2, 70.0, 0.4 * THICK)]
    A, B, D = (np.zeros((3, 3)) for _ in range(3))
    z = -THICK / 2.0
    for E1, E2, nu, G, ang, t in plies:
        den = 1.0 - nu * nu * E2 / E1
        Q = np.array([[E1, nu * E2, 0], [nu * E2, E2, 0], [0, 0, G * den]]) / den
        c, s = math.cos(math.radians(ang)), math.sin(math.radians(ang))
        T = np.array([[c * c, s * s, s * c], [s * s, c * c, -s * c], [-2 * s * c, 2 * s * c, c * c - s * s]])
        Qb = T.T @ Q @ T
        A += Qb * t
        if kind != "isotropic":
            B += 0.5 * Qb * ((z + t) ** 2 - z * z)
        D += Qb * ((z + t) ** 3 - z ** 3) / 3.0
        z += t
    return A, B, D


def _plate(n, rule, order, rho, window, crease, seed, cut=None):
    """One plate as plain arrays: the mesh by its size, the state (displacement, hinge stiffness)
    by the seed. cut: vertices of a cut that ends inside the plate."""
    rng = np.random.default_rng([seed, n])
    nodes = _nodes(n, np.random.default_rng(n), 0.2 * H)
    xy, w = _cells(nodes, n, rule)
    v = cut if cut is not None else None if crease == "none" else _crease(crease, n)
    return {"n": n, "nodes": nodes, "xy": xy, "w": w, "v": v, "cuts": [] if v is None else [_cut(v, cut is None)],
            "rho": rho * H, "order": order, "window": window, "Kt": 10.0 ** rng.uniform(-4, -1),
            "x": _field(nodes, (n - 1) * H, rng)}


def _plates(case, seed):
    if case["kind"] == "assemble":
        return [_plate(case["n_side"], case["rule"], case["order"], case["rho"], case["window"], case["crease"], seed)]
    if case["kind"] == "batch":
        sides = np.linspace(case["side_min"], case["side_max"], case["plates"]).round().astype(int)
        return [_plate(int(n), case["rule"], 2, 3.5, 0, ("line", "arc")[k % 2], seed + 1000 * k)
                for k, n in enumerate(sides)]
    n = case["n_side"]
    return [_plate(n, case["rule"], case["order"], case["rho"], case["window"], None, seed, _crease("line", n, 0.2, 0.7))]


def _moved(case, seed):
    """The cut after a tip move of a rebuild case: both tips by the seed."""
    rng = np.random.default_rng([seed, case["n_side"]])
    return [_cut(_crease("line", case["n_side"], rng.uniform(0.15, 0.25), rng.uniform(0.65, 0.85)), False)]


def _points(case, seed):
    """Scattered points over a node grid; the order of the points and the cut by the seed."""
    n, rng, own = case["n_side"], np.random.default_rng(case["n_side"]), np.random.default_rng(seed)
    nodes, side = _nodes(n, rng, 0.2 * H), (n - 1) * H
    xy = own.permutation(rng.uniform(0.0, side, (case["points"], 2)))
    y = ((n - 1) // 2 + own.uniform(0.3, 0.7)) * H
    rho_node = rng.uniform(2.7 * H, 3.5 * H, len(nodes)) if case["per_node"] else None
    return nodes, xy, rho_node, [_cut(np.array([[0.0, y], [side, y]]))]


# ---- the framework's side ----------------------------------------------------------------------

_streams = {}


def _stream():
    if "s" not in _streams:
        _streams["s"] = torch.cuda.Stream()
    return _streams["s"]


def _context():
    import curvami_gb300 as cg
    ctx = cg.Context(0)
    ctx.set_stream(_stream().cuda_stream)
    return ctx


def _as_plate(p):
    from curvami_gb300 import synth
    folds = []
    if p["v"] is not None:
        L, R, w, t = _sides(p["v"])
        folds.append(synth.Fold(synth.PointSet(L, w.copy(), t.copy()), synth.PointSet(R, w.copy(), t.copy()), p["Kt"]))
    return synth.Plate(name="case", node_xy=p["nodes"], faces=synth.PointSet(p["xy"], p["w"]), creases=p["cuts"],
                       folds=folds, rho=p["rho"], order=p["order"], kernel=p["window"], E=E_MOD, nu=NU, thickness=THICK)


class _View:
    """A device array of the library as a torch tensor; `keep` lives as long as the tensor."""

    def __init__(self, ptr, shape, typestr, keep):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _values(sh):
    """The device arrays of a shape set (cgb_shape_device)."""
    p = [ctypes.c_void_p() for _ in range(5)]
    sh.ctx.check(sh.ctx.lib.cgb_shape_device(sh.h, *[ctypes.addressof(q) for q in p]))
    k = sh.nnz
    shapes = [("ptr", (sh.n_gp + 1,), "<i8"), ("idx", (k,), "<i4"), ("psi", (k,), "<f8"), ("dpsi", (k, 2), "<f8"),
              ("ddpsi", (k, 3), "<f8")]
    return {name: torch.as_tensor(_View(q.value, shape, ty, sh), device="cuda") for q, (name, shape, ty) in zip(p, shapes)}


def _flags(case):
    import curvami_gb300 as cg
    f = cg.HINGE | (cg.TANGENT if case.get("want_K", True) else 0)
    if case.get("mode", "mixed") != "fp64":
        f |= cg.MIXED
    if case.get("mode") == "mixed_det":
        f |= cg.DETERMINISTIC
    if case.get("hinge_exact"):
        f |= cg.HINGE_EXACT
    return f


def prepare(case, seed):
    import curvami_gb300 as cg
    st = {"case": case}
    if case["kind"] == "shape":
        nodes, xy, rho_node, cuts = _points(case, seed)
        ctx = _context()
        ctx.set_nodes(nodes)
        st.update(ctx=ctx, xy=xy, kw=dict(rho=case["rho"] * H, order=case["order"], creases=cuts, rho_node=rho_node,
                                          kernel=case["window"], precision=case["precision"]))
        return st
    plates = _plates(case, seed)
    if case["kind"] == "batch":
        model = cg.PlateBatch([_as_plate(p) for p in plates], _context())
    else:
        model = cg.PlateModel(_as_plate(plates[0]), _context())
    st["model"] = model
    st["x"] = np.concatenate([p["x"] for p in plates])
    st["ABD"] = _layup(case.get("layup", "isotropic"))
    model.asm.set_material(*st["ABD"])
    if case["kind"] == "rebuild":
        st["cuts"] = _moved(case, seed)
    if case["kind"] == "batch" or case.get("io") == "device":
        with torch.cuda.stream(_stream()):
            st["xd"] = torch.from_numpy(st["x"]).cuda()
            st["Fd"] = torch.empty(model.asm.n_dofs, dtype=DOUBLE, device="cuda")
            if case.get("want_K", True):
                st["Kd"] = torch.empty(model.asm.nnz, dtype=DOUBLE, device="cuda")
            _stream().synchronize()
    if case["kind"] == "batch":
        st["graph"] = model.asm.graph(st["xd"].data_ptr(), st["Kd"].data_ptr(), st["Fd"].data_ptr(), _flags(case))
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "shape":
        import curvami_gb300 as cg
        return _values(cg.shape_functions(st["ctx"], st["xy"], **st["kw"]))
    model = st["model"]
    if case["kind"] == "rebuild":
        model.rebuild(st["cuts"])
        return [_values(sh) for sh in model.shape_sets()]
    if case["kind"] == "post":
        from curvami_gb300 import export
        return {"energies": np.array(model.asm.energies(st["x"])),
                "state": export.point_state(model.ctx, model.faces, st["x"], *st["ABD"])}
    mixed = case.get("mode", "mixed") != "fp64"
    if "graph" not in st and case["io"] == "host":
        K, F = model.asm.assemble(st["x"], _flags(case))
        out = {"F": F}
        if K is not None:
            out["K"] = K.astype(np.float32) if mixed else K
        return out
    if "graph" in st:
        st["graph"].launch()
    else:
        Kd = st.get("Kd")
        model.asm.assemble_device(st["xd"].data_ptr(), None if Kd is None else Kd.data_ptr(), st["Fd"].data_ptr(),
                                  _flags(case))
    out = {"F": st["Fd"]}
    if "Kd" in st:
        with torch.cuda.stream(_stream()):
            out["K"] = st["Kd"].float() if mixed else st["Kd"]
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------

def _neighbours(rho):
    return math.pi * rho * rho


def work(case):
    if case["kind"] in ("shape", "rebuild"):
        if case["kind"] == "shape":
            pts, n = case["points"], _neighbours(case["rho"])
        else:
            pts, n = (case["n_side"] - 1) ** 2 * case["rule"] ** 2, _neighbours(case["rho"])
        o = case["order"]
        np_, nr = (o + 1) * (o + 2) // 2, (2 * o + 1) * (2 * o + 2) // 2
        # per neighbour: six weight jets against the raw moments, six sums over the basis; per
        # point: one factorisation and six solves; neighbour index in or out, six values out
        return {"bytes": pts * (16 + 8 + n * (4 + 48)), "flops": pts * (n * (12 * nr + 12 * np_ + 60) + np_ ** 3 + 24 * np_ ** 2)}
    if case["kind"] == "batch":
        sides = np.linspace(case["side_min"], case["side_max"], case["plates"]).round()
        pts, nodes, rho = float(((sides - 1) ** 2).sum()) * case["rule"] ** 2, float((sides ** 2).sum()), 3.5
    else:
        n = case["n_side"]
        pts, nodes, rho = (n - 1) ** 2 * case["rule"] ** 2, n * n, case["rho"]
    n = _neighbours(rho)
    bytes_ = pts * n * 44 + 48 * nodes       # five derivatives and the index per neighbour, x in, F out
    if case["kind"] == "post":
        return {"bytes": pts * (n * 52 + 264) + 24 * nodes, "flops": pts * (36 * n + 250)}
    flops = pts * (60 * n + 300)             # kinematic sums and the nodal forces
    if case.get("want_K", True):
        blocks = nodes * 2.0 * math.pi * rho * rho      # a block column: half a disc of radius 2 rho
        bytes_ += blocks * (9 * 8 + 4)
        flops += pts * 72 * n * (n + 1) / 2             # 36 multiply-adds per 3x3 block of a pair
    return {"bytes": bytes_, "flops": flops}


# ---- exact: the method in plain torch, FP64 --------------------------------------------------------

def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _expand(count):
    """Row of every item, and its number within the row, of rows of `count` items."""
    row = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    start = torch.cumsum(count, 0) - count
    return row, torch.arange(len(row), device="cuda") - start[row]


def _gather(nodes, xy, rho):
    """Neighbour lists: nodes within the (node's) radius, in the order of the 3 x 3 cells
    around the point (x outer, y inner), ascending in a cell."""
    cell = float(rho.max()) if torch.is_tensor(rho) else rho
    lo = nodes.min(0).values
    cols = int(math.ceil(float(nodes[:, 0].max() - lo[0]) / cell)) + 1
    key = torch.floor((nodes - lo) / cell).long()
    key = key[:, 1] * cols + key[:, 0]
    by_key = torch.sort(key, stable=True)
    ncell = int(key.max()) + 1
    start = torch.searchsorted(by_key.values, torch.arange(ncell + 1, device="cuda"))
    q = torch.floor((xy - lo) / cell).long()
    r2 = rho * rho if torch.is_tensor(rho) else torch.full((len(nodes),), rho * rho, dtype=DOUBLE, device="cuda")
    gs, js = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            k = (q[:, 1] + dy) * cols + q[:, 0] + dx
            ok = (k >= 0) & (k < ncell)
            k = torch.where(ok, k, torch.zeros_like(k))
            g, at = _expand(torch.where(ok, start[k + 1] - start[k], torch.zeros_like(k)))
            j = by_key.indices[start[k][g] + at]
            d = nodes[j] - xy[g]
            d = d * d
            m = d[:, 0] + d[:, 1] <= r2[j]
            gs.append(g[m])
            js.append(j[m])
    g, order = torch.sort(torch.cat(gs), stable=True)
    idx = torch.cat(js)[order]
    ptr = torch.zeros(len(xy) + 1, dtype=torch.long, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(g, minlength=len(xy)), 0)
    return ptr, idx


def _indicator(P, cut):
    """Side function of a crease and its derivatives at the points P: f, fx, fy, fxx, fyy, fxy."""
    V = _dev(cut["vertices"])
    A, v = V[:-1], V[1:] - V[:-1]
    v2 = (v * v).sum(1)
    out = torch.zeros((len(P), 6), dtype=DOUBLE, device="cuda")
    tmin = torch.zeros(len(A), dtype=DOUBLE, device="cuda")
    tmax = torch.ones(len(A), dtype=DOUBLE, device="cuda")
    if cut["extend_start"]:
        tmin[0] = -math.inf
    if cut["extend_end"]:
        tmax[-1] = math.inf
    for c0 in range(0, len(P), 200000):
        p = P[c0:c0 + 200000]
        t = ((p[:, None, :] - A) * v).sum(2) / v2
        t = torch.minimum(torch.maximum(t, tmin), tmax)
        C = A + t[..., None] * v
        d2 = ((p[:, None, :] - C) ** 2).sum(2)
        near = (d2 == d2.min(1, keepdim=True).values).to(torch.int8).argmax(1)
        row = torch.arange(len(p), device="cuda")
        C, t, d = C[row, near], t[row, near], torch.sqrt(d2[row, near])
        u = (p - C) / d[:, None]
        n = torch.stack([-v[near, 1], v[near, 0]], 1) / torch.sqrt(v2[near])[:, None]
        f = (u * n).sum(1)
        cap = ((near == 0) & (t == 0.0) & (not cut["extend_start"])) | ((near == len(A) - 1) & (t == 1.0) & (not cut["extend_end"]))
        side = torch.where(f >= 0, 1.0, -1.0).to(DOUBLE)
        full = torch.stack([f, (n[:, 0] - f * u[:, 0]) / d, (n[:, 1] - f * u[:, 1]) / d,
                            (3 * f * u[:, 0] ** 2 - 2 * n[:, 0] * u[:, 0] - f) / d ** 2,
                            (3 * f * u[:, 1] ** 2 - 2 * n[:, 1] * u[:, 1] - f) / d ** 2,
                            (3 * f * u[:, 0] * u[:, 1] - n[:, 0] * u[:, 1] - u[:, 0] * n[:, 1]) / d ** 2], 1)
        plain = torch.zeros_like(full)
        plain[:, 0] = side
        out[c0:c0 + 200000] = torch.where(cap[:, None], full, plain)
    return out


def _window(kind, s):
    if kind == 0:
        return 1 - 6 * s ** 2 + 8 * s ** 3 - 3 * s ** 4, -12 * s + 24 * s ** 2 - 12 * s ** 3, -12 + 48 * s - 36 * s ** 2
    r, lo = 1 - s, s <= 0.5
    return (torch.where(lo, 2.0 / 3.0 - 4 * s ** 2 + 4 * s ** 3, 4.0 / 3.0 * r ** 3),
            torch.where(lo, -8 * s + 12 * s ** 2, -4 * r ** 2), torch.where(lo, -8 + 24 * s, 8 * r))


def _basis(order, x, y):
    """Monomials of degree <= order and their derivatives: p, px, py, pxx, pyy, pxy."""
    def mono(a, b, ca=1.0):
        return torch.zeros_like(x) if a < 0 or b < 0 else ca * x ** a * y ** b
    out = [[], [], [], [], [], []]
    for d in range(order + 1):
        for b in range(d + 1):
            a = d - b
            for o, (i, j, k) in zip(out, [(a, b, 1.0), (a - 1, b, a), (a, b - 1, b), (a - 2, b, a * (a - 1)),
                                          (a, b - 2, b * (b - 1)), (a - 1, b - 1, a * b)]):
                o.append(mono(i, j, float(k)))
    return [torch.stack(o, 1) for o in out]


def _outer(a, b):
    return a[:, :, None] * b[:, None, :]


def _shape_exact(nodes, xy, rho, rho_node, order, window, cuts):
    """Reproducing-kernel shape functions with crease visibility: neighbour lists, values,
    gradients and Hessians (xx, yy, xy)."""
    nodes, xy = _dev(nodes), _dev(xy)
    rn = None if rho_node is None else _dev(rho_node)
    ptr, idx = _gather(nodes, xy, rho if rn is None else rn)
    psi = torch.empty(len(idx), dtype=DOUBLE, device="cuda")
    dpsi = torch.empty((len(idx), 2), dtype=DOUBLE, device="cuda")
    ddpsi = torch.empty((len(idx), 3), dtype=DOUBLE, device="cuda")
    inds = [_indicator(xy, c) for c in cuts]
    sides = [torch.where(_indicator(nodes, c)[:, 0] >= 0, 1.0, -1.0).to(DOUBLE) for c in cuts]
    step = 40000 if order < 3 else 8000
    bounds = ptr[torch.arange(0, len(xy) + step, step, device="cuda").clamp(max=len(xy))].tolist()
    for c, (e0, e1) in enumerate(zip(bounds[:-1], bounds[1:])):
        g0, g1 = c * step, min(len(xy), (c + 1) * step)
        if g1 <= g0:
            break
        g, _ = _expand(ptr[g0 + 1:g1 + 1] - ptr[g0:g1])
        j = idx[e0:e1]
        X = xy[g0:g1]
        d = (X[g] - nodes[j]) / rho
        xi, eta = d[:, 0], d[:, 1]
        fac = torch.ones_like(xi) if rn is None else rho / rn[j]
        zx, zy = xi * fac, eta * fac
        s = torch.sqrt(zx * zx + zy * zy)
        w, d1, d2 = _window(window, s)
        inv = torch.where(s == 0, torch.zeros_like(s), 1.0 / s)
        dx, dy = zx * inv, zy * inv
        J = [w, d1 * dx * fac, d1 * dy * fac,
             torch.where(s == 0, d1 * d2, d2 * dx * dx + d1 * zx * zx * inv ** 3) * fac * fac,
             torch.where(s == 0, d1 * d2, d2 * dy * dy + d1 * zy * zy * inv ** 3) * fac * fac,
             (d2 * dx * dy - d1 * zx * zy * inv ** 3) * fac * fac]
        J = [torch.where(s < 1, a, torch.zeros_like(a)) for a in J]
        for I, sn in zip(inds, sides):
            I, sn = I[g0:g1][g], sn[j]
            W = 0.5 * (1 + sn * I[:, 0])
            Wx, Wy = (0.5 * sn * I[:, k] * rho for k in (1, 2))
            Wxx, Wyy, Wxy = (0.5 * sn * I[:, k] * rho * rho for k in (3, 4, 5))
            o = J
            J = [o[0] * W, o[1] * W + o[0] * Wx, o[2] * W + o[0] * Wy, o[3] * W + 2 * o[1] * Wx + o[0] * Wxx,
                 o[4] * W + 2 * o[2] * Wy + o[0] * Wyy, o[5] * W + o[1] * Wy + o[2] * Wx + o[0] * Wxy]
        p, px, py, pxx, pyy, pxy = _basis(order, xi, eta)

        def summed(v):
            return torch.zeros((g1 - g0,) + tuple(v.shape[1:]), dtype=DOUBLE, device="cuda").index_add_(0, g, v)

        def sym(a, b):
            o = _outer(a, b)
            return o + o.transpose(1, 2)

        c3 = [a[:, None, None] for a in J]
        pp, sx, sy = _outer(p, p), sym(px, p), sym(py, p)
        M = summed(c3[0] * pp)
        Mx = summed(c3[1] * pp + c3[0] * sx)
        My = summed(c3[2] * pp + c3[0] * sy)
        Mxx = summed(c3[3] * pp + 2 * c3[1] * sx + c3[0] * (sym(pxx, p) + 2 * _outer(px, px)))
        Myy = summed(c3[4] * pp + 2 * c3[2] * sy + c3[0] * (sym(pyy, p) + 2 * _outer(py, py)))
        Mxy = summed(c3[5] * pp + c3[1] * sy + c3[2] * sx + c3[0] * (sym(pxy, p) + sym(px, py)))
        del pp, sx, sy, c3
        LU = torch.linalg.lu_factor(M)

        def solve(r):
            return torch.linalg.lu_solve(*LU, r[:, :, None])[:, :, 0]

        def mul(S, r):
            return (S * r[:, None, :]).sum(2)

        e0v = torch.zeros((g1 - g0, M.shape[1]), dtype=DOUBLE, device="cuda")
        e0v[:, 0] = 1.0
        b = solve(e0v)
        bx, by = solve(-mul(Mx, b)), solve(-mul(My, b))
        bxx, byy = solve(-mul(Mxx, b) - 2 * mul(Mx, bx)), solve(-mul(Myy, b) - 2 * mul(My, by))
        bxy = solve(-mul(Mxy, b) - mul(Mx, by) - mul(My, bx))
        dot = lambda u, q: (u[g] * q).sum(1)  # noqa: E731
        C = dot(b, p)
        Cx, Cy = dot(bx, p) + dot(b, px), dot(by, p) + dot(b, py)
        Cxx = dot(bxx, p) + 2 * dot(bx, px) + dot(b, pxx)
        Cyy = dot(byy, p) + 2 * dot(by, py) + dot(b, pyy)
        Cxy = dot(bxy, p) + dot(bx, py) + dot(by, px) + dot(b, pxy)
        w, wx, wy, wxx, wyy, wxy = J
        psi[e0:e1] = C * w
        dpsi[e0:e1] = torch.stack([Cx * w + C * wx, Cy * w + C * wy], 1) / rho
        ddpsi[e0:e1] = torch.stack([Cxx * w + 2 * Cx * wx + C * wxx, Cyy * w + 2 * Cy * wy + C * wyy,
                                    Cxy * w + Cx * wy + Cy * wx + C * wxy], 1) / rho ** 2
    return {"ptr": ptr, "idx": idx, "psi": psi, "dpsi": dpsi, "ddpsi": ddpsi}


def _of_plate(p, xy, cuts=None):
    return _shape_exact(p["nodes"], xy, p["rho"], None, p["order"], p["window"], p["cuts"] if cuts is None else cuts)


def _state(S, x, A, B, D):
    """Kinematics and resultants at every point of a shape set."""
    n = len(S["ptr"]) - 1
    g, _ = _expand(S["ptr"][1:] - S["ptr"][:-1])
    u = x[S["idx"]]
    add = lambda c: torch.zeros((n, 3), dtype=DOUBLE, device="cuda").index_add_(0, g, u * c[:, None])  # noqa: E731
    k = {"g": g, "u": add(S["psi"]), "rxx": add(S["ddpsi"][:, 0]), "ryy": add(S["ddpsi"][:, 1]), "rxy": add(S["ddpsi"][:, 2])}
    k["a1"], k["a2"] = add(S["dpsi"][:, 0]), add(S["dpsi"][:, 1])
    k["a1"][:, 0] += 1.0
    k["a2"][:, 1] += 1.0
    dot = lambda a, b: (a * b).sum(1)  # noqa: E731
    C00, C11, C01 = dot(k["a1"], k["a1"]), dot(k["a2"], k["a2"]), dot(k["a1"], k["a2"])
    det = C00 * C11 - C01 * C01
    k["Ci"] = torch.stack([C11, -C01, -C01, C00], 1) / det[:, None]
    nrm = torch.linalg.cross(k["a1"], k["a2"])
    k["b"] = nrm / torch.sqrt(dot(nrm, nrm))[:, None]
    k["e0"] = torch.stack([0.5 * (C00 - 1), 0.5 * (C11 - 1), C01], 1)
    k["e1"] = torch.stack([-dot(k["rxx"], k["b"]), -dot(k["ryy"], k["b"]), -2 * dot(k["rxy"], k["b"])], 1)
    A, B, D = (_dev(m) for m in (A, B, D))
    k["N"], k["M"] = k["e0"] @ A.T + k["e1"] @ B.T, k["e0"] @ B + k["e1"] @ D.T
    return k


def _angle(F, t):
    a1L, a2L, a1R, a2R = F[:, 0:3], F[:, 3:6], F[:, 6:9], F[:, 9:12]
    unit = lambda v: v / torch.sqrt((v * v).sum(1, keepdim=True))  # noqa: E731
    bL, bR = unit(torch.linalg.cross(a1L, a2L)), unit(torch.linalg.cross(a1R, a2R))
    tt = unit(a1L * t[:, :1] + a2L * t[:, 1:])
    return torch.atan2(-(torch.linalg.cross(bL, bR) * tt).sum(1), (bL * bR).sum(1))


def _hinge(p, x, want_hess):
    """Per merged (crease point, node): point, node, force, the dof gradient G and the sums Bs;
    and per point the hinge's factors and Hessian; and the hinge energy."""
    L, R, w, t = _sides(p["v"])
    w, t = _dev(w), _dev(t)
    m, N = len(w), len(p["nodes"])
    SL, SR = _of_plate(p, L), _of_plate(p, R)
    F = torch.zeros((m, 12), dtype=DOUBLE, device="cuda")
    F[:, [0, 4, 6, 10]] = 1.0
    parts = []
    for k, S in enumerate((SL, SR)):
        g, _ = _expand(S["ptr"][1:] - S["ptr"][:-1])
        parts.append((g, S["idx"], S["dpsi"]))
        for q in range(2):
            F[:, 6 * k + 3 * q:6 * k + 3 * q + 3].index_add_(0, g, x[S["idx"]] * S["dpsi"][:, q:q + 1])
    F.requires_grad_(True)
    th = _angle(F, t)
    grad = torch.autograd.grad(th.sum(), F, create_graph=want_hess)[0]
    hess = torch.stack([torch.autograd.grad(grad[:, q].sum(), F, retain_graph=True)[0] for q in range(12)], 1) if want_hess else None
    th, grad = th.detach(), grad.detach()
    key = torch.cat([g * N + j for g, j, _ in parts])
    uniq, inv = torch.unique(key, return_inverse=True)
    G = torch.zeros((len(uniq), 3), dtype=DOUBLE, device="cuda")
    Bs = torch.zeros((len(uniq), 4), dtype=DOUBLE, device="cuda")
    at = 0
    for k, (g, j, d) in enumerate(parts):
        u = inv[at:at + len(g)]
        at += len(g)
        G.index_add_(0, u, grad[g, 6 * k:6 * k + 3] * d[:, :1] + grad[g, 6 * k + 3:6 * k + 6] * d[:, 1:])
        Bs[:, 2 * k:2 * k + 2].index_add_(0, u, d)
    return {"point": uniq // N, "node": uniq % N, "G": G, "Bs": Bs, "Wm": w * p["Kt"] * th, "WK": w * p["Kt"], "H": hess,
            "E": (0.5 * w * p["Kt"] * th * th).sum()}


def _pairs(ptr, e0, e1):
    """Local pairs i <= j (as entries) of the lists of the entries [e0, e1)."""
    e = torch.arange(e0, e1, device="cuda")
    end = ptr[torch.searchsorted(ptr, e, right=True)]
    row, at = _expand(end - e)
    return e[row], e[row] + at


def _assembly_exact(plates, ABD, want_K, exact_hinge):
    nodes = [len(p["nodes"]) for p in plates]
    off = np.concatenate([[0], np.cumsum(nodes)])
    N = int(off[-1])
    F = torch.zeros((N, 3), dtype=DOUBLE, device="cuda")
    keys, sums = [], []
    A, B, D = (_dev(m) for m in ABD)
    for p, o in zip(plates, off):
        o = int(o)
        x = _dev(p["x"].reshape(-1, 3))
        S, W = _of_plate(p, p["xy"]), _dev(p["w"])
        k = _state(S, x, *ABD)
        g = k["g"]
        dx, dy = S["dpsi"][:, 0], S["dpsi"][:, 1]
        dxx, dyy, dxy = (S["ddpsi"][:, q] for q in range(3))
        c0 = k["Ci"][g, 0] * dx + k["Ci"][g, 1] * dy
        c1 = k["Ci"][g, 2] * dx + k["Ci"][g, 3] * dy
        gI = k["a1"][g] * c0[:, None] + k["a2"][g] * c1[:, None]
        dot = lambda a, b: (a * b).sum(1)  # noqa: E731
        beta = torch.stack([-dxx + dot(k["rxx"][g], gI), -dyy + dot(k["ryy"][g], gI), 2 * (-dxy + dot(k["rxy"][g], gI))], 1)
        Tu = dot(beta, k["M"][g])
        f = (k["a1"][g] * (dx * k["N"][g, 0] + dy * k["N"][g, 2])[:, None]
             + k["a2"][g] * (dy * k["N"][g, 1] + dx * k["N"][g, 2])[:, None] + k["b"][g] * Tu[:, None])
        F[o:o + len(x)].index_add_(0, S["idx"], f * W[g][:, None])
        if want_K:
            Bm = torch.stack([k["a1"][g] * dx[:, None], k["a2"][g] * dy[:, None],
                              k["a1"][g] * dy[:, None] + k["a2"][g] * dx[:, None]], 1)
            Bb = beta[:, :, None] * k["b"][g][:, None, :]
            P = torch.einsum("rs,esc->erc", A, Bm) + torch.einsum("rs,esc->erc", B, Bb)
            Q = torch.einsum("sr,esc->erc", B, Bm) + torch.einsum("rs,esc->erc", D, Bb)
            vc = k["rxx"] * k["M"][:, :1] + k["ryy"] * k["M"][:, 1:2] + 2 * k["rxy"] * k["M"][:, 2:3]
            bv = dot(k["b"], vc)[g]
            nj = torch.stack([k["N"][g, 0] * dx + k["N"][g, 2] * dy, k["N"][g, 2] * dx + k["N"][g, 1] * dy], 1)
            total = len(g)
            mean = max(1.0, total / (len(S["ptr"]) - 1))
            step = max(1000, int(4e6 / mean))
            for e0 in range(0, total, step):
                a, b = _pairs(S["ptr"], e0, min(total, e0 + step))
                Kb = (torch.einsum("erc,erd->ecd", Bm[a], P[b]) + torch.einsum("erc,erd->ecd", Bb[a], Q[b]))
                bb = k["b"][g[a]]
                Kb -= Tu[a][:, None, None] * _outer(gI[b], bb)
                Kb -= Tu[b][:, None, None] * _outer(bb, gI[a])
                Kb += (bv[a] * (dx[a] * c0[b] + dy[a] * c1[b]))[:, None, None] * _outer(bb, bb)
                Kb += (dx[a] * nj[b, 0] + dy[a] * nj[b, 1])[:, None, None] * torch.eye(3, dtype=DOUBLE, device="cuda")
                Kb *= W[g[a]][:, None, None]
                ni, nj_ = S["idx"][a], S["idx"][b]
                Kb = torch.where((ni > nj_)[:, None, None], Kb.transpose(1, 2), Kb)
                key = (torch.maximum(ni, nj_) + o) * N + torch.minimum(ni, nj_) + o
                u, inv = torch.unique(key, return_inverse=True)
                keys.append(u)
                sums.append(torch.zeros((len(u), 9), dtype=DOUBLE, device="cuda").index_add_(0, inv, Kb.reshape(-1, 9)))
        if p["v"] is not None:
            h = _hinge(p, x, want_K and exact_hinge)
            F[o:o + len(x)].index_add_(0, h["node"], h["G"] * h["Wm"][h["point"]][:, None])
            if want_K:
                hp = torch.zeros(int(h["point"].max()) + 2, dtype=torch.long, device="cuda")
                hp[1:] = torch.cumsum(torch.bincount(h["point"]), 0)
                for e0 in range(0, len(h["point"]), 20000):
                    a, b = _pairs(hp, e0, min(len(h["point"]), e0 + 20000))
                    Kb = _outer(h["G"][a], h["G"][b]) * h["WK"][h["point"][a]][:, None, None]
                    if h["H"] is not None:
                        Hs = h["H"][h["point"][a]].reshape(-1, 4, 3, 4, 3)
                        Kb += h["Wm"][h["point"][a]][:, None, None] * torch.einsum("es,escud,eu->ecd", h["Bs"][a], Hs, h["Bs"][b])
                    key = (h["node"][b] + o) * N + h["node"][a] + o
                    u, inv = torch.unique(key, return_inverse=True)
                    keys.append(u)
                    sums.append(torch.zeros((len(u), 9), dtype=DOUBLE, device="cuda").index_add_(0, inv, Kb.reshape(-1, 9)))
    out = {"F": F.reshape(-1)}
    if want_K:
        # the block-upper CSC values: scalar column 3j + c lists the rows 3i + r of its blocks
        blocks, inv = torch.unique(torch.cat(keys), return_inverse=True)
        K = torch.zeros((len(blocks), 9), dtype=DOUBLE, device="cuda").index_add_(0, inv, torch.cat(sums))
        col = blocks // N
        length = torch.bincount(col, minlength=N)
        first = torch.cumsum(length, 0) - length
        pos = torch.arange(len(blocks), device="cuda") - first[col]
        values = torch.empty(9 * len(blocks), dtype=DOUBLE, device="cuda")
        for r in range(3):
            for c in range(3):
                values[9 * first[col] + 3 * c * length[col] + 3 * pos + r] = K[:, 3 * r + c]
        out["K"] = values
    return out


def exact(case, seed):
    if case["kind"] == "shape":
        nodes, xy, rho_node, cuts = _points(case, seed)
        S = _shape_exact(nodes, xy, case["rho"] * H, rho_node, case["order"], case["window"], cuts)
        return {"ptr": None, "idx": None, **{k: S[k] for k in ("psi", "dpsi", "ddpsi")}}
    plates = _plates(case, seed)
    if case["kind"] == "rebuild":
        p, cuts = plates[0], _moved(case, seed)
        L, R, _, _ = _sides(p["v"])
        sets = [_of_plate(p, xy, cuts) for xy in (p["xy"], L, R)]
        return [{"ptr": None, "idx": None, **{k: S[k] for k in ("psi", "dpsi", "ddpsi")}} for S in sets]
    if case["kind"] == "post":
        p = plates[0]
        x, ABD = _dev(p["x"].reshape(-1, 3)), _layup("isotropic")
        k, W = _state(_of_plate(p, p["xy"]), x, *ABD), _dev(p["w"])
        half = torch.tensor([1.0, 1.0, 0.5], dtype=DOUBLE, device="cuda")
        state = torch.cat([k["u"], k["a1"], k["a2"], k["rxx"], k["ryy"], k["rxy"], k["b"], k["e0"] * half, k["e1"] * half,
                           k["N"], k["M"]], 1)
        em, eb = (0.5 * W * (k["e0"] * k["N"]).sum(1)).sum(), (0.5 * W * (k["e1"] * k["M"]).sum(1)).sum()
        return {"energies": torch.stack([em, eb, _hinge(p, x, False)["E"]]), "state": state}
    return _assembly_exact(plates, _layup(case.get("layup", "isotropic")), case.get("want_K", True), case.get("hinge_exact", False))
