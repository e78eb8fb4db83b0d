"""The work that users of this library have it do, as timed cases.

Every case goes through the public classes (`SDF3`, `VesicleBatch`, `Transport`).  Fields are
noisy ellipsoidal vesicles of the sizes that the repository's own workloads, tests and
recorded histories use, and odd and anisotropic grids between them.  `exact` restates the
operations in FP64 with plain torch (class `Exact`).
"""
import importlib
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

PKG = "2018_7_vesicle_gb300"


def _mod(name=""):
    return importlib.import_module(PKG + ("." + name if name else ""))


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------


def _grid(rows, cols, pges):
    return {"rows": rows, "cols": cols, "pges": pges}


def listed():
    return [
        # the smallest call: a driver that watches area and volume after every step
        {"name": "area_volume_f64_48", "op": "area_volume", "prec": "f64", **_grid(48, 48, 48)},
        # the reinitialization of a non-distance sphere, the FP64 form's workload at 64^3
        {"name": "reinit_f64_64", "op": "reinit", "scheme": "weno5", "prec": "f64", "iters": 100, **_grid(64, 64, 64)},
        # one vesicle step in the plain FP64 form at 128^3
        {"name": "step_f64_128", "op": "step", "prec": "f64", "ext": 30, "iters": 20, "graph": False,
         **_grid(128, 128, 128)},
        # the headline workload: one vesicle step in the mixed form at 256^3, replayed as a graph
        {"name": "step_f32_256", "op": "step", "prec": "f32", "ext": 30, "iters": 20, "graph": True,
         **_grid(256, 256, 256)},
        # 64 vesicles of uneven sizes advanced together
        {"name": "batch_f32_64", "op": "batch", "prec": "f32", "ext": 30, "iters": 20, "count": 64, "lo": 48, "hi": 160},
        # the relaxation driver's step at its own 96^3 configuration, mixed form, as a graph
        {"name": "relax_f32_96", "op": "relax", "prec": "f32", "ext": 100, "iters": 100, "graph": True,
         **_grid(96, 96, 96)},
        # the relaxation step that reproduces the recorded FP64 histories (64^3)
        {"name": "relax_f64_64", "op": "relax", "prec": "f64", "ext": 100, "iters": 100, "graph": False,
         **_grid(64, 64, 64)},
        # differentiation: transport forward and its adjoint, 40 steps with reinitialization
        {"name": "transport_f32_128", "op": "transport", "prec": "f32", "steps": 40, "every": 10, "iters": 10,
         **_grid(128, 128, 128)},
        # all fields of the auxiliary (domain) toolbox of a multiphase vesicle
        {"name": "aux_toolbox_f32_256", "op": "aux", "prec": "f32", **_grid(256, 256, 256)},
        # redistancing a surface field on the interface, an odd anisotropic box
        {"name": "redistance_f32_odd", "op": "redistance", "scheme": "weno5", "prec": "f32", "iters": 10, "ext": 5,
         **_grid(161, 113, 97)},
        # extension of a curvature-like field with the WENORK3 scheme on a small ragged grid
        {"name": "extend_f32_odd", "op": "extend", "scheme": "eno3", "prec": "f32", "ext": 30, **_grid(61, 83, 45)},
        # advection by a given velocity in the plain form on an odd grid
        {"name": "advect_f64_odd", "op": "advect", "prec": "f64", "steps": 4, **_grid(111, 95, 127)},
    ]


def _stages(c):
    """RK stages of a case's loops (what its cost follows)."""
    op = c["op"]
    if op in ("reinit", "extend"):
        n = c["iters"] if op == "reinit" else c["ext"]
        return n * (2 if c["scheme"] == "enork2" else 3)
    if op == "advect":
        return 3 * c["steps"]
    if op in ("step", "batch"):
        return 3 * (c["ext"] + 1 + c["iters"])
    if op == "relax":
        return 7 * c["ext"] + 3 * c["iters"]
    if op == "redistance":
        per = 2 if c["scheme"] == "enork2" else 3
        return c["iters"] * per * (per * c["ext"] + 1) + per * c["ext"]
    if op == "transport":
        # the forward pass, its recomputation and an adjoint worth several forward stages
        return 10 * 3 * (c["steps"] + c["steps"] // max(1, c["every"]) * c["iters"])
    return 3


def _nodes(c):
    if c["op"] == "batch":
        return sum(math.prod(s) for s, _ in _batch_shapes(c))
    return c["rows"] * c["cols"] * c["pges"]


def draw(rng):
    """One more case: an operation, a precision and sizes over their whole range."""
    op = rng.choice(["area_volume", "toolbox", "aux", "reinit", "reinit", "extend", "extend", "advect", "redistance",
                     "step", "step", "relax", "batch", "transport"])
    c = {"op": op, "prec": rng.choice(["f32", "f64"])}
    if op in ("reinit", "extend", "redistance"):
        c["scheme"] = rng.choice(["weno5", "eno3", "enork2"])
    if op in ("step", "relax"):
        c["graph"] = rng.choice([True, False])
    if op in ("batch", "transport"):
        c["prec"] = "f32"
    f64 = c["prec"] == "f64"
    hi = {"relax": 64 if f64 else 128, "redistance": 72 if f64 else 176, "transport": 128}.get(op, 128 if f64 else 256)
    if op == "batch":
        c |= {"ext": rng.randint(5, 30), "iters": rng.randint(5, 20), "count": rng.randint(3, 48), "lo": 40, "hi": 144}
        return c

    def size():
        return int(round(math.exp(rng.uniform(math.log(24), math.log(hi)))))

    n = size()
    for axis in ("rows", "cols", "pges"):
        c[axis] = max(24, min(hi, int(round(n * rng.uniform(0.75, 1.33)))))
    if op == "reinit":
        c["iters"] = rng.randint(5, 100)
    elif op == "extend":
        c["ext"] = rng.randint(5, 60)
    elif op == "advect":
        c["steps"] = rng.randint(1, 10)
    elif op == "redistance":
        c |= {"iters": rng.randint(2, 10), "ext": rng.randint(2, 5)}
    elif op == "step":
        c |= {"ext": rng.randint(5, 30), "iters": rng.randint(5, 20)}
    elif op == "relax":
        c |= {"ext": rng.randint(10, 100), "iters": rng.choice([0, 20, 100])}
    elif op == "transport":
        c |= {"steps": rng.randint(4, 40), "every": rng.choice([5, 10, 50]), "iters": rng.randint(3, 10)}
    # no dearer than the largest listed case of the precision
    most = (2.0e6 * 160) if f64 else (16.8e6 * 160)
    for key in ("iters", "ext", "steps"):
        if key in c and _nodes(c) * _stages(c) > most:
            c[key] = max(1, int(c[key] * most / (_nodes(c) * _stages(c))))
    return c


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------

DT = {"f32": torch.float32, "f64": torch.float64}


def _mesh(c, half=(1.5, 1.5, 1.5)):
    """Node coordinates and spacings of a box [-half, half] (x: columns, y: rows, z: pages)."""
    v = [np.linspace(-half[a], half[a], c[k]) for a, k in enumerate(("cols", "rows", "pges"))]
    x, y, z = _mod("shapes").meshgrid(*v, device="cuda")
    return x, y, z, tuple(float(a[1] - a[0]) for a in v)


def _box(c, reach=1.5):
    """A box whose spacings are near each other: the longest axis reaches `reach`."""
    n = max(c["rows"], c["cols"], c["pges"])
    return tuple(max(1.15, reach * c[k] / n) for k in ("cols", "rows", "pges"))


def _noise(x, y, z, seed, amplitude, modes=6):
    g = np.random.default_rng(seed)
    out = torch.zeros_like(x)
    for _ in range(modes):
        k, ph = g.uniform(-2.5, 2.5, 3), g.uniform(0, 2 * math.pi)
        out += float(g.uniform(0.3, 1.0)) * torch.sin(float(k[0]) * x + float(k[1]) * y + float(k[2]) * z + float(ph))
    return out * (amplitude / modes)


def _distance_like(x, y, z, axes, seed, amplitude=0.03):
    """A field near the signed distance of a perturbed ellipsoid: (q - 1) q / |(x/a^2, ..)|."""
    a, b, c = axes
    q = torch.sqrt(x**2 / a**2 + y**2 / b**2 + z**2 / c**2)
    s = torch.sqrt(x**2 / a**4 + y**2 / b**4 + z**2 / c**4)
    return (q - 1) * q / torch.clamp(s, min=1e-3) + _noise(x, y, z, seed, amplitude)


def _axes(seed, lo=0.62, hi=0.95):
    g = np.random.default_rng(seed + 77)
    return tuple(float(v) for v in g.uniform(lo, hi, 3))


def _batch_shapes(c):
    """((rows, cols, pges), half axes) of every member: edges spread over [lo, hi]."""
    g = np.random.default_rng(1000 * c["count"] + c["lo"] + c["hi"])
    out = []
    for _ in range(c["count"]):
        s = tuple(int(v) for v in np.round(np.exp(g.uniform(math.log(c["lo"]), math.log(c["hi"]), 3))))
        out.append((s, tuple(float(v) for v in g.uniform(0.4, 1.0, 3))))
    return out


def _initial(c, seed):
    """The level set that the case starts from (FP64, then in the case's precision), and mesh."""
    op = c["op"]
    if op == "step":
        # oblate vesicle of reduced volume 0.65 with spherical-harmonic noise, not a distance
        S = _mod("shapes")
        x, y, z, h = _mesh(c)
        F = S.noisy_oblate(x, y, z, axes=(1.0, 1.0, S.oblate_c_for_reduced_volume(0.65)), seed=seed)
    elif op == "reinit":
        x, y, z, h = _mesh(c, (1.0, 1.0, 1.0))
        g = np.random.default_rng(seed)
        o = [float(v) for v in g.uniform(-0.05, 0.05, 3)]
        r = float(g.uniform(0.55, 0.65))
        F = (torch.sqrt((x - o[0])**2 + (y - o[1])**2 + (z - o[2])**2) - r) * (
            0.1 + (x - 0.35)**2 + (y - 0.35)**2 + (z - 0.35)**2)
    elif op == "relax":
        x, y, z, h = _mesh(c, (1.0, 1.0, 1.0))
        g = np.random.default_rng(seed)
        F = _distance_like(x, y, z, (0.62, 0.62, float(g.uniform(0.38, 0.46))), seed, 0.01)
    else:
        x, y, z, h = _mesh(c, _box(c))
        F = _distance_like(x, y, z, _axes(seed), seed)
    return x, y, z, h, _colmajor(F, DT[c["prec"]])


def _colmajor(t, dtype):
    return t.to(dtype).permute(2, 1, 0).contiguous().permute(2, 1, 0)


def _surface_field(x, y, z, seed):
    g = np.random.default_rng(seed + 5)
    p = [float(v) for v in g.uniform(0, 1, 2)]
    return torch.sin(3 * x + p[0]) * torch.cos(2 * y + p[1]) + 0.5 * z**2


def _curvature_like(x, y, z, seed):
    return 2.0 / torch.sqrt(x**2 + y**2 + z**2 + 0.3) + _noise(x, y, z, seed + 9, 2.0)


def _velocity_of(x, y, z, seed):
    g = np.random.default_rng(seed + 13)
    p = [float(v) for v in g.uniform(0, 2 * math.pi, 3)]
    return (torch.sin(2 * y + p[0]) * torch.cos(z), torch.sin(2 * z + p[1]) * torch.cos(x),
            torch.sin(2 * x + p[2]) * torch.cos(y))


def _domain(x, y, z, seed):
    g = np.random.default_rng(seed + 21)
    n = [float(v) for v in g.uniform(-0.3, 0.3, 2)]
    return z + n[0] * x + n[1] * y - float(g.uniform(0.1, 0.25)) + 0.12 * torch.sin(2 * x + y + 0.7 * z)


def _transport_data(c, seed):
    x, y, z, h = _mesh(c, _box(c))
    phi0 = _colmajor(_distance_like(x, y, z, _axes(seed, 0.55, 0.8), seed), DT[c["prec"]])
    g = np.random.default_rng(seed + 31)
    amp = [float(v) for v in g.normal(0.0, 0.1, 3)]
    v = [_colmajor(a * u, DT[c["prec"]]) for a, u in zip((0.25 + amp[0], 0.2 + amp[1], 0.2 + amp[2]),
                                                         _velocity_of(x, y, z, seed))]
    dt = 0.5 * min(h) / max(1e-3, max(float(t.abs().max()) for t in v))
    target = _colmajor(_distance_like(x, y, z, _axes(seed + 1, 0.55, 0.8), seed + 1), torch.float64)
    return x, y, z, h, phi0, v, dt, target


def prepare(case, seed):
    c = dict(case)
    pkg = _mod()
    s = {"c": c}
    op = c["op"]
    if op == "batch":
        B = _mod("batch")
        S = _mod("shapes")
        g = np.random.default_rng(seed)
        maps, fields = [], []
        for (rows, cols, pges), axes in _batch_shapes(c):
            v = [np.linspace(-1.2, 1.2, n) for n in (cols, rows, pges)]
            axes = tuple(float(a * g.uniform(0.97, 1.0)) for a in axes)
            x, y, z, F = S.ellipsoid_field(*v, axes, device="cuda")
            h = tuple(float(a[1] - a[0]) for a in v)
            m = pkg.SDF3(pkg.GD3(x, y, z, spacing=h), Val=_colmajor(F, torch.float32), precision="f32")
            m.setDistance()
            maps.append(m)
            fields.append(m.F.clone())
        s |= {"batch": B.VesicleBatch(maps), "fields": fields}
        return s
    if op == "transport":
        A = _mod("adjoint")
        x, y, z, h, phi0, v, dt, target = _transport_data(c, seed)
        plan = A.TransportPlan(steps=c["steps"], reinit_every=c["every"], reinit_iters=c["iters"], checkpoint_every=10)
        grid = pkg.GD3(x, y, z, spacing=h)
        s |= {"tr": A.Transport(grid, dt, plan, precision=c["prec"]), "target": target, "cell": h[0] * h[1] * h[2],
              "eps": 1.5 * grid.Ds, "leaves": [t.requires_grad_(True) for t in (phi0, *v)]}
        return s
    x, y, z, h, F = _initial(c, seed)
    m = pkg.SDF3(pkg.GD3(x, y, z, spacing=h), Val=F.clone(), precision=c["prec"])
    s |= {"m": m, "F0": F}
    d = DT[c["prec"]]
    if op in ("step", "relax", "reinit", "extend"):
        m.setDistance()
    if op == "aux":
        m.A = _colmajor(_domain(x, y, z, seed), d)
    elif op == "redistance":
        s["A"] = _colmajor(_surface_field(x, y, z, seed), d)
    elif op == "extend":
        s["C"] = _colmajor(_curvature_like(x, y, z, seed), d)
    elif op == "advect":
        s["v"] = [_colmajor(t, d) for t in _velocity_of(x, y, z, seed)]
        s["dt"] = torch.tensor([0.5 * min(h)], dtype=torch.float64, device="cuda")
    elif op == "relax":
        s["A0"], s["V0"] = (float(t) for t in m.area_volume().cpu())  # what the relaxation holds
    return s


_FEW = 6  # members of a batch that come back one by one (and that `exact` follows)

# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------

_DIST = ("xpr", "xpl", "ypf", "ypb", "zpu", "zpd")


def run(s):
    c, op = s["c"], s["c"]["op"]
    if op == "batch":
        b = s["batch"]
        for m, F in zip(b.maps, s["fields"]):
            m.F.copy_(F)
            m.setDistance()
        infos = b.step_batched(c["ext"], c["iters"], 0.5)
        flat = [m.F.permute(2, 1, 0).reshape(-1) for m in b.maps]
        return {"F": flat[:_FEW], "others": torch.cat(flat[_FEW:]) if len(flat) > _FEW else None,
                "info": torch.stack(infos)}
    if op == "transport":
        A = _mod("adjoint")
        phi = s["tr"](*s["leaves"])
        loss = A.heaviside_mismatch(phi, s["target"], s["eps"], s["cell"])
        return {"phi": phi, "loss": loss, "grads": list(torch.autograd.grad(loss, s["leaves"]))}
    m = s["m"]
    if op == "area_volume":
        return m.area_volume()
    if op == "toolbox":
        m.GPUsetCalculusToolBox()
        return {n: getattr(m, n) for n in _mod("sdf3").TOOLBOX_FIELDS}
    if op == "aux":
        m.GPUAsetCalculusToolBox()
        return {n: getattr(m, n) for n in _mod("sdf3").AUX_FIELDS}
    if op == "reinit":
        f = {"weno5": m.WENO5RK3Reinitialization, "eno3": m.WENORK3Reinitialization,
             "enork2": m.ENORK2Reinitialization}[c["scheme"]]
        return f(s["F0"], c["iters"])
    if op == "extend":
        f = {"weno5": m.WENO5RK3Extend, "eno3": m.WENORK3Extend, "enork2": m.ENORK2Extend}[c["scheme"]]
        return f(s["C"], c["ext"])
    if op == "advect":
        return m.WENO5RK3Advection(s["F0"], *s["v"], s["dt"], c["steps"])
    if op == "redistance":
        f = {"weno5": m.WENO5RK3ClosetPointSurfaceRedistance, "eno3": m.WENORK3ClosetPointSurfaceRedistance,
             "enork2": m.ENORK2ClosetPointSurfaceRedistance}[c["scheme"]]
        return f(s["A"], c["iters"], c["ext"])
    # a step of a driver that is handed a field: the field in, its distances, the step
    m.F.copy_(s["F0"])
    m.setDistance()
    if op == "step":
        info = m.vesicle_step(c["ext"], c["iters"], 0.5, graph=c["graph"])
    else:
        info = m.relax_step(s["A0"], s["V0"], kappa=1.0, spon_c=0.0, cfl=0.5, alpha=0.5, ext_iters=c["ext"],
                            reinit_iters=c["iters"], graph=c["graph"])
    return {"F": m.F, "info": info, "dist": [getattr(m, n) for n in _DIST]}


# ---------------------------------------------------------------------------------------
# the work that cannot be done without
# ---------------------------------------------------------------------------------------

# operations per node and stage: one upwind WENO5 reconstruction per axis is about 55
# (5 differences, 3 candidates, 3 smoothness indicators and weights, the quotient), a
# quadratic-ENO one about 12; the combination and the transport or norm about 12
_WENO, _ENO2 = 3 * 55 + 12, 3 * 12 + 12


def work(case):
    c, n, w = case, _nodes(case), 4 if case["prec"] == "f32" else 8
    op, per = c["op"], _WENO
    words = {"area_volume": 1, "toolbox": 19, "aux": 31, "reinit": 8 if c.get("scheme") == "weno5" else 2,
             "extend": 9 if c.get("scheme") == "weno5" else 3, "advect": 5, "redistance": 3, "step": 8, "batch": 8,
             "relax": 8, "transport": 10}[op]
    stages = _stages(c)
    if c.get("scheme") == "enork2":
        per = _ENO2
    if op in ("area_volume", "toolbox", "aux"):
        flops = n * {"area_volume": 60, "toolbox": 150, "aux": 350}[op]
    elif op == "relax":
        flops = n * (4 * c["ext"] * _ENO2 + 3 * (c["ext"] + c["iters"]) * _WENO)
    elif op == "transport":
        flops = n * 3 * 4 * _WENO * (c["steps"] + c["steps"] // max(1, c["every"]) * c["iters"])
    else:
        flops = n * stages * per
    return {"bytes": n * w * words, "flops": flops}


# ---------------------------------------------------------------------------------------
# the same results in 64 bits, by plain torch
# ---------------------------------------------------------------------------------------


def _weno5(a, b, c, d, e):
    q1 = a / 3 - b * (7 / 6) + c * (11 / 6)
    q2 = -b / 6 + c * (5 / 6) + d / 3
    q3 = c / 3 + d * (5 / 6) - e / 6
    w1 = 0.1 / (13 / 12 * (a - 2 * b + c)**2 + 0.25 * (a - 4 * b + 3 * c)**2 + 1e-6)**2
    w2 = 0.6 / (13 / 12 * (b - 2 * c + d)**2 + 0.25 * (b - d)**2 + 1e-6)**2
    w3 = 0.3 / (13 / 12 * (c - 2 * d + e)**2 + 0.25 * (3 * c - 4 * d + e)**2 + 1e-6)**2
    return (w1 * q1 + w2 * q2 + w3 * q3) / (w1 + w2 + w3)


def _minmod(a, b):
    return torch.where(a * b < 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _minabs(a, b):
    return torch.where(a.abs() < b.abs(), a, b)


def _nu_smooth(e, u):
    """Smoothness of the three stencils of faces e[0..5], cells u[0..4], in the middle cell."""
    a, b, c, d, f, g = e
    w = d - c
    s0 = 4 * (w / (g - c))**2 * (((u[4] - u[3]) / (g - d))**2 * (10 * w * w + (f - c) * (f - d))
                                 + (u[4] - u[3]) * (u[2] - u[3]) / ((g - d) * (f - c))
                                 * (20 * w * w + 2 * (f - c) * (f - d) + (g - c) * (2 * f - d - c))
                                 + ((u[2] - u[3]) / (f - c))**2 * (10 * w * w + (g + f - 2 * c) * (g + f - d - c)))
    s1 = 4 * (w / (f - b))**2 * (((u[1] - u[2]) / (d - b))**2 * (10 * w * w + (f - c) * (f - d))
                                 + (u[3] - u[2]) * (u[1] - u[2]) / ((f - c) * (d - b))
                                 * (20 * w * w - (f - d) * (c - b) - (f - c) * (d - b))
                                 + ((u[3] - u[2]) / (f - c))**2 * (10 * w * w + (c - b) * (d - b)))
    s2 = 4 * (w / (d - a))**2 * (((u[0] - u[1]) / (c - a))**2 * (10 * w * w + (d - b) * (c - b))
                                 + (u[2] - u[1]) * (u[0] - u[1]) / ((d - b) * (c - a))
                                 * (20 * w * w + 2 * (d - b) * (c - b) + (d - a) * (d + c - 2 * b))
                                 + ((u[2] - u[1]) / (d - b))**2 * (10 * w * w + (2 * d - a - b) * (d + c - b - a)))
    return s0, s1, s2


def _nu_right(e, u):
    """Nonuniform WENO value at face e[3] (the right face of the middle cell)."""
    a, b, c, d, f, g = e
    v0 = u[3] + (u[2] - u[3]) * (f - d) / (g - c) * (g - d) / (f - c) \
        - (u[4] - u[3]) * (f - d) / (g - c) * (d - c) / (g - d)
    v1 = u[2] + (u[3] - u[2]) * (d - c) / (f - b) * (d - b) / (f - c) \
        - (u[1] - u[2]) * (d - c) / (f - b) * (f - d) / (d - b)
    v2 = u[1] + (u[0] - u[1]) * (d - c) / (c - a) * (d - b) / (d - a) \
        + (u[2] - u[1]) * (1 + (d - c) / (d - b) + (d - c) / (d - a))
    k0 = (d - a) / (g - a) * (d - b) / (g - b)
    k1 = (d - a) / (g - a) * (g - d) / (g - b) * (1 + (g - b) / (f - a))
    k2 = (f - d) / (g - a) * (g - d) / (f - a)
    s = _nu_smooth(e, u)
    w = [k / (t + 1e-6)**2 for k, t in zip((k0, k1, k2), s)]
    return (v0 * w[0] + v1 * w[1] + v2 * w[2]) / (w[0] + w[1] + w[2])


def _weno_pair(xs, hs):
    """(forward, backward) nonuniform WENO derivatives at xs[3]."""
    u = [(hs[m + 1] - hs[m]) / (xs[m + 1] - xs[m]) for m in range(6)]
    back = _nu_right(xs[:6], u[:5])
    # the forward value is the backward one of the mirrored line
    fore = _nu_right([-x for x in xs[:0:-1]], u[:0:-1])
    return fore, back


def _eno3_pair(x, h):
    f = [(h[m + 1] - h[m]) / (x[m + 1] - x[m]) for m in range(6)]
    g = [(f[m + 1] - f[m]) / (x[m + 2] - x[m]) for m in range(5)]
    t = [(g[m + 1] - g[m]) / (x[m + 3] - x[m]) for m in range(4)]
    m2, m1, z, p1, p2 = x[1], x[2], x[3], x[4], x[5]
    back = f[2] + _minmod(g[1], g[2]) * (z - m1) + torch.where(
        g[1].abs() < g[2].abs(), (z - m1) * (z - m2) * _minabs(t[1], t[0]), (z - m1) * (z - p1) * _minabs(t[1], t[2]))
    fore = f[3] + _minmod(g[2], g[3]) * (z - p1) + torch.where(
        g[2].abs() < g[3].abs(), (z - m1) * (z - p1) * _minabs(t[1], t[2]), (z - p1) * (z - p2) * _minabs(t[2], t[3]))
    return fore, back


def _lagrange(y, t):
    """Value at t of the polynomial through (m, y[m])."""
    out = torch.zeros_like(t)
    for m in range(len(y)):
        w = torch.ones_like(t)
        for q in range(len(y)):
            if q != m:
                w = w * (t - q) / (m - q)
        out = out + y[m] * w
    return out


def _lagrange_slope(y, t):
    out = torch.zeros_like(t)
    for m in range(len(y)):
        for r in range(len(y)):
            if r == m:
                continue
            w = torch.full_like(t, 1.0 / (m - r))
            for q in range(len(y)):
                if q not in (m, r):
                    w = w * (t - q) / (m - q)
            out = out + y[m] * w
    return out


class Exact:
    """The level-set operations on one grid in FP64.  Axis a: 0 x (columns), 1 y (rows), 2 z."""

    DIM = (1, 0, 2)

    def __init__(self, size, h, scheme="weno5"):
        self.size, self.h, self.ds, self.scheme = tuple(size), tuple(h), sum(h) / 3, scheme
        self.at = []
        for a in range(3):
            n = self.size[self.DIM[a]]
            self.at.append(torch.clamp(torch.arange(-3, n + 3, device="cuda"), 0, n - 1))

    def line(self, f, a):
        p = f.index_select(self.DIM[a], self.at[a])
        return [p.narrow(self.DIM[a], s, self.size[self.DIM[a]]) for s in range(7)]

    # -- distances: six fields, the spacing where the edge is not crossed
    def distances(self, f):
        out = []
        for a in range(3):
            p, h, dim = self.line(f, a), self.h[a], self.DIM[a]
            at = torch.nonzero((p[3] * p[4] < 0).reshape(-1)).squeeze(1)
            v = [t.reshape(-1)[at] for t in p]
            d2 = _minmod(v[4] - 2 * v[3] + v[2], v[5] - 2 * v[4] + v[3])
            curved = d2.abs() > 10e-10
            safe = torch.where(curved, d2, torch.ones_like(d2))
            disc = torch.where(curved, (0.5 * d2 - v[3] - v[4])**2 - 4 * v[3] * v[4], torch.ones_like(d2))
            eno = h * torch.where(curved, 0.5 + (v[3] - v[4] - torch.sign(v[3] - v[4]) * torch.sqrt(disc)) / safe,
                                  v[3] / (v[3] - v[4]))
            if self.scheme == "enork2":
                d = eno
            else:
                # degree 5 on the nodes -2..3 (weno5), cubic on -1..2 (eno3); the root lies in the cell
                y, lo0 = (v[1:7], 2.0) if self.scheme == "weno5" else (v[2:6], 1.0)
                with torch.no_grad():
                    lo, hi = torch.full_like(v[3], lo0), torch.full_like(v[3], lo0 + 1)
                    for _ in range(54):
                        mid = 0.5 * (lo + hi)
                        left = _lagrange(y, mid) * v[3] > 0
                        lo, hi = torch.where(left, mid, lo), torch.where(left, hi, mid)
                    t = 0.5 * (lo + hi)
                    slope = _lagrange_slope(y, t)
                t = torch.clamp(t - _lagrange(y, t) / slope, lo0, lo0 + 1)  # also the root's derivative
                kink = (v[2] * v[3] < 0) | (v[4] * v[5] < 0)
                d = torch.where(kink, eno, (t - lo0) * h)
            base = torch.full(self.size, h, dtype=torch.float64, device="cuda").reshape(-1)
            fore = base.index_put((at,), d)
            step = math.prod(self.size[dim + 1:])
            out += [fore.reshape(self.size), base.index_put((at + step,), h - d).reshape(self.size)]
        return out

    def pseudo_dt(self, d):
        m = d[0]
        for t in d[1:]:
            m = torch.minimum(m, t)
        return 0.3 * m

    # -- one-sided derivatives with the interface inserted where `cut`
    def pair(self, f, a, d, cut, values=None):
        p, h = self.line(f, a), self.h[a]
        r1, l1 = d[2 * a], d[2 * a + 1]
        if self.scheme == "enork2":
            vr, vl = (values[2 * a], values[2 * a + 1]) if values else (torch.zeros_like(f), torch.zeros_like(f))
            c2 = p[2] - 2 * p[3] + p[4]
            mr = 0.5 * _minmod(c2, p[3] - 2 * p[4] + p[5]) / h**2
            ml = 0.5 * _minmod(c2, p[3] - 2 * p[2] + p[1]) / h**2
            fore = (torch.where(r1 == h, p[4], vr) - p[3]) / r1 - r1 * mr
            back = (p[3] - torch.where(l1 == h, p[2], vl)) / l1 + l1 * ml
            return fore, back, p
        v = [(p[m + 1] - p[m]) / h for m in range(6)]
        back, fore = _weno5(*v[:5]), _weno5(*v[:0:-1])
        if cut is None:
            return fore, back, p
        where = cut(p, r1, l1, h)
        at = torch.nonzero(where.reshape(-1)).squeeze(1)
        q = [t.reshape(-1)[at] for t in p]
        r, l = r1.reshape(-1)[at], l1.reshape(-1)[at]
        vr, vl = [t.reshape(-1)[at] for t in values[2 * a:2 * a + 2]] if values else (torch.zeros_like(r),) * 2
        R, L = r < h, l < h
        full = torch.full_like(r, h)
        xs = [torch.where(L, -2 * full, -3 * full), torch.where(L, -full, -2 * full), torch.where(L, -l, -full),
              torch.zeros_like(r), torch.where(R, r, full), torch.where(R, full, 2 * full),
              torch.where(R, 2 * full, 3 * full)]
        hs = [torch.where(L, q[1], q[0]), torch.where(L, q[2], q[1]), torch.where(L, vl, q[2]), q[3],
              torch.where(R, vr, q[4]), torch.where(R, q[4], q[5]), torch.where(R, q[5], q[6])]
        df, db = (_weno_pair if self.scheme == "weno5" else _eno3_pair)(xs, hs)
        fore = fore.contiguous().reshape(-1).index_put((at,), df).reshape(self.size)
        back = back.contiguous().reshape(-1).index_put((at,), db).reshape(self.size)
        return fore, back, p

    # -- reinitialization
    def reinit_step(self, f, d, neg):
        s = torch.zeros_like(f)
        sign_change = (lambda p, r, l, h: (p[2] * p[3] < 0) | (p[3] * p[4] < 0))
        for a in range(3):
            fore, back, _ = self.pair(f, a, d, sign_change)
            fore, back = torch.where(neg, -fore, fore), torch.where(neg, -back, back)
            s = s + torch.maximum(torch.clamp(back, min=0)**2, torch.clamp(fore, max=0)**2)
        norm = torch.where(s > 0, torch.sqrt(torch.where(s > 0, s, torch.ones_like(s))), torch.zeros_like(s))
        step = (norm - 1) * self.pseudo_dt(d) * torch.where(neg, -1.0, 1.0)
        if self.scheme != "enork2":
            fixed = d[0] < 1e-6 * self.h[0]
            for t in d[1:]:
                fixed = fixed | (t < 1e-6 * self.h[0])
            step = torch.where(fixed, torch.zeros_like(step), step)
        return step

    def march(self, f, step):
        """One RK step of f <- f - step(f)."""
        g = f - step(f)
        if self.scheme == "enork2":
            return (f + g - step(g)) / 2
        g = 0.75 * f + 0.25 * (g - step(g))
        return f / 3 + 2 / 3 * (g - step(g))

    def reinit(self, f, iters, d=None):
        d = self.distances(f) if d is None else d
        neg = f < 0
        for _ in range(iters):
            f = self.march(f, lambda t: self.reinit_step(t, d, neg))
        return f

    # -- extension
    def normals(self, F, d, floor=1e-6):
        n = []
        for a in range(3):
            r1, l1, h = d[2 * a], d[2 * a + 1], self.h[a]
            fore, back, p = self.pair(F, a, d, lambda p, r, l, h: (r < h) | (l < h))
            if self.scheme == "enork2":
                right, left = torch.where(r1 == h, p[4], 0.0), torch.where(l1 == h, p[2], 0.0)
            else:
                right, left = p[4], p[2]
            n.append(torch.where(right.abs() < left.abs(), fore, back))
        m = torch.clamp(torch.sqrt(n[0]**2 + n[1]**2 + n[2]**2), min=floor)
        return [torch.sign(F) * (t / m) for t in n]

    def crossings(self, C, d):
        out = []
        for a in range(3):
            p, h = self.line(C, a), self.h[a]
            r1, l1 = d[2 * a], d[2 * a + 1]
            if self.scheme == "weno5":
                cf, cb = _lagrange(p[1:7], 2 + r1 / h), _lagrange(p[0:6], 3 - l1 / h)
            elif self.scheme == "eno3":
                cf, cb = _lagrange(p[2:6], 1 + r1 / h), _lagrange(p[1:5], 2 - l1 / h)
            else:
                c2 = p[4] - 2 * p[3] + p[2]
                qf = 0.5 * _minmod(c2, p[5] - 2 * p[4] + p[3]) / h**2
                qb = 0.5 * _minmod(c2, p[3] - 2 * p[2] + p[1]) / h**2
                xf, xb = r1 - h / 2, h / 2 - l1
                cf = qf * xf**2 + (p[4] - p[3]) / h * xf + (p[4] + p[3]) / 2 - qf * h**2 / 4
                cb = qb * xb**2 + (p[3] - p[2]) / h * xb + (p[2] + p[3]) / 2 - qb * h**2 / 4
            out += [cf, cb]
        return out

    def extend_step(self, C, d, v, values, dt, fixed):
        s = torch.zeros_like(C)
        for a in range(3):
            fore, back, _ = self.pair(C, a, d, lambda p, r, l, h: (r < h) | (l < h), values)
            s = s + torch.clamp(v[a], max=0) * fore + torch.clamp(v[a], min=0) * back
        return torch.where(fixed, torch.zeros_like(s), s * dt)

    def extend(self, C, iters, F, d=None, floor=1e-6, v=None):
        d = self.distances(F) if d is None else d
        v = self.normals(F, d, floor) if v is None else v
        values, dt = self.crossings(C, d), self.pseudo_dt(d)
        fixed = torch.zeros_like(F, dtype=torch.bool)
        if self.scheme != "enork2":
            for t in d:
                fixed = fixed | (t < 1e-6 * self.h[0])
        for _ in range(iters):
            C = self.march(C, lambda t: self.extend_step(t, d, v, values, dt, fixed))
        return C

    def redistance(self, A, iters, ext, F):
        dA, dF, neg = self.distances(A), self.distances(F), A < 0
        v = self.normals(F, dF, 1e-14)

        def extended(t):
            return self.extend(t, ext, F, dF, v=v)

        for _ in range(iters):
            A = extended(A)
            t = extended(A - self.reinit_step(A, dA, neg))
            if self.scheme == "enork2":
                A = (A + (t - self.reinit_step(t, dA, neg))) / 2
                continue
            t = extended(0.75 * A + 0.25 * (t - self.reinit_step(t, dA, neg)))
            A = A / 3 + 2 / 3 * (t - self.reinit_step(t, dA, neg))
        return extended(A)

    # -- advection
    def advect_step(self, F, v, dt):
        s = torch.zeros_like(F)
        for a in range(3):
            fore, back, _ = self.pair(F, a, [None] * 6, None)
            s = s + torch.clamp(v[a], max=0) * fore + torch.clamp(v[a], min=0) * back
        return dt * s

    def advect(self, F, v, dt, steps=1):
        for _ in range(steps):
            F = self.march(F, lambda t: self.advect_step(t, v, dt))
        return F

    # -- the calculus toolbox (neighbours clamped at the edge)
    def near(self, f):
        """f at a node's neighbours: near(i, j, k), offsets in x, y, z."""
        g = f
        for a in range(3):
            g = g.index_select(self.DIM[a], self.at[a][2:-2])
        r, c, p = self.size
        return lambda x, y, z: g[1 + y:1 + y + r, 1 + x:1 + x + c, 1 + z:1 + z + p]

    def first_second(self, f):
        n = self.near(f)
        e = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
        d = [(n(*e[a]) - n(*(-t for t in e[a]))) / (2 * self.h[a]) for a in range(3)]
        dd = [(n(*e[a]) - 2 * f + n(*(-t for t in e[a]))) / self.h[a]**2 for a in range(3)]
        q = 4 * self.ds**2
        xy = (n(1, 1, 0) + n(-1, -1, 0) - n(-1, 1, 0) - n(1, -1, 0)) / q
        yz = (n(0, 1, 1) + n(0, -1, -1) - n(0, 1, -1) - n(0, -1, 1)) / q
        zx = (n(1, 0, 1) + n(-1, 0, -1) - n(-1, 0, 1) - n(1, 0, -1)) / q
        return d, dd, (xy, yz, zx)

    def primal(self, f, d, lap, mag):
        """Heaviside and Dirac functions of f from its primal max(f, 0)."""
        p, pp, _ = self.first_second(torch.clamp(f, min=0))
        dot = p[0] * d[0] + p[1] * d[1] + p[2] * d[2]
        return dot / mag**2, (pp[0] + pp[1] + pp[2]) / mag**2 - dot * lap / mag**4

    def toolbox(self, F):
        (x, y, z), (xx, yy, zz), (xy, yz, zx) = self.first_second(F)
        m = torch.clamp(torch.sqrt(x * x + y * y + z * z), min=1e-14)
        lap = xx + yy + zz
        quad = x * (xx * x + xy * y + zx * z) + y * (xy * x + yy * y + yz * z) + z * (zx * x + yz * y + zz * z)
        q1 = (yy * zz - yz * yz) * x + (zx * yz - xy * zz) * y + (xy * yz - zx * yy) * z
        q2 = (yz * zx - xy * zz) * x + (xx * zz - zx * zx) * y + (zx * xy - xx * yz) * z
        q3 = (xy * yz - yy * zx) * x + (zx * xy - xx * yz) * y + (xx * yy - xy * xy) * z
        H, D = self.primal(F, (x, y, z), lap, m)
        return dict(Fx=x, Fy=y, Fz=z, FGradMag=m, Nx=x / m, Ny=y / m, Nz=z / m, Fxx=xx, Fyy=yy, Fzz=zz, Fxy=xy, Fyz=yz,
                    Fzx=zx, FLaplacian=lap, MeanCurvature=-lap / m + quad / m**3,
                    GaussianCurvature=(x * q1 + y * q2 + z * q3) / m**4, Heaviside=H, DiracDelta=D)

    def area_volume(self, F, t=None):
        t = self.toolbox(F) if t is None else t
        return self.ds**3 * torch.stack([torch.where(F.abs() < 2 * self.ds, t["DiracDelta"], 0.0).sum(),
                                         torch.where(F < 2 * self.ds, 1 - t["Heaviside"], 0.0).sum()])

    # -- SD.GD3's periodic operators
    def roll(self, f, a, s):
        return torch.roll(f, -s, self.DIM[a])

    def gradient(self, f):
        return [(self.roll(f, a, 1) - self.roll(f, a, -1)) / (2 * self.h[a]) for a in range(3)]

    def laplacian(self, f):
        return sum((self.roll(f, a, 1) - 2 * f + self.roll(f, a, -1)) / self.h[a]**2 for a in range(3))

    def smooth(self, f, dt, alpha):
        lam = 0.0
        for a in range(3):
            n, shape = self.size[self.DIM[a]], [1, 1, 1]
            shape[self.DIM[a]] = n
            k = torch.arange(n, dtype=torch.float64, device="cuda")
            lam = lam + ((2 * torch.cos(2 * math.pi * k / n) - 2) / self.h[a]**2).reshape(shape)
        return torch.fft.ifftn(torch.fft.fftn(f) / (1 + alpha * dt * lam**2)).real

    # -- whole steps
    def step(self, F, ext, iters, cfl):
        t = self.toolbox(F)
        av = self.area_volume(F, t)
        vn = self.extend(t["MeanCurvature"], ext, F)
        top = vn[F.abs() < 2 * self.ds].abs().max()
        dt = cfl * self.ds / top
        F = self.advect(F, [vn * t[n] for n in ("Nx", "Ny", "Nz")], dt)
        d = self.distances(F)
        return self.reinit(F, iters, d), torch.stack([av[0], av[1], dt, top]), d

    def relax(self, F, A0, V0, cfl, alpha, ext, iters):
        eno3, enork2 = Exact(self.size, self.h, "eno3"), Exact(self.size, self.h, "enork2")
        t = self.toolbox(F)
        area, volume = self.area_volume(F, t)
        H, K, G = eno3.extend(t["MeanCurvature"], ext, F), t["GaussianCurvature"], t["FGradMag"]
        nsb = enork2.extend(self.laplacian(H) + 0.5 * H * (H * H - 4 * K), ext, F)
        band = F.abs() < 2 * self.ds
        top = nsb[band].abs().max()
        dt = cfl * self.ds / top

        def integral(f, mask):
            return self.ds**3 * torch.where(mask, f * t["DiracDelta"] * G, 0.0).sum()

        c11, c12, hn, n1 = (integral(f, band) for f in (H * H, H, H * nsb, nsb))
        s1, s2 = hn - (A0 - area) / dt, n1 + (V0 - volume) / dt
        det = c11 * A0 - c12 * c12
        ten, pre = (s1 * A0 - c12 * s2) / det, (c11 * s2 - c12 * s1) / det
        v = enork2.extend(self.smooth((ten * H - nsb + pre) * G, dt, alpha), ext, F)
        F = F - dt * v
        d = self.distances(F)
        energy = integral(H * H, F.abs() < 2 * self.ds)
        info = torch.stack([area, volume, dt, top, c11, c12, hn, n1, ten, pre, energy])
        return self.reinit(F, iters, d), info, d

    # -- the auxiliary toolbox of the domain level set A on F = 0
    def auxiliary(self, A, F):
        t = self.toolbox(F)
        f, N, mF = (t["Fx"], t["Fy"], t["Fz"]), (t["Nx"], t["Ny"], t["Nz"]), t["FGradMag"]
        HF = ((t["Fxx"], t["Fxy"], t["Fzx"]), (t["Fxy"], t["Fyy"], t["Fyz"]), (t["Fzx"], t["Fyz"], t["Fzz"]))
        a, aa, (axy, ayz, azx) = self.first_second(A)
        HA = ((aa[0], axy, azx), (axy, aa[1], ayz), (azx, ayz, aa[2]))

        def dot(u, v):
            return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]

        def cross(u, v):
            return (u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0])

        def times(M, v):
            return tuple(dot(r, v) for r in M)

        def norm(v):
            return torch.clamp(torch.sqrt(dot(v, v)), min=1e-14)

        mA = norm(a)
        C = cross(f, a)
        mC = norm(C)
        tan = tuple(u / mC for u in C)
        con = cross(tan, N)
        w = [p + q for p, q in zip(cross(times(HF, tan), a), cross(f, times(HA, tan)))]
        Hf = times(HF, f)
        gradN = tuple(tuple(HF[i][j] / mF - f[i] * Hf[j] / mF**3 for j in range(3)) for i in range(3))
        lap = aa[0] + aa[1] + aa[2]
        H, D = self.primal(A, a, lap, mA)
        ch = cross(self.gradient(t["Heaviside"]), self.gradient(H))
        return dict(Ax=a[0], Ay=a[1], Az=a[2], AGradMag=mA, Cx=C[0], Cy=C[1], Cz=C[2], NormCrossAF=mC, tx=tan[0],
                    ty=tan[1], tz=tan[2], nx=con[0], ny=con[1], nz=con[2], Axx=aa[0], Ayy=aa[1], Azz=aa[2], Axy=axy,
                    Ayz=ayz, Azx=azx, ALaplacian=lap, GeodesicCurvature=dot(con, w) / mC,
                    NormalCurvature=-dot(tan, times(gradN, tan)), GeodesicTorsion=-dot(tan, times(gradN, con)),
                    BPerpendicular=-dot(con, times(gradN, con)), AHeaviside=H, ADiracDelta=D,
                    AFDiracDelta=dot(C, ch) / mC**2,
                    ADiracDeltaDn=(self.laplacian(H) - D * self.laplacian(A)) / mA)


def _exact_transport(c, seed):
    x, y, z, h, phi0, v, dt, target = _transport_data(c, seed)
    E = Exact(phi0.shape, h)
    leaves = [t.detach().double().contiguous().requires_grad_(True) for t in (phi0, *v)]
    phi, v = leaves[0], leaves[1:]

    def advect(f, *v):
        return E.march(f, lambda t: E.advect_step(t, v, dt))

    def pseudo(f, neg, *d):
        return E.march(f, lambda t: E.reinit_step(t, d, neg))

    for s in range(c["steps"]):
        phi = checkpoint(advect, phi, *v, use_reentrant=False)
        if (s + 1) % c["every"] == 0:
            d, neg = E.distances(phi), phi.detach() < 0
            for _ in range(c["iters"]):
                phi = checkpoint(pseudo, phi, neg, *d, use_reentrant=False)
    eps = 1.5 * E.ds

    def heaviside(f):
        t = torch.clamp(f / eps, -1.0, 1.0)
        return 0.5 * (1 + t + torch.sin(math.pi * t) / math.pi)

    loss = ((heaviside(phi) - heaviside(target))**2).sum() * (h[0] * h[1] * h[2])
    if c["steps"] >= c["every"]:
        # through a reinitialization the derivative of a stencil next to a short cell gap follows
        # the last digits of the state it is taken at, so the FP64 state's gradient is another one
        return {"phi": phi.detach(), "loss": loss.detach(), "grads": None}
    grads = torch.autograd.grad(loss, leaves)
    return {"phi": phi.detach(), "loss": loss.detach(), "grads": list(grads)}


def exact(case, seed):
    c, op = dict(case), case["op"]
    if op == "transport":
        # the FP64 tape of one stage at a time has to fit, and the sweep to end in seconds
        return _exact_transport(c, seed) if _nodes(c) * _stages(c) <= 1.3e9 * 4 else None
    with torch.no_grad():
        if op == "batch":
            g = np.random.default_rng(seed)
            fields = []
            for n, ((rows, cols, pges), axes) in enumerate(_batch_shapes(c)):
                v = [np.linspace(-1.2, 1.2, k) for k in (cols, rows, pges)]
                axes = tuple(float(a * g.uniform(0.97, 1.0)) for a in axes)
                if n >= _FEW:  # all of them would take minutes
                    break
                x, y, z = _mod("shapes").meshgrid(*v, device="cuda")
                F = torch.sqrt(x**2 / axes[0]**2 + y**2 / axes[1]**2 + z**2 / axes[2]**2) - 1
                h = tuple(float(a[1] - a[0]) for a in v)
                F = Exact(F.shape, h).step(F.float().double(), c["ext"], c["iters"], 0.5)[0]
                fields.append(F.permute(2, 1, 0).reshape(-1))
            return {"F": fields, "others": None, "info": None}
        x, y, z, h, F = _initial(c, seed)
        F = F.double().contiguous()
        prec = DT[c["prec"]]
        E = Exact(F.shape, h, c.get("scheme", "weno5"))

        def given(t):
            return t.to(prec).double().contiguous()

        if op == "area_volume":
            return E.area_volume(F)
        if op == "toolbox":
            return E.toolbox(F)
        if op == "aux":
            return E.auxiliary(given(_domain(x, y, z, seed)), F)
        if op == "reinit":
            return E.reinit(F, c["iters"])
        if op == "extend":
            return E.extend(given(_curvature_like(x, y, z, seed)), c["ext"], F)
        if op == "advect":
            return E.advect(F, [given(t) for t in _velocity_of(x, y, z, seed)], 0.5 * min(h), c["steps"])
        if op == "redistance":
            return E.redistance(given(_surface_field(x, y, z, seed)), c["iters"], c["ext"], F)
        if op == "step":
            F, info, d = E.step(F, c["ext"], c["iters"], 0.5)
        else:
            F, info, d = E.relax(F, *E.area_volume(F), 0.5, 0.5, c["ext"], c["iters"])
        return {"F": F, "info": info, "dist": d}
