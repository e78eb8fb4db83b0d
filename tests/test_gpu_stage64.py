"""The plain FP64 stage kernels at the sizes and values where their short arithmetic and
their split into tiles and band blocks can go wrong: grids around the 32 x 4 tile, a single
page, and fields with infinities, NaN and values outside the range of the short quotients.
Bit for bit the loops composed of the drop-in kernels (the general per-node code), NaN where
those have NaN.  GPU only."""
import importlib

import numpy as np
import pytest
import torch

from gpu_util import dev, empty, host, ptr, stream

pytestmark = pytest.mark.gpu

S = importlib.import_module("2018_7_vesicle_gb300.shapes")
SIZES = [(31, 3, 1), (33, 5, 2), (32, 4, 9), (1, 7, 11), (7, 41, 6)]


def level_set(size, spacing, radius, seed):
    r, c, p = size
    v = [np.linspace(-(n - 1) / 2, (n - 1) / 2, n) * h for n, h in zip((c, r, p), spacing)]
    x, y, z = S.meshgrid(*v)
    F = np.sqrt((x - 0.013)**2 + (y + 0.021)**2 + (z - 0.007)**2) - radius
    return x, y, z, np.asfortranarray(F * (1 + 0.1 * np.sin(3 * x + 2 * y + seed)))


def plant(F, kind):
    """Values that the short sequences do not take, away from and next to the interface."""
    F = F.copy(order="F")
    flat = F.reshape(-1, order="F")  # a view: F is in Fortran order
    at = np.arange(3, F.size, max(7, F.size // 6))
    if kind == "nonfinite":
        flat[at[0::2]], flat[at[1::2]] = np.inf, np.nan
    elif kind == "huge":
        flat[at] = 1e200
    elif kind == "tiny":
        flat[at] = 1e-250
        flat[:F.size // 3] *= 1e-305
    elif kind == "zero":
        flat[at] = 0.0
        flat[at // 2] = -0.0
    return F


def where_min(ts):
    """The smaller of two as the kernels take it, (x < y) ? x : y, in their tree order."""
    def m(x, y):
        return torch.where(x < y, x, y)

    return m(m(ts[0], ts[1]), m(m(ts[2], ts[3]), m(ts[4], ts[5])))


class Loops:
    """The method loops of one object composed of the drop-in kernels (the general per-node
    code, one launch per kernel) and elementwise torch operations."""

    def __init__(self, vsl, m, F, scheme):
        self.vsl, self.m, self.scheme, self.g = vsl, m, scheme, m.GD3
        self.tail = (*m.GD3.args(), m.GD3.NumElt, stream())
        F = dev(F)
        if scheme == "weno5":
            self.d = list(m._dist())
        else:
            self.d = [empty(m.GD3.Size, fill=s) for s in (m.GD3.Dx,) * 2 + (m.GD3.Dy,) * 2 + (m.GD3.Dz,) * 2]
            fn = "vsl_cubic_boundary_correction" if scheme == "eno3" else "vsl_enork2_boundary_correction"
            vsl.call(fn, *map(ptr, self.d), ptr(F), m.GD3.NumElt, *m.GD3.args(), stream())
        self.dt = 0.3 * where_min(self.d)
        self.F, self.mask = F, (F < 0)

    def march(self, f, step):
        a = f - step(f)
        if self.scheme == "enork2":
            return (f + a - step(a)) / 2
        b = 0.75 * f + 0.25 * (a - step(a))
        return (1. / 3.) * f + (2. / 3.) * (b - step(b))

    def call(self, base, *fields):
        fn = {"weno5": "vsl_" + base, "eno3": f"vsl_{base}_eno3", "enork2": f"vsl_enork2_{base}"}[self.scheme]
        if base == "boundary_interpolant" and self.scheme != "weno5":
            fn = {"eno3": "vsl_boundary_interpolate_eno3", "enork2": "vsl_enork2_boundary_interpolate"}[self.scheme]
        self.vsl.call(fn, *map(ptr, fields), *self.tail)

    def reinit(self, iters):
        def step(f):
            out = empty(self.g.Size)
            self.call("re_step", out, f, self.mask, self.dt, *self.d)
            return out

        f = self.F
        for _ in range(iters):
            f = self.march(f, step)
        return f

    def extend(self, C, iters):
        n = [empty(self.g.Size) for _ in range(3)]
        self.call("upwind_normal", *n, self.F, *self.d)
        r = torch.sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2])
        r = torch.where(r < 1e-6, 1e-6, r)
        s = torch.where(self.F > 0, 1.0, torch.where(self.F < 0, -1.0, 0.0)).double()
        v = [s * (t / r) for t in n]
        cp = [empty(self.g.Size, fill=0.0) for _ in range(6)]
        C = dev(C)
        self.call("boundary_interpolant", *cp, *self.d, C)

        def step(f):
            out = empty(self.g.Size)
            self.call("extend_step", out, self.dt, f, *v, *self.d, *cp)
            return out

        for _ in range(iters):
            C = self.march(C, step)
        return C

    def advect(self, v, dt, steps):
        def step(f):
            out = empty(self.g.Size)
            self.vsl.call("vsl_advection_step", ptr(out), *map(ptr, v), ptr(f), *self.g.args(), stream())
            return dt * out

        f = self.F
        for _ in range(steps):
            f = self.march(f, step)
        return f


@pytest.mark.parametrize("kind", ["plain", "nonfinite", "huge", "tiny", "zero"])
@pytest.mark.parametrize("size", SIZES)
def test_stages_are_the_general_code(pkg, vsl, size, kind):
    h = (0.07, 0.09, 0.08)
    x, y, z, F0 = level_set(size, h, 0.35 * min(max(size) * 0.08, 3.0), 1)
    F = plant(F0, kind)
    C = plant(np.asfortranarray(np.cos(2 * x) + y * z), kind)
    m = pkg.SDF3(pkg.GD3(x, y, z, spacing=h), Val=F, precision="f64")
    m.setDistance()
    L = {s: Loops(vsl, m, F, s) for s in ("weno5", "eno3", "enork2")}
    v = [dev(t) for t in (np.sin(y + 1), np.cos(x), np.where(z > 0, -0.0, z))]
    pairs = {
        "reinit": (m.WENO5RK3Reinitialization(F, 3), L["weno5"].reinit(3)),
        "reinit_eno3": (m.WENORK3Reinitialization(F, 2), L["eno3"].reinit(2)),
        "reinit_enork2": (m.ENORK2Reinitialization(F, 3), L["enork2"].reinit(3)),
        "extend": (m.WENO5RK3Extend(C, 3), L["weno5"].extend(C, 3)),
        "extend_eno3": (m.WENORK3Extend(C, 2), L["eno3"].extend(C, 2)),
        "extend_enork2": (m.ENORK2Extend(C, 3), L["enork2"].extend(C, 3)),
        "advect": (m.WENO5RK3Advection(F, *v, 0.02, 2), L["weno5"].advect(v, 0.02, 2)),
    }
    bad = {}
    for name, (got, want) in pairs.items():
        got, want = host(got), host(want)
        if not np.array_equal(got, want, equal_nan=True):
            off = ~((got == want) | (np.isnan(got) & np.isnan(want)))
            bad[name] = (int(off.sum()), got[off][:3], want[off][:3])
    assert not bad, bad


@pytest.mark.parametrize("h", [1e-30, 1e25])
def test_extreme_spacings_take_the_general_code(pkg, vsl, oracle_mod, h):
    O = oracle_mod
    K = O.kernels("port_crpow")
    size = (9, 7, 6)
    x, y, z, F = level_set(size, (h, h, h), 2.1 * h, 0)
    F = np.asfortranarray(np.sqrt(x**2 + y**2 + (z + 0.1 * h)**2) - 2.1 * h)
    g = O.Grid(*size, h, h, h)
    m = pkg.SDF3(pkg.GD3(x, y, z, spacing=(h, h, h)), Val=F, precision="f64")
    m.setDistance()
    with np.errstate(all="ignore"):
        want = O.reinit_weno5(K, g, F, 2, O.set_distance(K, g, F))
    assert np.array_equal(host(m.WENO5RK3Reinitialization(F, 2)), want, equal_nan=True)
