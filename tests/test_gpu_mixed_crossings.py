"""The mixed form's interface set-up: distances by the short root form and the block-wise crossing
values, against the FP64 form on the same (promoted) fields.

* Distances: both are roots of the same quintic, FP64 Brent on its monomial form to 1.4e-13 h, the
  short form to 4e-16 h, each rounded once to FP32 -- so they differ by an FP32 unit in the last
  place at most where 3e-13 h (the error of h less a distance included) crosses a rounding
  boundary.  That holds where the root is determined: one only in the cell (of several, Brent's
  choice turns on the rounding, in either precision) and not within 1e-6 h of a node; kinks take
  the quadratic formula, whose quotient by a small second difference differs with the rounding
  too.  There, and outside the range of the short form, the general form runs: the values are in
  the cell.
* Extension: the FP32 form's 5e-5 (as elsewhere) on grids narrower than the stencil and with less
  and more listed nodes than a block deals with at once."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

sdf3 = importlib.import_module("2018_7_vesicle_gb300.sdf3")
SPACING = (0.0371, 0.05, 0.04)


def grid_of(size):
    rows, cols, pges = size
    axes = [(np.arange(n) - (n - 1) / 2) * h for n, h in zip((cols, rows, pges), SPACING)]
    return sdf3.GD3(*sdf3.GD3.meshgrid(*axes), spacing=SPACING)


def field_of(grid, size, kind):
    rng = np.random.default_rng(5)
    X, Y, Z = (t.cpu().numpy() for t in (grid.X, grid.Y, grid.Z))
    F = np.sqrt((X - 0.011)**2 + (Y + 0.007)**2 + (Z - 0.003)**2) - 0.4 * max(size) * 0.04
    noise = rng.normal(size=size) * 0.04
    F = F + {"smooth": 0.0, "rough": 0.5, "folded": 2.0}.get(kind, 0.1) * noise
    if kind == "near":  # crossings next to nodes, and nodes on the surface
        F = np.where(rng.random(size) < 0.2, F * 1e-8, F)
        F = np.where(rng.random(size) < 0.05, 0.0, F)
    scale = {"large": 1e33, "small": 1e-25}.get(kind, 1.0)
    return torch.tensor((F * scale).astype(np.float32), device="cuda")


def determined(F, ax, u):
    """Forward edges along dim ax whose quintic falls or rises all the way, u away from its ends."""
    n = F.shape[ax]
    v = [np.take(F, np.clip(np.arange(n) + s, 0, n - 1), axis=ax) / np.abs(F).max() for s in range(-2, 4)]
    A = np.array([[0, 6, -5, -5, 5, -1], [0, -60, 80, -5, -20, 5], [120, -40, -150, 50, 30, -10],
                  [0, 120, 80, -70, -20, 10], [0, -30, -5, 35, 5, -5], [0, 4, 0, -5, 0, 1]])  # of sample m, u^p / 120
    c = [sum(A[m, p] * v[m] for m in range(6)) for p in range(6)]
    slope = np.stack([sum(p * c[p] * t**(p - 1) for p in range(1, 6)) for t in np.linspace(0, 1, 33)])
    mono = np.all(slope > 0.02 * np.abs(c[1]), axis=0) | np.all(slope < -0.02 * np.abs(c[1]), axis=0)
    kink = (v[1] * v[2] < 0) | (v[3] * v[4] < 0)
    return (v[2] * v[3] < 0) & ~kink & mono & (u > 1e-6) & (u < 1 - 1e-6)


@pytest.mark.parametrize("size", [(1, 9, 14), (6, 33, 7), (40, 37, 35)])
@pytest.mark.parametrize("kind", ["smooth", "rough", "folded", "near", "large", "small"])
def test_distances_are_the_fp64_roots_rounded(size, kind):
    grid = grid_of(size)
    F = field_of(grid, size, kind)
    m32, m64 = (sdf3.SDF3(grid, Val=F.to(t), precision=p) for t, p in ((torch.float32, "f32"), (torch.float64, "f64")))
    m32.setDistance()
    m64.setDistance()
    checked = 0
    d32, d64 = ([t.cpu().numpy() for t in m._dist()] for m in (m32, m64))
    for q in range(3):
        ax, h = (1, 0, 2)[q], (grid.Dx, grid.Dy, grid.Dz)[q]
        single = determined(F.double().cpu().numpy(), ax, d64[2 * q] / h)
        checked += int(single.sum())
        for which, far in ((2 * q, 0), (2 * q + 1, 1)):
            # the far end of the edge holds h less the distance
            a, b = (np.roll(d[which], -far, axis=ax) for d in (d32, d64))
            off = np.abs(a.astype(np.float64) - b.astype(np.float32).astype(np.float64))
            assert np.all(off[single] <= (np.spacing(np.maximum(a, b.astype(np.float32))) + 3e-13 * h)[single])
            assert np.all(np.isnan(a) | ((a >= 0) & (a <= np.float32(h))))
            assert np.array_equal(np.isnan(a), np.isnan(b))
    assert checked > 0


@pytest.mark.parametrize("size", [(3, 12, 5), (9, 8, 7), (35, 31, 29)])
@pytest.mark.parametrize("eno3", [False, True])
def test_extension_against_fp64(size, eno3):
    grid = grid_of(size)
    F = field_of(grid, size, "smooth")
    C = torch.cos(9 * grid.X + 7 * grid.Y) * torch.sin(8 * grid.Z + 0.3)
    out = []
    for prec, t in (("f32", torch.float32), ("f64", torch.float64)):
        m = sdf3.SDF3(grid, Val=F.to(t), precision=prec)
        m.setDistance()
        f = m.WENORK3Extend if eno3 else m.WENO5RK3Extend
        out.append(f(sdf3.as_field(C.float(), t), 5).double())
    err = float((out[0] - out[1]).norm() / out[1].norm())
    assert err <= 5e-5, err


@pytest.mark.parametrize("size", [(31, 7, 3), (33, 17, 40), (70, 64, 61), (160, 150, 140)])
def test_area_and_volume_terms_over_the_block(size):
    """The FP32 form's FP64 terms of the promoted field, pooled per warp and per block, against the
    plain form on that field: the same terms to a few FP64 roundings each, summed in another order."""
    grid = grid_of(size)
    F = field_of(grid, size, "smooth")
    a32, a64 = (sdf3.SDF3(grid, Val=F.to(t), precision=p).area_volume().cpu().numpy()
                for t, p in ((torch.float32, "f32"), (torch.float64, "f64")))
    assert np.all(np.abs(a32 - a64) <= 1e-11 * np.abs(a64)), (a32, a64)
