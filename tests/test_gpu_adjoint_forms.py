"""The adjoint's passes where their split into paths can go wrong.

* Advection: one step against autograd through the same WENO5 TVD-RK3 update written in torch
  (FP64), on grids narrower than a stencil and around the 32 x 8 block, with differences inside
  and outside the range of the short quotients.  The fields are rough (differences of the size
  of the values), so a partial's rounding is a few tens of the type's epsilon: 1e-4 of the
  largest partial in FP32, 1e-11 in FP64.
* Reinitialization: FP64 directional derivative against central differences (step 1e-6: 1e-10
  of truncation and of cancellation each; 1e-5 as elsewhere) on narrow grids, whose band nodes'
  stencils reach past two faces at once."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 4, 9), (3, 33, 5), (33, 9, 2), (64, 7, 3)]  # rows (y), cols (x), pges (z)


@pytest.fixture(scope="module")
def A(pkg, vsl):
    return importlib.import_module(pkg.__name__ + ".adjoint")


@pytest.fixture(scope="module")
def S(pkg):
    return importlib.import_module(pkg.__name__ + ".sdf3")


def make_grid(S, size):
    rows, cols, pges = size
    spacing = (0.1, 0.125, 0.11)
    return S.GD3(*S.GD3.meshgrid(*[np.arange(n) * h for n, h in zip((cols, rows, pges), spacing)]), spacing=spacing)


def weno5(v):
    """One-sided derivative from five first differences, biased toward the third."""
    v1, v2, v3, v4, v5 = v
    q = (v1 / 3 - 7 / 6 * v2 + 11 / 6 * v3, -v2 / 6 + 5 / 6 * v3 + v4 / 3, v3 / 3 + 5 / 6 * v4 - v5 / 6)
    s = (13 / 12 * (v1 - 2 * v2 + v3) ** 2 + (v1 - 4 * v2 + 3 * v3) ** 2 / 4,
         13 / 12 * (v2 - 2 * v3 + v4) ** 2 + (v2 - v4) ** 2 / 4,
         13 / 12 * (v3 - 2 * v4 + v5) ** 2 + (3 * v3 - 4 * v4 + v5) ** 2 / 4)
    a = [d / (sk + 1e-6) ** 2 for d, sk in zip((0.1, 0.6, 0.3), s)]
    return sum(ak * qk for ak, qk in zip(a, q)) / sum(a)


def stage(p, vel, h, dt):
    """dt * sum over the axes of min(0, v) D+ + max(0, v) D-; lines clamped at the faces."""
    out = 0
    for dim, v, hh in zip((1, 0, 2), vel, h):  # x runs along the columns
        n = p.shape[dim]
        line = [p.index_select(dim, (torch.arange(n, device=p.device) + s).clamp(0, n - 1)) for s in range(-3, 4)]
        d = [(line[m + 1] - line[m]) / hh for m in range(6)]
        out = out + v.clamp(max=0) * weno5(d[:0:-1]) + v.clamp(min=0) * weno5(d[:5])
    return dt * out


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("amplitude", ["one", "large"])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_advection_step_against_autograd(A, S, size, amplitude, precision):
    grid = make_grid(S, size)
    scale = 1.0 if amplitude == "one" else (1e5 if precision == "f32" else 1e33)
    dtype = torch.float32 if precision == "f32" else torch.float64
    rng = np.random.default_rng(21)
    phi, w = (torch.tensor(rng.normal(size=size), dtype=dtype, device="cuda") for _ in range(2))
    phi = phi * scale
    vel = [torch.tensor(rng.normal(size=size), dtype=dtype, device="cuda") for _ in range(3)]
    dt = 0.0078125
    tr = A.Transport(grid, dt, A.TransportPlan(steps=1, reinit_every=0, reinit_iters=0, checkpoint_every=1), precision)
    args = [S.as_field(t, dtype).clone().requires_grad_(True) for t in (phi, *vel)]
    (tr(*args) * w).sum().backward()

    p, *v = [t.double().clone().requires_grad_(True) for t in (phi, *vel)]
    h = (grid.Dx, grid.Dy, grid.Dz)
    u1 = p - stage(p, v, h, dt)
    u2 = 0.75 * p + 0.25 * (u1 - stage(u1, v, h, dt))
    u3 = p / 3 + 2 / 3 * (u2 - stage(u2, v, h, dt))
    (u3 * w.double()).sum().backward()
    tol = 1e-4 if precision == "f32" else 1e-11
    for got, want in zip(args, (p, *v)):
        err, top = float((got.grad.double() - want.grad).abs().max()), float(want.grad.abs().max())
        assert err <= tol * top, (err, top)


@pytest.mark.parametrize("size", [(5, 33, 4), (9, 6, 40)])
def test_reinitialization_on_narrow_grids(A, S, size):
    grid = make_grid(S, size)
    X, Y, Z = (t - t.mean() for t in (grid.X, grid.Y, grid.Z))
    # two fronts across the long axis
    along = X if size[1] > size[2] else Z
    phi0 = S.as_field((along.abs() - 0.83) * (1 + 0.2 * along ** 2) + 0.05 * torch.sin(7 * Y + 5 * X + 3 * Z + 0.4),
                      torch.float64)
    zero = [torch.zeros_like(phi0) for _ in range(3)]
    tr = A.Transport(grid, 1e-3, A.TransportPlan(steps=1, reinit_every=1, reinit_iters=2, checkpoint_every=1), "f64")
    w = S.as_field(torch.cos(3 * X + 2 * Y - Z), torch.float64)
    d = S.as_field(torch.sin(2 * X - 3 * Y + 4 * Z + 0.2), torch.float64)
    p0 = phi0.clone().requires_grad_(True)
    (tr(p0, *zero) * w).sum().backward()
    with torch.no_grad():
        plus, minus = (float((tr(phi0 + s * 1e-6 * d, *zero) * w).sum()) for s in (1, -1))
    fd, an = (plus - minus) / 2e-6, float((p0.grad * d).sum())
    assert abs(fd - an) <= 1e-5 * abs(an), (fd, an)
