"""Rounding of the FP64 advection adjoint: the gradient of one WENO5 TVD-RK3 step against the same
step differentiated on numpy's long doubles (forward mode, all directions at once).

The field is smooth on its grid, as fields of the workload are, so that the partials of the weights
come from differences of nearly equal candidates.  Tolerance: a gradient's entry sums 21 partials in
each of three stages, each rounded a few tens of times on terms no larger than the largest: a
hundred of FP64's epsilon, 2.2e-14 of the largest entry.  GPU only."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LD = np.longdouble
SIZE, H, DT = (7, 6, 8), (0.05, 0.055, 0.06), 0.0078125  # rows (y), cols (x), pges (z); hx, hy, hz


class Dual:
    """Values and their derivatives by every input (leading axis of d)."""

    def __init__(self, v, d):
        self.v, self.d = v, d

    def __add__(self, o):
        return Dual(self.v + o.v, self.d + o.d) if isinstance(o, Dual) else Dual(self.v + o, self.d)

    __radd__ = __add__

    def __neg__(self):
        return Dual(-self.v, -self.d)

    def __sub__(self, o):
        return self + (-o)

    def __mul__(self, o):
        return Dual(self.v * o.v, self.d * o.v + self.v * o.d) if isinstance(o, Dual) else Dual(self.v * o, self.d * o)

    __rmul__ = __mul__

    def inverse(self):
        return Dual(1 / self.v, -self.d / (self.v * self.v))

    def take(self, dim, idx):
        return Dual(np.take(self.v, idx, dim), np.take(self.d, idx, dim + 1))


def ratio(a, b):
    return LD(a) / LD(b)


def weno5(v):
    v1, v2, v3, v4, v5 = v
    q = (v1 * ratio(1, 3) - v2 * ratio(7, 6) + v3 * ratio(11, 6), v2 * ratio(-1, 6) + v3 * ratio(5, 6) + v4 * ratio(1, 3),
         v3 * ratio(1, 3) + v4 * ratio(5, 6) - v5 * ratio(1, 6))
    sq = lambda x: x * x  # noqa: E731
    s = (sq(v1 - 2 * v2 + v3) * ratio(13, 12) + sq(v1 - 4 * v2 + 3 * v3) * ratio(1, 4),
         sq(v2 - 2 * v3 + v4) * ratio(13, 12) + sq(v2 - v4) * ratio(1, 4),
         sq(v3 - 2 * v4 + v5) * ratio(13, 12) + sq(3 * v3 - 4 * v4 + v5) * ratio(1, 4))
    a = [sq((sk + LD(1e-6)).inverse()) * d for d, sk in zip((LD(0.1), LD(0.6), LD(0.3)), s)]
    tot = (a[0] + a[1] + a[2]).inverse()
    return (a[0] * q[0] + a[1] * q[1] + a[2] * q[2]) * tot


def stage(p, vel):
    out = None
    for dim, v, h in zip((1, 0, 2), vel, H):
        n = p.v.shape[dim]
        line = [p.take(dim, np.clip(np.arange(n) + s, 0, n - 1)) for s in range(-3, 4)]
        d = [(line[m + 1] - line[m]) * (1 / LD(h)) for m in range(6)]
        t = weno5(d[:0:-1]) * np.minimum(v, 0) + weno5(d[:5]) * np.maximum(v, 0)
        out = t if out is None else out + t
    return out * LD(DT)


def test_fp64_advection_gradient(pkg, vsl):
    A, S = (importlib.import_module(pkg.__name__ + "." + n) for n in ("adjoint", "sdf3"))
    rows, cols, pges = SIZE
    x, y, z = np.meshgrid(*[np.arange(n) * h for n, h in zip((cols, rows, pges), H)])
    phi = np.sqrt((x - 0.11)**2 + (y - 0.17)**2 + (z - 0.2)**2 + 0.01) - 0.2 + 0.02 * np.sin(9 * x + 7 * y - 5 * z)
    vel = [np.sin(5 * y + 1), np.cos(4 * z), np.sin(3 * x - 0.4)]
    w = np.cos(6 * x + 2) * np.sin(5 * y + 3 * z)
    n = phi.size
    p = Dual(phi.astype(LD), np.eye(n, dtype=LD).reshape(n, *SIZE))
    v = [t.astype(LD) for t in vel]
    u1 = p - stage(p, v)
    u2 = p * ratio(3, 4) + (u1 - stage(u1, v)) * ratio(1, 4)
    u3 = p * ratio(1, 3) + (u2 - stage(u2, v)) * ratio(2, 3)
    want = (u3.d * w.astype(LD)).sum(axis=(1, 2, 3)).reshape(SIZE)

    grid = S.GD3(*S.GD3.meshgrid(*[np.arange(m) * h for m, h in zip((cols, rows, pges), H)]), spacing=H)
    tr = A.Transport(grid, DT, A.TransportPlan(steps=1, reinit_every=0, reinit_iters=0, checkpoint_every=1), "f64")
    args = [S.as_field(torch.tensor(t, device="cuda"), torch.float64).clone().requires_grad_(True) for t in (phi, *vel)]
    (tr(*args) * torch.tensor(w, device="cuda")).sum().backward()
    got = args[0].grad.cpu().numpy()
    err = float(np.abs(got.astype(LD) - want).max() / np.abs(want).max())
    print("error", err)
    assert err <= 2.2e-14
