"""Reinitialization of fields with more band nodes than run as tasks (interfaces a few nodes apart
through the whole grid), FP32: bit for bit the batched form, whose band never does.  GPU only."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZE, H = (64, 60, 56), (0.05, 0.055, 0.06)


@pytest.mark.parametrize("period,dense", [(0.55, True), (8.0, False)])
def test_dense_band_is_the_batched_form(pkg, vsl, period, dense):
    B = importlib.import_module(pkg.__name__ + ".batch")
    S = importlib.import_module(pkg.__name__ + ".shapes")
    rows, cols, pges = SIZE
    x, y, z = S.meshgrid(*[(np.arange(n) - (n - 1) / 2) * h for n, h in zip((cols, rows, pges), H)], device="cuda")
    k = 2 * np.pi / period
    F = (torch.sin(k * x) * torch.cos(k * y) + torch.sin(k * y) * torch.cos(k * z) + torch.sin(k * z) * torch.cos(k * x)) / k + 0.001
    crossed = torch.zeros_like(F, dtype=torch.bool)
    for d, n in enumerate(F.shape):
        s = F.narrow(d, 0, n - 1) * F.narrow(d, 1, n - 1) < 0
        crossed.narrow(d, 0, n - 1).logical_or_(s)
        crossed.narrow(d, 1, n - 1).logical_or_(s)
    assert (int(crossed.sum()) > 80000) == dense  # REINIT_TASKS_MOST: 40000
    m = pkg.SDF3(pkg.GD3(x, y, z, spacing=H), Val=F, precision="f32")
    m.setDistance()
    assert torch.equal(m.WENO5RK3Reinitialization(m.F, 4), B.reinitialize_batched([m], [m.F], 4)[0])
    A = torch.sin(3 * x) * torch.cos(2 * y) + 0.5 * z**2 + F
    got = m.WENORK3ClosetPointSurfaceRedistance(A, 2, 1)
    assert torch.equal(got, B.redistance_batched([m], [A], 2, 1, eno3=True)[0])


@pytest.mark.parametrize("eno3", [False, True])
def test_redistance_of_a_wavy_field(pkg, vsl, eno3):
    """A surface field with 78,000 band nodes on an odd box, redistanced: the reinitialization stages
    see the extensions' outputs, whose values reach more of the stencils' branches."""
    B = importlib.import_module(pkg.__name__ + ".batch")
    S = importlib.import_module(pkg.__name__ + ".shapes")
    rows, cols, pges = 161, 113, 97
    half = [1.5 * n / rows if n < rows else 1.5 for n in (cols, rows, pges)]
    v = [np.linspace(-max(1.15, b), max(1.15, b), n) for b, n in zip(half, (cols, rows, pges))]
    x, y, z = S.meshgrid(*v, device="cuda")
    F = torch.sqrt(x**2 / 0.8 + y**2 / 0.6 + z**2 / 0.5) - 0.9 + 0.02 * torch.sin(2 * x + y - 1.5 * z)
    A = torch.sin(3 * x + 0.8) * torch.cos(2 * y + 0.2) + 0.5 * z**2
    m = pkg.SDF3(pkg.GD3(x, y, z, spacing=tuple(float(a[1] - a[0]) for a in v)), Val=F, precision="f32")
    fn = m.WENORK3ClosetPointSurfaceRedistance if eno3 else m.WENO5RK3ClosetPointSurfaceRedistance
    for it, ext in ((1, 1), (3, 2)):
        assert torch.equal(fn(A, it, ext), B.redistance_batched([m], [A], it, ext, eno3=eno3)[0])
