"""The bi-Laplacian smoothing's symbol tables against numpy's FFT with the symbol written out:
uneven small grids, and one axis too long for the tables in shared memory.  FP64 to 1e-12 and
FP32 to 2e-6 of the norm (the transforms' rounding, about eps sqrt(log2 N) each way).  The fixed-
order sums of the block partials: fewer partials than a warp, than a block, and more."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

sdf3 = importlib.import_module("2018_7_vesicle_gb300.sdf3")


def grid_of(size, spacing=(0.05, 0.0625, 0.04)):
    rows, cols, pges = size
    axes = [(np.arange(n) - (n - 1) / 2) * h for n, h in zip((cols, rows, pges), spacing)]
    return sdf3.GD3(*sdf3.GD3.meshgrid(*axes), spacing=spacing)


@pytest.mark.parametrize("size", [(5, 3, 2), (33, 32, 31), (6150, 2, 3)])
@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_symbol_against_numpy(size, exact, dtype):
    grid = grid_of(size)
    rhs = np.random.default_rng(2).normal(size=size)
    rhs32 = torch.tensor(rhs, dtype=dtype, device="cuda")
    dt, alpha = 3e-6, 0.7
    got = (grid.smoothGMRES if exact else grid.smoothFFT)(rhs32, dt, alpha,
                                                          precision="f64" if dtype == torch.float64 else "f32")
    parts = []
    for dim, h in zip((1, 0, 2), (grid.Dx, grid.Dy, grid.Dz)):
        n = size[dim]
        if exact:
            p = (2 * np.cos(2 * np.pi * np.arange(n) / n) - 2) / h**2
        else:
            p = 2 * np.pi * (-0.5 * n + (np.arange(n) - n // 2) % n) / (n * h)
        shape = [1, 1, 1]
        shape[dim] = n
        parts.append(p.reshape(shape))
    s = sum(parts) if exact else sum(p**2 for p in parts)
    want = np.real(np.fft.ifftn(np.fft.fftn(rhs32.double().cpu().numpy()) / (1 + alpha * dt * s**2)))
    err = np.linalg.norm(got.double().cpu().numpy() - want) / np.linalg.norm(want)
    assert err <= (1e-12 if dtype == torch.float64 else 2e-6), err


@pytest.mark.parametrize("size", [(3, 4, 5), (32, 8, 33), (20, 24, 40), (64, 64, 70)])
def test_sums_of_partials(size):
    """Area and volume against the toolbox fields' own sums (FP64, 1e-12)."""
    grid = grid_of(size)
    F = torch.sqrt(grid.X**2 + grid.Y**2 + grid.Z**2) - 0.2 * max(size) * 0.05
    m = sdf3.SDF3(grid, Val=F, precision="f64")
    got = m.area_volume().cpu().numpy()
    m.GPUsetCalculusToolBox()
    ds = (grid.Dx + grid.Dy + grid.Dz) / 3
    delta, heav = m.DiracDelta, m.Heaviside
    area = float(torch.where(m.F.abs() < 2 * ds, delta, 0 * delta).sum()) * ds**3
    vol = float(torch.where(m.F < 2 * ds, 1 - heav, 0 * heav).sum()) * ds**3
    assert abs(got[0] - area) <= 1e-12 * abs(area) + 1e-300
    assert abs(got[1] - vol) <= 1e-12 * abs(vol)
