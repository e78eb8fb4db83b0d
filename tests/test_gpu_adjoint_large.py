"""Gradients through advection and reinitialization at 128^3, the size that the differentiation
workload runs at, against central differences of the forward map: three directions of the initial
field (two smooth, one a bump on the interface) and the eight velocity amplitudes in FP64, the FP32
gradient against those.

Steps and tolerances.  The forward map jumps where an interface distance passes the fixed-node
threshold; of the 120,000 crossed edges here a change of the field by d carries d / spacing past it, so
the steps (1e-8 of the field, 1e-7 of the amplitudes, which move the field a tenth as far) are those
that carry none.  The fields are subtracted before they are summed: rounding 1e-16 / 1e-8 per node,
and 1e-16 / 1e-7 of a loss that is half its gradient: below 1e-6, 1e-5 asked.  FP32: 1e-3 on the small
grid (spacing 0.1) is the field's rounding over the spacing; 0.016 here: 5e-3."""
import numpy as np
import pytest
import torch

from test_gpu_adjoint import A, S, amplitude_gradient, colmajor, mismatch_setup, smooth_weight  # noqa: F401

pytestmark = pytest.mark.gpu

SIZE = (128, 128, 128)


def test_field_directions(A, S):  # noqa: F811
    grid, phi0, modes, a0, _, dt, plan, _, _ = mismatch_setup(A, S, SIZE, steps=2)
    v = [colmajor(S, t) for t in A.velocity(a0, modes)]
    tr = A.Transport(grid, dt, plan, "f64")
    w = colmajor(S, smooth_weight(grid, 8))
    p0 = phi0.clone().requires_grad_(True)
    (tr(p0, *v) * w).sum().backward()
    X, Y, Z = grid.X, grid.Y, grid.Z
    bump = torch.exp(-((X - 0.6) ** 2 + (Y + 0.03) ** 2 + Z ** 2) / 0.1 ** 2)
    for d in (smooth_weight(grid, 9), smooth_weight(grid, 10), bump):
        d = colmajor(S, d)
        with torch.no_grad():
            fd = float(((tr(phi0 + 1e-8 * d, *v) - tr(phi0 - 1e-8 * d, *v)) * w).sum()) / 2e-8
        an = float((p0.grad * d).sum())
        assert abs(fd - an) <= 1e-5 * abs(an), (fd, an)


def test_amplitudes(A, S):  # noqa: F811
    setup = mismatch_setup(A, S, SIZE, steps=4)
    grid, phi0, modes, a0, _, dt, plan, eps, dv = setup
    _, g64, tr, target = amplitude_gradient(A, S, "f64", setup)
    _, g32, _, _ = amplitude_gradient(A, S, "f32", setup)

    def loss(a):
        with torch.no_grad():
            return float(A.heaviside_mismatch(tr(phi0, *A.velocity(a, modes)), target, eps, dv))

    fd = np.zeros(8)
    for m in range(8):
        e = torch.zeros(8, dtype=torch.float64, device="cuda")
        e[m] = 1e-7
        fd[m] = (loss(a0 + e) - loss(a0 - e)) / 2e-7
    top = np.abs(fd).max()
    assert np.abs(fd - g64).max() <= 1e-5 * top, (fd, g64)
    assert np.abs(g32 - g64).max() <= 5e-3 * top, (g32, g64)
