"""FP32 extensions of fields that hold infinities, NaN and values whose weights overflow, on a grid
whose band runs as tasks (which evaluate the upwind side alone): bit for bit the batched form, which
evaluates both sides, and NaN where that has NaN.  GPU only."""
import importlib

import numpy as np
import pytest
import torch

from test_gpu_stage64 import level_set

pytestmark = pytest.mark.gpu

SIZE, H = (64, 48, 40), (0.07, 0.09, 0.08)
VALUES = {"nonfinite": (np.inf, np.nan, -np.inf), "huge": (1e30,), "large": (1e12,)}


def same(a, b):
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(), b.nan_to_num())


@pytest.mark.parametrize("kind", VALUES)
def test_extension_of_odd_values(pkg, vsl, kind):
    B = importlib.import_module(pkg.__name__ + ".batch")
    x, y, z, F = level_set(SIZE, H, 0.9, 1)
    C = np.ascontiguousarray(np.cos(2 * x) + y * z)
    for q, v in enumerate(VALUES[kind]):
        C.reshape(-1)[11 + q::997] = v
    m = pkg.SDF3(pkg.GD3(x, y, z, spacing=H), Val=F, precision="f32")
    m.setDistance()
    C = m._field(torch.tensor(C))
    got = m.WENO5RK3Extend(C, 2)
    assert bool(torch.isnan(got).any()) and same(got, B.extend_batched([m], [C], 2)[0])
    got = m.WENORK3ClosetPointSurfaceRedistance(C, 1, 1)
    assert same(got, B.redistance_batched([m], [C], 1, 1, eno3=True)[0])
