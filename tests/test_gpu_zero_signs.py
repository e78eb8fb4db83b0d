"""The sign of zeros in the plain FP64 form: a quotient of a zero keeps its sign, as the general
division does.  Toolbox fields of planar level sets (whose cross products and curvatures are zeros
of either sign) against the oracle, bit for bit.  GPU only."""
import numpy as np
import pytest

from gpu_util import dev, host
from test_gpu_stage64 import level_set

pytestmark = pytest.mark.gpu

SIZE = (9, 35, 6)


def same_bits(a, b):
    a, b = (np.ascontiguousarray(t, np.float64) for t in (a, b))
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("plane", [(0, 0, 1, 1, -1, 0), (0, 0, -1, -1, 1, 0), (1, 0, 0, 0, -1, 1), (0, 1, 0, 1, 0, -1)])
def test_toolbox_zeros(pkg, vsl, oracle_mod, plane):
    O = oracle_mod
    K = O.kernels("port_crpow")
    x, y, z, _ = level_set(SIZE, (0.125, 0.25, 0.5), 1.0, 0)
    a, b, c, d, e, f = plane
    F, A = (np.asfortranarray(t) for t in (a * x + b * y + c * z, d * x + e * y + f * z))
    g = O.grid_from_mesh(x, y, z)
    ref, tb = O.auxiliary_toolbox(K, g, F, A)
    m = pkg.SDF3(pkg.GD3(x, y, z), Val=F, precision="f64")
    m.A = dev(A)
    m.GPUAsetCalculusToolBox()
    m.GPUsetCalculusToolBox()
    kernel = [n for n in O.AUX_FIELDS if n not in ("AFDiracDelta", "ADiracDeltaDn")]
    off = [n for n in kernel if not same_bits(host(getattr(m, n)), ref[n])]
    off += [n for n in O.TOOLBOX_FIELDS if not same_bits(host(getattr(m, n)), tb[n])]
    assert any((np.signbit(ref[n]) & (ref[n] == 0)).any() for n in kernel)
    assert not off
