"""FP64 workspaces that do not grow (no GPU): the bytes at 13 x 9 x 11 nodes of the operations whose
list of flagged nodes shares storage that is free by then, or that have no such list."""
import pytest

SIZES = {"reinit_eno3": 101888, "surface_redistance": 303872, "advection": 22528, "advection_adjoint": 259840,
         "reinit_adjoint": 407808,
         "reinit_enork2": 101888, "surface_redistance_enork2": 303872, "surface_redistance_eno3": 303872}


@pytest.mark.parametrize("op", SIZES)
def test_fp64_workspace_bytes(vsl, op):
    assert vsl.workspace_bytes(op, 13, 9, 11, 8) == SIZES[op]
