"""The plain form's FP64 kernels are compiled in the files that round every product by itself, and
only there: none of them is in the FP32 form's object files (no GPU; the host stubs' names)."""
import os
import shutil
import subprocess

import pytest

FP64 = ("k_toolbox64", "k_auxi_dropin", "tool64", "k_weno64", "k_eno64")


@pytest.mark.parametrize("name", ["vsl_toolbox_f32", "vsl_auxi_f32", "vsl_fused_f32", "vsl_relax_f32"])
def test_fp32_objects_hold_no_fp64_kernel(vsl, name):
    if shutil.which("nm") is None:
        pytest.skip("no nm")
    obj = os.path.join(os.path.dirname(vsl.path), "obj", name + ".o")
    names = subprocess.run(["nm", obj], capture_output=True, text=True, check=True).stdout
    assert "stub" in names
    assert not [k for k in FP64 if k in names]
