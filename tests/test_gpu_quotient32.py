"""The FP32 short quotients of the adjoint (Short32 of csrc/vsl_adjoint.cu, compiled from its text)
on the GPU: the reciprocal that they correct with is the correctly rounded one for every
significand.  That of ones is the one for which an ulp's error of the hardware reciprocal would
not do.  GPU only."""
import importlib
import os
import re
import subprocess

import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2018_7_vesicle_gb300", "csrc")

MAIN = r"""
#include <cstdio>
__global__ void check(unsigned *bad, int e)
{
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 threads
    const float b = __int_as_float((unsigned)(127 + e) << 23 | m);
    if ((Short32(1.f) / Short32(b)).v != __frcp_rn(b)) atomicAdd(bad, 1u);
}
int main()
{
    unsigned *bad, n = 0;
    if (cudaMalloc(&bad, sizeof n) != cudaSuccess || cudaMemset(bad, 0, sizeof n) != cudaSuccess) return 1;
    for (int e = -40; e <= 40; e += 8) check<<<(1 << 23) / 256, 256>>>(bad, e);
    if (cudaMemcpy(&n, bad, sizeof n, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("%u\n", n);
    return 0;
}
"""


def test_reciprocals_of_all_significands(pkg, tmp_path):
    B = importlib.import_module(pkg.__name__ + "._build")
    with open(os.path.join(CSRC, "vsl_adjoint.cu")) as f:
        struct = re.search(r"^struct Short32 \{.*?^\};", f.read(), flags=re.M | re.S).group(0)
    with open(os.path.join(CSRC, "vsl_device.cuh")) as f:
        rcp = re.search(r"^__device__ __forceinline__ float rcp_ftz\(float x\)\n\{.*?^\}", f.read(), flags=re.M | re.S).group(0)
    (tmp_path / "q.cu").write_text(rcp + "\n" + struct + MAIN)
    exe = tmp_path / "q"
    subprocess.run([B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "-o", str(exe), str(tmp_path / "q.cu")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, check=True)
    assert r.stdout.split() == ["0"]
