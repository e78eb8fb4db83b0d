"""The FP64 WENO stage kernels with two pages to a block (grids of at least three times the band
blocks' count of such blocks), on a grid ragged in every direction with an odd last page: bit for
bit the general per-node code, as tests/test_gpu_stage64.py holds the one-page form.  GPU only."""
import pytest
import torch

import test_gpu_stage64 as one_page

pytestmark = pytest.mark.gpu

SIZE = (65, 70, 75)


@pytest.mark.parametrize("kind", ["plain", "nonfinite", "tiny"])
def test_two_pages_to_a_block(pkg, vsl, kind):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, cols, pges = SIZE
    assert -(-rows // 32) * -(-cols // 4) * ((pges + 1) // 2) >= 3 * 4 * sms
    one_page.test_stages_are_the_general_code(pkg, vsl, SIZE, kind)
