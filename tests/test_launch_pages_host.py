"""The library's choice of pages per block (no GPU: the rule, at its stand-in number of SMs): flat grids
whose blocks already fill the GPU are not split further, where the split was measured to be slower
than the default; small grids are split."""
import importlib

import pytest

T = importlib.import_module("2018_7_vesicle_gb300.autotune")


@pytest.mark.parametrize("size,kind", [((300, 300, 6), "extend"), ((300, 300, 6), "enork2_extend"),
                                       ((256, 256, 8), "extend"), ((100, 100, 7), "extend"), ((640, 640, 3), "enork2_extend")])
def test_full_flat_grids_stay_whole(vsl, size, kind):
    assert T.launch_pages(size, kind) >= size[2]


@pytest.mark.parametrize("kind", list(T.KINDS))
def test_small_grids_are_split(vsl, kind):
    assert T.launch_pages((64, 64, 64), kind) <= 5
    assert T.launch_pages((256, 256, 256), kind) == T.DEFAULT_PAGES
