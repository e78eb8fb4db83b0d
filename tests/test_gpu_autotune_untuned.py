"""The tuner and the library's own choice of pages per block: the launch of an untuned shape is among
the timed candidates, so that the kept choice is never slower than it, and `launch_pages` reports
what a shape launches with.  GPU only."""
import importlib

import pytest

from test_gpu_autotune import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(33, 40, 36), (96, 64, 7)])
@pytest.mark.parametrize("candidates", ["default", "waves"])
def test_untuned_launch_is_a_candidate(pkg, vsl, size, candidates):
    T = importlib.import_module(pkg.__name__ + ".autotune")
    m = make(pkg, size)
    own = {k: T.launch_pages(size, k) for k in T.KINDS}
    assert all(1 <= p <= T.DEFAULT_PAGES for p in own.values()) and own["reinit"] < 4
    report = T.tune_shape(m, iters=1, reps=1, **({} if candidates == "default" else {"candidates": "waves"}))
    for kind, r in report.items():
        assert own[kind] in r["ms"] and r["ms"][r["pages"]] <= r["ms"][own[kind]]
        assert T.launch_pages(size, kind) == T.get_pages(size, kind) == r["pages"]
    T.clear_shape(size)
    assert {k: T.launch_pages(size, k) for k in T.KINDS} == own
