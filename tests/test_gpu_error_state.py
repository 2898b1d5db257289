"""A call that failed says so once: the next calls do not report its error."""
import numpy as np
import pytest

import gmr

pytestmark = pytest.mark.gpu


def test_a_failed_call_leaves_no_error_behind():
    m = gmr.gen_mosaic(300, 64, 8, 0.02, 0.002, 3)
    plan = gmr.Plan.build(gmr.repair(m, 1), 300, 64)
    x = np.ones((64, 2), np.float32)
    want = gmr.Engine(plan).multiply(x, 0)
    for call in (lambda: gmr.Engine(plan, device=63), lambda: gmr.repair(m, device=63),
                 lambda: gmr.Plan.build(gmr.repair(m, 1), 300, 64, device=63)):
        with pytest.raises(gmr.GmrError):
            call()
        eng = gmr.Engine(plan)
        assert np.abs(eng.multiply(x, 0) - want).max() <= 1e-5 * np.abs(want).max()
