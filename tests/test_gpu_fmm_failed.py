"""An FMM evaluation that fails after its launches leaves nothing running that
the next call's tree, lists and staging would be written under."""
import numpy as np
import pytest

import amk
from conftest import gaussian_cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,order,leaf", [("fp64", 6, 32), ("tensor", 6, 128)])
def test_calls_after_a_failed_evaluation(monkeypatch, precision, order, leaf):
    big = gaussian_cloud(300000, 1)
    small = [gaussian_cloud(n, n) for n in (250000, 20011, 900)]
    with amk.Simulation() as s:
        s.set_fmm_precision(precision)
        want = [s.solve_fmm(*c, order, 0.5, leaf_capacity=leaf) for c in small]
    with amk.Simulation() as s:
        s.set_fmm_precision(precision)
        for c, w in zip(small, want):
            monkeypatch.setenv("AMK_FMM_FAIL", "1")
            with pytest.raises(Exception, match="AMK_FMM_FAIL"):
                s.solve_fmm(*big, order, 0.4, leaf_capacity=leaf)
            monkeypatch.delenv("AMK_FMM_FAIL")
            got = s.solve_fmm(*c, order, 0.5, leaf_capacity=leaf)
            for a, b in zip(got, w):
                assert np.array_equal(a, b)
