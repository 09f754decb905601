"""A depth of -0.0 is a dry cell, not a negative depth: a lake with islands
whose dry cells hold -0.0 takes the steps that it takes with 0.0, value for value."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["fwave", "hllc"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_dry_cells_of_negative_zero_depth(precision, method):
    from braids_hkt_gb300.solver import RiverSolver
    case = S.lake_at_rest()
    plus = case["q"].copy()
    dry = plus[0] == 0.0
    assert dry.any()
    minus = plus.copy()
    minus[0, dry] = -0.0
    a, b = (RiverSolver(case, precision=precision, method=method) for _ in range(2))
    a.set_state(plus)
    b.set_state(minus)
    assert int(a.substep(0.01)[0]) == int(b.substep(0.01)[0]) == 0
    np.testing.assert_array_equal(a.state(), b.state())
    a.set_state(plus)
    b.set_state(minus)
    da, db = a.advance(0.5, 0.0), b.advance(0.5, 0.0)
    assert da["failed"] == db["failed"] == 0 and da["hydraulic_rejections"] == db["hydraulic_rejections"]
    assert da["hydraulic_substeps"] == db["hydraulic_substeps"]
    np.testing.assert_array_equal(a.state(), b.state())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_step_leaves_no_negative_zero_depth(precision):
    from braids_hkt_gb300.solver import RiverSolver
    case = S.lake_at_rest()
    q = case["q"].copy()
    q[0, q[0] == 0.0] = -0.0
    s = RiverSolver(case, precision=precision)
    s.set_state(q)
    s.substep(0.01)
    assert not np.signbit(s.state()[0]).any()
