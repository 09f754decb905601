"""A state that is not finite is refused by the f-wave method in both forms: the
trial reports a status and the interval fails as the oracle's does, with the
bound state as it was."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("make", [S.small_channel, S.cartesian_channel])
@pytest.mark.parametrize("row,value", [(0, np.nan), (0, np.inf), (0, -1.0), (0, -np.inf), (1, np.nan), (1, np.inf),
                                       (2, -np.inf), (2, np.nan)])
def test_nonfinite_or_negative_cell(make, row, value, precision):
    from braids_hkt_gb300.solver import RiverSolver
    case = make()
    q = case["q"].copy()
    q[row, case["mesh"].nc // 2] = value
    s = RiverSolver(case, precision=precision)
    s.set_state(q)
    assert int(s.substep(0.004)[0]) != 0
    np.testing.assert_array_equal(s.state(), q)
    d = s.advance(0.05, 0.0, raise_on_failure=False)
    code, _, stats = Oracle(case).advance(q.copy(), 0.05, 0.0)
    assert code != 0 and d["failed"] != 0 and d["hydraulic_substeps"] == stats["substeps"] == 0
    np.testing.assert_array_equal(s.state(), q)


@pytest.mark.parametrize("make", [S.small_channel, S.cartesian_channel, S.dam_break])
@pytest.mark.parametrize("row,value,word", [(0, np.nan, 5), (0, np.inf, 5), (0, -1.0, 1), (1, np.nan, 5), (1, np.inf, 5),
                                            (2, -np.inf, 5), (1, 1e200, 5)])
def test_status_word(make, row, value, word):
    """Spatial (1) and rate (4) failures of the FP64 form. A wave speed that is not a
    number is passed over, as in the reference's extrema: no frequency failure (16)."""
    from braids_hkt_gb300.solver import RiverSolver
    case = make()
    q = case["q"].copy()
    q[row, int(np.argmax(q[0]))] = value
    s = RiverSolver(case)
    s.set_state(q)
    assert int(s.rate(0.004)[2]) & ~32 == word


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_residual_beside_a_dry_cell_of_nonfinite_momentum(value):
    """A dry cell's momentum takes no part: its residual fails (1), and the rates of
    its neighbours are those beside a dry cell at rest."""
    from braids_hkt_gb300.solver import RiverSolver
    case = S.lake_at_rest()
    q = S.perturbed_state(case, 3, 0.2, 0.5)
    dry = int(np.flatnonzero(q[0] == 0.0)[0])
    s = RiverSolver(case)
    s.set_state(q)
    rest = s.rate(0.004)
    q[1, dry] = value
    s.set_state(q)
    rate, water, status, freq = s.rate(0.004)
    assert int(rest[2]) == 0 and int(status) == 1 and freq == rest[3]
    np.testing.assert_array_equal(rate.cpu().numpy(), rest[0].cpu().numpy())
    np.testing.assert_array_equal(water.cpu().numpy(), rest[1].cpu().numpy())
    assert int(s.substep(0.004)[0]) == 0                 # the drag sets it to zero


def test_bed_update_of_a_state_that_is_not_a_number():
    """Refused by the slope operator with the bed as it was; the cell carries no
    transport, so the budget residual is a number."""
    from braids_hkt_gb300.solver import RiverSolver
    case = S.cartesian_channel()
    case["exner"] = S.exner_params(case)
    q = S.perturbed_state(case, 3, 0.1, 1.0)
    q[2, case["mesh"].nc // 2] = np.nan
    s = RiverSolver(case)
    s.set_state(q)
    row = s.morphology(1.0)
    assert not row["ok"] and row["slope_failure"] and np.isfinite(row["residual"])
    np.testing.assert_array_equal(s.z.cpu().numpy(), case["z"])


def test_bed_update_beside_an_infinite_depth():
    """A cell of infinite depth has no speed and no transport: the update of still
    water is accepted and moves nothing; one of infinite stress is refused."""
    from braids_hkt_gb300.solver import RiverSolver
    case = S.cartesian_channel()
    case["exner"] = S.exner_params(case)
    q = case["q"].copy()
    q[0, case["mesh"].nc // 2] = np.inf
    s = RiverSolver(case)
    s.set_state(q)
    row = s.morphology(1.0)
    assert row["ok"] and not row["slope_failure"] and row["residual"] == 0.0 and row["change"] == 0.0
    np.testing.assert_array_equal(s.z.cpu().numpy(), case["z"])
    q = case["q"].copy()
    q[1, case["mesh"].nc // 2] = 1e200
    s.set_state(q)
    row = s.morphology(1.0)
    assert not row["ok"] and row["slope_failure"]
    np.testing.assert_array_equal(s.z.cpu().numpy(), case["z"])
