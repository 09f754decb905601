"""Openings wider than a cluster of blocks (above 1,024 faces a scenario): the one
block that takes them against the oracle. FP64 to 1e-12; in the mixed form a
conveyance weight is a product of two FP32 powers (a few units in the last
place each, 2^-20 together), normalised by their sum, and a face's water is
rounded to FP32: 2^-18 relative. A batch with a narrow opening equals each alone."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu


def opening(faces):
    case = S.cartesian_channel(length=15.0, width=3.0 * faces, spacing=3.0, discharge=2.0 * faces)
    q = S.perturbed_state(case, 9, 0.05, 0.2)
    q[1] += 2.0 / 3.0
    return dict(case, q=q)


@pytest.mark.parametrize("faces", [513, 1025, 1600, 4001])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fluxes(faces, precision):
    from braids_hkt_gb300.solver import RiverSolver
    case = opening(faces)
    _, water, status, _ = RiverSolver(case, precision=precision).rate(0.01)
    st, _, water_o, _ = Oracle(case, threads=4).rate(case["q"].copy(), 0.01, 0.0)
    assert int(status) == st == 0
    k = case["mesh"].boundary_faces
    a, b = water.cpu().numpy()[k], water_o[k]
    if precision == "fp64":
        assert np.max(np.abs(a - b) / np.maximum(1.0, np.abs(b))) < 1e-12
    else:
        assert np.max(np.abs(a - b) / np.maximum(1.0, np.abs(b))) < 2.0 ** -18


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_wide_and_narrow_batch(precision):
    from braids_hkt_gb300.solver import RiverSolver
    cases = [opening(3), opening(1100)]
    batch = RiverSolver(cases, precision=precision)
    batch.advance(0.05, 0.0)
    for i, case in enumerate(cases[1:], 1):
        alone = RiverSolver(case, precision=precision)
        alone.advance(0.05, 0.0)
        np.testing.assert_array_equal(batch.state(i), alone.state())
        assert batch.ledger()[i] == alone.ledger()[0]
