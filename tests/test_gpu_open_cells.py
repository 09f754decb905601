"""Open faces that share an owner, and outlets that would take more than their
owner holds, in the boundary kernel with a thread per face: channels one cell
long, so that each cell owns an inlet and an outlet face, from one face a side
to several blocks of a cluster, and a draining stage outlet. FP64 residuals
against the oracle to 1e-12 (the inlet's powers and roots differ in the last
place), the batch against each channel alone bit for bit."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu


def one_cell_long(width):
    case = S.cartesian_channel(length=3.0, width=3.0 * width, spacing=3.0, discharge=2.0 * width)
    q = S.perturbed_state(case, 9, 0.05, 0.2)
    q[1] += 2.0
    return dict(case, q=q)


def draining(width):
    """Shallow water running off over a low stage outlet."""
    case = S.cartesian_channel(length=15.0, width=3.0 * width, spacing=3.0, discharge=0.5 * width)
    rng = np.random.default_rng(width)
    h = rng.uniform(0.01, 0.3, case["mesh"].nc)
    case["forcing"] = np.array([[0.5 * width, 0.0], [0.0, -3.0]])
    return dict(case, q=np.ascontiguousarray(np.stack((h, h * rng.uniform(0.0, 2.0, h.size), 0.1 * h))))


def agree(case, dt, capped):
    from braids_hkt_gb300.solver import RiverSolver
    rate, water, status, freq = RiverSolver(case).rate(dt)
    st, rate_o, water_o, freq_o = Oracle(case).rate(case["q"].copy(), dt, 0.0)
    assert (int(status) == 0) == (st == 0)
    for a, b in ((rate, rate_o), (water, water_o)):
        assert np.max(np.abs(a.cpu().numpy() - b) / np.maximum(1.0, np.abs(b))) < 1e-12
    assert abs(freq - freq_o) <= 1e-12 * freq_o
    # the step length matters where an outlet is capped, and there alone
    m = case["mesh"]
    outlet = m.boundary_faces[m.boundary_offset[1]:]
    free = Oracle(case).rate(case["q"].copy(), 1e-9, 0.0)[2]
    assert (np.abs(water_o[outlet]) < 0.999 * np.abs(free[outlet])).any() == capped


@pytest.mark.parametrize("width", [1, 2, 31, 65, 300])
@pytest.mark.parametrize("dt,capped", [(0.01, False), (30.0, True)])
def test_cells_with_an_inlet_and_an_outlet_face(width, dt, capped):
    agree(one_cell_long(width), dt, capped)


@pytest.mark.parametrize("width", [1, 65, 300])
@pytest.mark.parametrize("dt,capped", [(0.01, False), (10.0, True)])
def test_outlets_capped_at_their_owners_stock(width, dt, capped):
    agree(draining(width), dt, capped)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_equals_each_alone(precision):
    from braids_hkt_gb300.solver import RiverSolver
    cases = [one_cell_long(1), draining(65), one_cell_long(300), one_cell_long(65), draining(2)]
    batch = RiverSolver(cases, precision=precision)
    for k in range(2):
        batch.advance(0.5, 0.5 * k)
    for i, case in enumerate(cases):
        alone = RiverSolver(case, precision=precision)
        for k in range(2):
            alone.advance(0.5, 0.5 * k)
        np.testing.assert_array_equal(batch.state(i), alone.state())
        assert batch.ledger()[i] == alone.ledger()[0]
