"""The boundary kernel over the widths of its work split.

Openings of one face, one tile of 64 and its neighbours, one block of 128 and
up to clusters of eight blocks (conveyance inlet, stage outlet), and the
section solves beside their 128 lanes (exact-discharge inlet, free weir,
critical outlet). One FP64 residual against the oracle, to the 1e-12 that
residuals with open boundaries hold (powers and roots differ in the last
place); the two openings of a batch equal each alone bit for bit.
"""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu


def opening(faces, modes):
    case = S.cartesian_channel(length=15.0, width=3.0 * faces, spacing=3.0, discharge=2.0 * faces)
    case["seg_mode"] = np.array(modes, np.int32)
    if modes[0] == 9:
        case["forcing"][1, 0] = 3.05
    if modes[1] == 5:
        case["outlet"] = {1: {"crest_m": 2.0, "coefficient_m_half_s": 1.7, "effective_width_m": 3.0 * faces}}
    q = S.perturbed_state(case, 9, 0.05, 0.2)
    q[1] += 2.0 / 3.0
    return dict(case, q=q)


@pytest.mark.parametrize("modes,faces", [((6, 2), n) for n in (1, 2, 63, 64, 65, 129, 300, 1030)] +
                         [((9, 5), n) for n in (1, 64, 127, 128, 129, 300)] + [((6, 4), n) for n in (1, 128, 129)])
def test_residual_matches_the_oracle(modes, faces):
    from braids_hkt_gb300.solver import RiverSolver
    case = opening(faces, modes)
    rate, water, status, freq = RiverSolver(case).rate(0.01)
    st, rate_o, water_o, freq_o = Oracle(case).rate(case["q"].copy(), 0.01, 0.0)
    assert int(status) == st == 0
    for a, b in ((rate, rate_o), (water, water_o)):
        assert np.max(np.abs(a.cpu().numpy() - b) / np.maximum(1.0, np.abs(b))) < 1e-12
    assert abs(freq - freq_o) <= 1e-12 * freq_o


def test_wide_and_narrow_openings_in_one_batch_equal_each_alone():
    from braids_hkt_gb300.solver import RiverSolver
    cases = [opening(n, (6, 2)) for n in (5, 700, 64)]
    batch = RiverSolver(cases)
    batch.advance(0.05, 0.0)
    for i, case in enumerate(cases):
        alone = RiverSolver(case)
        alone.advance(0.05, 0.0)
        np.testing.assert_array_equal(batch.state(i), alone.state())
        assert batch.ledger()[i] == alone.ledger()[0]
