"""More scenarios in one batch than a grid's second dimension holds (65,535):
the compensated sums and the bed update of each equal those of one alone, bit
for bit, in the first, the last and the scenarios about the limit."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


def test_sums_and_bed_update_of_a_large_batch():
    from braids_hkt_gb300.solver import RiverSolver
    case = S.cartesian_channel(length=9.0, width=6.0, spacing=3.0, sigma=0.05)
    case["q"] = S.perturbed_state(case, 4, 0.05, 2.0)
    case["exner"] = S.exner_params(case, diameter=0.0005)
    count = 65_537
    alone = RiverSolver(case)
    batch = RiverSolver([case] * count)
    totals = alone.totals()
    many = batch.totals()
    assert np.all(many == totals)
    start = alone.q.clone()
    budget = np.stack(alone._budget(start), axis=1)[0]
    assert np.all(np.stack(batch._budget(batch.q.clone()), axis=1) == budget)
    row = alone.morphology(20.0)
    rows = batch.morphology(20.0)
    bed, beds = alone.z.cpu().numpy(), batch.z.cpu().numpy().reshape(count, -1)
    for i in (0, 1, 65_534, 65_535, 65_536):
        assert rows[i] == row
        np.testing.assert_array_equal(beds[i], bed)
    assert np.all(beds == bed)
