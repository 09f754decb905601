"""Mixed form, cells redone with limited fluxes: a wet/dry lake of triangles whose
shore cells drain, alone and in a batch with squares or with cells of up to 32
faces. The three take other instances of the redo (a thread per entry, or four
per cell that take the entries in turn) and give the same bits; the water of the
closed lake stays, to 64 eps of what it holds a substep."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from test_gpu_wide_cells import bricks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other", [S.cartesian_channel, bricks])
@pytest.mark.parametrize("length", [80.0, 300.0])
def test_draining_shores(length, other):
    from braids_hkt_gb300.solver import RiverSolver
    case = S.lake_at_rest(length=length, width=0.5 * length, spacing=length / 40)
    case["q"] = S.perturbed_state(case, 3, 0.2, 0.5, 0.1)
    alone, both = RiverSolver(case, precision="mixed"), RiverSolver([other(), case], precision="mixed")
    volume, substeps = alone.totals()[0], 0
    for k in range(4):
        a, b = alone.advance(0.2, 0.2 * k), both.advance(0.2, 0.2 * k)
        assert a == b[1]
        np.testing.assert_array_equal(both.state(1), alone.state())
        substeps += a["hydraulic_substeps"]
    assert abs(alone.totals()[0] - volume) <= 64 * np.finfo(float).eps * substeps * volume
