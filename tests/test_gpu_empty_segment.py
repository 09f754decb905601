"""Forcing tables are sampled for a segment without faces too, whichever
boundary kernel the batch takes (modes 2 and 6: a thread per face; a free
weir: section solves)."""
import copy

import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [S.small_channel, S.weir_channel])
def test_table_of_a_segment_without_faces(make):
    from braids_hkt_gb300.solver import RiverSolver
    case = make()
    mesh = copy.copy(case["mesh"])
    mesh.boundary_offset = np.append(mesh.boundary_offset, mesh.boundary_offset[-1]).astype(np.int32)
    case.update(mesh=mesh, seg_mode=np.append(case["seg_mode"], 2).astype(np.int32), stage_policy=np.zeros(3, np.int32),
                forcing=np.column_stack((case["forcing"], (0.0, 3.0))))
    s = RiverSolver(case)
    value = np.array([[[20.0, 24.0], [0.0, 0.0], [1.0, 2.0]], [[0.0, 0.0], [3.0, 3.0], [3.0, 3.5]]])
    s.set_forcing_table([0.0, 10.0], value)
    s.rate(0.01, 5.0)
    np.testing.assert_allclose(s.forcing(), value.mean(axis=2), rtol=1e-15)
