"""Bed update of scenarios around the 1,024 cells of a block of the trial sweep
(one short, equal, one over) and of several blocks, against the oracle: the
trial bed to 1e-12 of the bed change, the reduced checks in their own terms.
The relative change is one quotient (1e-10, as elsewhere); the boundary volume
and residual are sums of products, n eps of their absolute sums, below 1e-12 of
the volume moved."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("size", [(93, 11), (64, 16), (205, 5), (128, 40), (6, 4)],
                         ids=["1023", "1024", "1025", "5120", "24"])
def test_bed_update_over_blocks(size, precision):
    from braids_hkt_gb300.solver import RiverSolver
    from oracle import Oracle
    nx, ny = size
    case = S.cartesian_channel(length=3.0 * nx, width=3.0 * ny, spacing=3.0, discharge=5.0 * 3.0 * ny)
    case["exner"] = S.exner_params(case, diameter=0.0005)
    m = case["mesh"]
    assert m.nc == nx * ny
    q = S.perturbed_state(case, 3, velocity=2.5, dry_fraction=.1)
    s = RiverSolver(case, precision=precision)
    s.set_state(q)
    st = s.morphology(5.0)
    code, zt, ref = Oracle(case, threads=4).exner(s.state(), 5.0)
    assert code == 0
    dz = np.abs(zt - case["z"]).max()
    moved = float(np.sum(np.abs(zt - case["z"]) * m.area))
    assert dz > 0 and st["ok"] == ref["ok"]
    if ref["ok"]:
        assert np.abs(s.z.cpu().numpy() - zt).max() <= 1e-12 * dz + 1e-15
    assert st["change"] == pytest.approx(ref["change"], rel=1e-10)
    assert st["donor"] == pytest.approx(ref["donor"], rel=1e-12)
    assert abs(st["boundary"] - ref["boundary"]) <= 1e-12 * max(moved, abs(ref["boundary"]))
    assert abs(st["residual"] - ref["residual"]) <= 1e-12 * moved
