"""Roughness at the ends of what brx_controls_set accepts: Chezy coefficients
whose square overflows (a frictionless bed), Manning coefficients whose
reciprocal does, or whose Chezy coefficient's square vanishes (a bed that
stops the water). One FP64 substep against the oracle to 1e-12, both methods."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["fwave", "hllc"])
@pytest.mark.parametrize("mode,value", [(1, 1e12), (1, 1e153), (1, 1e160), (1, 1e300), (1, 1e-160), (1, 1e-300), (2, 1e-200),
                                        (2, 1e-310), (2, 1e200), (2, 1e300)])
def test_drag_at_the_ends_of_its_range(mode, value, method):
    from braids_hkt_gb300.solver import RiverSolver
    case = S.lake_at_rest()
    case["controls"] = dict(case["controls"], roughness_mode=mode, roughness_value=value)
    q = S.perturbed_state(case, 5, 0.1, 0.5)
    s = RiverSolver(case, method=method)
    s.set_state(q)
    status, _ = s.substep(0.004)
    o = Oracle(case)
    st, out = (o.single(q, 0.004) if method == "fwave" else o.hllc_step(q, 0.004))[:2]
    assert int(status) == st == 0
    assert np.max(np.abs(s.state() - out) / np.maximum(1.0, np.abs(out))) < 1e-12
