"""The FP64 face sweep and donor limiter against the oracle on every wave pattern.

Faces between two wet states take the written-out solve, faces with a dry
state the general one. On a closed domain the residual of either uses the
oracle's own operations, so it equals the oracle's bit for bit: still water,
equal depths, double rarefactions, double shocks, mixed waves, supercritical
streams in both directions, films about the dry depth, dry patches.
"""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu

# depth range [m], speed range [m/s], one velocity for all cells, bed relief scale, share of dry cells
STATES = {
    "still": ((1.0, 1.0), 0.0, None, 0.0, 0.0),
    "stream": ((1.5, 1.5), 0.0, (7.0, 0.5), 0.0, 0.0),
    "subcritical": ((0.8, 1.2), 0.8, None, 0.2, 0.0),
    "crossing": ((0.3, 3.0), 3.0, None, 0.5, 0.0),
    "supercritical": ((0.2, 0.4), 0.5, (-6.0, 4.0), 0.1, 0.0),
    "films": ((0.9e-6, 4e-6), 1e-3, None, 1e-6, 0.0),
    "patches": ((0.05, 1.0), 2.0, None, 1.0, 0.4),
}


@pytest.mark.parametrize("name", sorted(STATES))
@pytest.mark.parametrize("mesh", ["triangles", "squares"])
@pytest.mark.parametrize("dt", [1e-4, 3.0])      # 3 s empties many cells: their donors' limited fluxes
def test_residual_equals_the_oracle_bit_for_bit(mesh, name, dt):
    from braids_hkt_gb300.solver import RiverSolver
    case = S.dam_break() if mesh == "triangles" else S.cartesian_channel(length=99.0, width=27.0, spacing=3.0)
    m = case["mesh"]
    m.bid[:] = -1
    m.boundary_offset = np.zeros(1, np.int32)
    m.boundary_faces = np.zeros(0, np.int32)
    depth, speed, stream, relief, dry = STATES[name]
    rng = np.random.default_rng(5)
    z = relief * rng.uniform(-1, 1, m.nc)
    h = rng.uniform(*depth, m.nc)
    h[rng.random(m.nc) < dry] = 0.0
    u, v = speed * rng.uniform(-1, 1, (2, m.nc)) + np.reshape(stream or (0.0, 0.0), (2, 1))
    case = dict(case, z=z, q=np.ascontiguousarray(np.stack((h, h * u, h * v))), seg_mode=np.zeros(0, np.int32),
                stage_policy=np.zeros(0, np.int32), forcing=np.zeros((2, 1)), exterior_bed=np.zeros(m.nf))
    solver = RiverSolver(case)
    rate, water, status, freq = solver.rate(dt)
    st, rate_o, water_o, freq_o = Oracle(case).rate(case["q"].copy(), dt, 0.0)
    np.testing.assert_array_equal(rate.cpu().numpy(), rate_o)
    np.testing.assert_array_equal(water.cpu().numpy(), water_o)
    assert freq == freq_o
