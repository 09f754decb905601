"""Compensated sums over many blocks: scenarios around the 2,048 cells of a
block (one short, equal, one over), of one cell row and of several blocks,
batched and alone, against math.fsum. The Neumaier error of n terms is below
eps + n^2 eps^2 times their absolute sum, each term has a few roundings, and the
energies' potential parts (beds below datum) cancel little: their absolute sums
are below four times the sums: 6 roundings x 4 eps is 5e-15, so 1e-14 relative
covers all."""
import math

import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


def channel(nx, ny):
    c = S.cartesian_channel(length=3.0 * nx, width=3.0 * ny, spacing=3.0)
    assert c["mesh"].nc == nx * ny
    return c


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sizes", [[(89, 23)], [(64, 32)], [(683, 3)], [(7, 3), (256, 40), (5, 3), (32, 64)]],
                         ids=["2047", "2048", "2049", "batch"])
def test_sums_over_blocks(sizes, precision):
    from braids_hkt_gb300.solver import RiverSolver
    cases = [channel(*n) for n in sizes]
    s = RiverSolver(cases, precision=precision)
    off = s.packed["cell_offset"]
    rng = np.random.default_rng(5)
    start = np.concatenate([S.perturbed_state(c, 3, dry_fraction=.1) for c in cases], axis=1)
    now = start.copy()
    now[0] *= rng.uniform(.5, 1.5, now.shape[1])
    s.set_state(now)
    q0 = s.torch.from_numpy(start).to(s.q.device)
    s.torch.cuda.synchronize()
    for _ in range(2):                      # the second call finds the tickets as the first left them
        budget = np.stack(s._budget(q0), axis=1)
        totals = np.atleast_2d(s.totals())
        for i, c in enumerate(cases):
            a, b = off[i], off[i + 1]
            area, z = c["mesh"].area, np.asarray(c["z"])
            h0, (h, hu, hv) = start[0, a:b], now[:, a:b]
            g, dry = c["controls"]["grav"], c["controls"]["dry"]
            wet = h > dry
            energy = .5 * g * h * h + g * h * z + np.where(wet, .5 * (hu * hu + hv * hv) / np.where(wet, h, 1.), 0.)
            got = [*budget[i], *totals[i]]
            for v, terms in zip(got, (h0 * area, h * area, np.maximum(h0, h) * area, h * area, energy * area)):
                ref = math.fsum(terms.tolist())
                assert abs(v - ref) <= 1e-14 * ref
