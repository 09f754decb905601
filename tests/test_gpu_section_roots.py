"""Section outlets whose equation has several roots: the GPU has to end on the
root that bisection ends on, as the oracle does.

The critical outlet (mode 4) on openings with a bench, a V, bars and steps: a
face's controlled discharge rises before it falls, and the critical discharge
drops whenever another face wets. The free weir (mode 5) beside a bank that
is hardly wetter than the dry depth: the bank's discharge sets in at a jump,
and the weir's coefficient is put between the discharges on the jump's two
sides. Both roots pass the closing test of the residual, so only the fluxes
tell them apart. FP64 residual against the oracle to 1e-12 (the sections'
operations are the oracle's; powers of the inlet differ in the last place),
one HLLC step to the same, and the mixed form's water to one FP32 rounding of
each face's flux (2^-23).
"""
import itertools

import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu

SHAPES = {"bench": lambda y, p: np.where(y < 15.0, 0.0, p), "vee": lambda y, p: p * np.abs(y - 45.0) / 45.0,
          "bars": lambda y, p: p * (np.floor(y / 9.0) % 2), "steps": lambda y, p: p * np.floor(y / 18.0) / 4.0}
# rise of the bed, surface above the rise, speeds over the low and the high part
STATES = [(0.961, 0.317, (0.85, 0.31))] + list(
    itertools.product((0.5, 0.96, 1.6), (0.1, 0.32, 0.9), ((0.85, 0.31), (1.8, 0.5), (0.2, 0.2))))


def reach(bed, surface, speed, mode, dry=None):
    """Five cells long, a bed and a speed per row of 3 m; open at both ends."""
    case = S.cartesian_channel(length=15.0, width=3.0 * len(bed), spacing=3.0)
    row = np.minimum(case["mesh"].xy[1] // 3.0, len(bed) - 1).astype(int)
    z = np.ascontiguousarray(np.asarray(bed, float)[row])
    h = np.maximum(surface - z, 0.0)
    q = np.ascontiguousarray(np.stack((h, h * np.asarray(speed, float)[row], np.zeros_like(h))))
    controls = dict(case["controls"], **({} if dry is None else {"dry": dry}))
    return dict(case, z=z, q=q, exterior_bed=S._exterior_bed(case["mesh"], z), controls=controls,
                seg_mode=np.array([6, mode], np.int32))


def critical(shape):
    y = 3.0 * np.arange(30) + 1.5
    bed = lambda p: SHAPES[shape](y, p)
    return [reach(bed(p), p + s, np.where(bed(p) < 0.5 * p, *u), 4) for p, s, u in STATES]


def lax(h, hi, u, g=9.81):
    return u - (h - hi) * np.sqrt(0.5 * g * (1 / h + 1 / hi)) if h > hi else u + 2 * (np.sqrt(g * hi) - np.sqrt(g * h))


def weirs():
    """A channel of ten rows and a bank of ten, the bank wet by 1.05 to 1.6 dry depths of 1 mm."""
    rng = np.random.default_rng(1)
    out = []
    for _ in range(40):
        depth, ratio, froude = rng.uniform(0.5, 2.0), rng.uniform(1.05, 1.6), rng.uniform(0.1, 0.4)
        u, slow, crest, share = froude * np.sqrt(9.81 * depth), 0.02 * rng.uniform(), rng.uniform(0.1, 0.5) * depth, \
            rng.uniform(0.2, 0.8)
        bank = depth - ratio * 1e-3
        jump = bank + 1e-3                              # the stage at which the bank's discharge sets in
        low = 30.0 * jump * lax(jump, depth, u)
        gain = 30.0 * 1e-3 * lax(1e-3, ratio * 1e-3, slow)
        case = reach([bank] * 10 + [0.0] * 10, depth, [slow] * 10 + [u] * 10, 5, 1e-3)
        case["outlet"] = {1: {"crest_m": crest, "coefficient_m_half_s": (low + share * gain) / (jump - crest) ** 1.5 / 60.0,
                              "effective_width_m": 60.0}}
        out.append(case)
    return out


def outlet(case):
    m = case["mesh"]
    return np.asarray(m.boundary_faces)[m.boundary_offset[1]:m.boundary_offset[2]]


def check_residuals(cases, precision):
    from braids_hkt_gb300.solver import RiverSolver
    s = RiverSolver(cases, precision=precision)
    rate, water, status, _ = s.rate(0.01)
    rate, water = rate.cpu().numpy(), water.cpu().numpy()
    accepted = 0
    for i, case in enumerate(cases):
        st, rate_o, water_o, _ = Oracle(case).rate(case["q"].copy(), 0.01, 0.0)
        assert (int(status[i]) == 0) == (st == 0)
        if st:
            continue
        accepted += 1
        c, f = (slice(s.packed[k][i], s.packed[k][i + 1]) for k in ("cell_offset", "face_offset"))
        if precision == "mixed":
            k = outlet(case)
            assert np.all(np.abs(water[f][k] - water_o[k]) <= 2.0 ** -23 * np.abs(water_o[k]) + 1e-12), i
        else:
            for a, b in ((rate[:, c], rate_o), (water[f], water_o)):
                assert np.max(np.abs(a - b) / np.maximum(1.0, np.abs(b))) < 1e-12, i
    assert accepted > len(cases) // 2


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", SHAPES)
def test_critical_outlet_on_an_uneven_bed(shape, precision):
    check_residuals(critical(shape), precision)


@pytest.mark.parametrize("shape", SHAPES)
def test_critical_outlet_on_an_uneven_bed_hllc(shape):
    from braids_hkt_gb300.solver import RiverSolver
    cases = critical(shape)
    s = RiverSolver(cases, method="hllc")
    status, _ = s.substep(0.01)
    for i, case in enumerate(cases):
        st, out, _, _, _ = Oracle(case).hllc_step(case["q"], 0.01)
        assert (int(status[i]) == 0) == (st == 0)
        if st == 0:
            assert np.max(np.abs(s.state(i) - out) / np.maximum(1.0, np.abs(out))) < 1e-12, i


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_weir_beside_a_hardly_wet_bank(precision):
    check_residuals(weirs(), precision)
