"""Mixed cell sweep by the most faces of a cell (triangles, quadrilaterals,
any): a triangle mesh in a batch with a quadrilateral one takes the wider form,
alone the narrow one, and has to give the same bits, as batches do. Meshes of
one block, around a block's 128 cells and of many, with steep and dry cells so
that the limiter works on every side. The limited gradients are continuous in
the state, so one trial stays within 1e-4 of the FP64 form's scale, the stated
accuracy of the mixed form."""
import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [12.0, 36.0, 40.0, 120.0, 600.0])
@pytest.mark.parametrize("dry", [0.0, 0.3])
def test_triangles_alone_and_with_quads(length, dry):
    from braids_hkt_gb300.solver import RiverSolver
    tri = S.small_channel(length=length, width=24.0, spacing=4.0)
    quad = S.cartesian_channel(length=36.0, width=24.0, spacing=3.0)
    tri["q"] = S.perturbed_state(tri, 3, amplitude=.5, dry_fraction=dry)
    quad["q"] = S.perturbed_state(quad, 5, amplitude=.5, dry_fraction=dry)
    alone, both = RiverSolver(tri, precision="mixed"), RiverSolver([quad, tri], precision="mixed")
    ref = RiverSolver(tri, precision="fp64")
    dt = 0.02
    sa, pa = alone.substep(dt, 0.0)
    sb, pb = both.substep(dt, 0.0)
    s64, _ = ref.substep(dt, 0.0)
    assert sa == sb[1] == s64 and pa == pb[1]
    q, q64 = alone.state(), ref.state()
    np.testing.assert_array_equal(both.state(1), q)
    scale = np.maximum(np.abs(q64).max(axis=1, keepdims=True), 1e-3)
    assert (np.abs(q - q64) / scale).max() <= 1e-4


def test_dam_break_alone_and_with_quads():
    """The same over adaptive intervals with draining cells, whose limited fluxes are redone."""
    from braids_hkt_gb300.solver import RiverSolver
    tri, quad = S.dam_break(), S.cartesian_channel(length=36.0, width=24.0, spacing=3.0)
    alone, both = RiverSolver(tri, precision="mixed"), RiverSolver([quad, tri], precision="mixed")
    for k in range(4):
        a, b = alone.advance(1.0, 1.0 * k), both.advance(1.0, 1.0 * k)
        assert a == b[1]
        np.testing.assert_array_equal(both.state(1), alone.state())


@pytest.mark.parametrize("froude", [0.01, 0.1, 0.5, 1.0, 3.0])
def test_wall_reflection_matches_fp64(froude):
    """Water thrown against every wall of a box: the FP32 shock at the wall (its
    depth ratio good to 1e-7) against FP64's, each momentum rate within the
    mixed form's 1e-4 of the largest."""
    from braids_hkt_gb300.solver import RiverSolver
    case = S.lake_at_rest(islands=False)
    m, h = case["mesh"], case["q"][0]
    away = m.xy - m.xy.mean(axis=1, keepdims=True)
    away = away / np.linalg.norm(away, axis=0)
    q = case["q"].copy()
    q[1:] = froude * h * np.sqrt(case["controls"]["grav"] * h) * away
    rates = []
    for precision in ("fp64", "mixed"):
        s = RiverSolver(case, precision=precision)
        s.set_state(q)
        r = s.rate(1e-3, 0.0)[0]
        rates.append(r.cpu().numpy() if hasattr(r, "cpu") else np.asarray(r))
    a, b = rates
    scale = np.abs(a[1:]).max()
    assert scale > 0 and np.abs(b[1:] - a[1:]).max() <= 1e-4 * scale


def test_method_switch_forms_its_bed_tables():
    """Each method forms its own bed tables: a solver switched between the methods
    with the bed changed in between gives the bits of one made for the method."""
    from braids_hkt_gb300.solver import METHODS, RiverSolver, check
    case = S.small_channel()
    q = S.perturbed_state(case, 3)
    s = RiverSolver(case, precision="mixed", method="hllc")
    for k, method in enumerate(["hllc", "fwave", "hllc", "fwave"]):
        check(s.lib.brx_method_set(s.h, METHODS[method]))
        alone = RiverSolver(case, precision="mixed", method=method)
        for t in (s, alone):
            t.set_state(q)
            t.z.copy_(t.torch.from_numpy(case["z"] * (1. + .1 * k)))
            t.substep(0.02, 0.0)
        np.testing.assert_array_equal(s.state(), alone.state())
