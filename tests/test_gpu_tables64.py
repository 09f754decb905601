"""The FP64 form's mesh tables belong to the method that reads them: an HLLC
solver holds none of the f-wave's (some 300 bytes a triangle), and a solver
whose method or boundary modes change forms them anew."""
import ctypes as C

import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


def test_hllc_solver_holds_no_fwave_tables():
    from braids_hkt_gb300.solver import RiverSolver
    case = S.channel(length=400.0, width=80.0)
    f, h = RiverSolver(case), RiverSolver(case, method="hllc")
    stencil = f.packed["nadj"] * (8 + 32 + 16) + 3 * 8 * f.nc       # entries, offsets, squares; inverse
    f.advance(0.1, 0.0)
    h.advance(0.1, 0.0)
    assert f.device_bytes() - (h.device_bytes() - stencil) >= 300 * f.nc


@pytest.mark.parametrize("make", [S.small_channel, S.cartesian_channel])
def test_tables_follow_the_method_and_the_modes(make):
    from braids_hkt_gb300.solver import METHODS, RiverSolver
    case = make()
    case["q"] = S.perturbed_state(case, 3, 0.05, 0.4)
    other = dict(case, seg_mode=np.array([6, 3], np.int32))
    s = RiverSolver(case, method="hllc")
    pointer = lambda a: a.ctypes.data_as(C.c_void_p)

    def same_residual(reference):
        a, b = s.rate(0.01), RiverSolver(reference).rate(0.01)
        assert int(a[2]) == int(b[2]) and a[3] == b[3]
        for x, y in zip(a[:2], b[:2]):
            np.testing.assert_array_equal(x.cpu().numpy(), y.cpu().numpy())

    assert s.lib.brx_method_set(s.h, METHODS["fwave"]) == 0
    same_residual(case)
    p = s.packed
    for c in (other, case):
        modes = np.ascontiguousarray(c["seg_mode"])
        assert s.lib.brx_boundary_set(s.h, pointer(modes), pointer(p["stage_policy"]), pointer(p["exterior_bed"]),
                                      pointer(p["forcing"])) == 0
        same_residual(c)
    assert s.lib.brx_method_set(s.h, METHODS["hllc"]) == 0
    s.advance(0.1, 0.0)
    fresh = RiverSolver(case, method="hllc")
    fresh.advance(0.1, 0.0)
    np.testing.assert_array_equal(s.state(), fresh.state())
