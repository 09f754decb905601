"""The FP64 sweeps of cells with at most four faces against the general ones.

brx_rate_noalloc runs the general cell sweep (up to 32 faces per cell, no
tables); brx_rate runs the sweep with tables and the pruned projection. On
closed domains both evaluate the same FP64 operations, so the residuals are
equal bit for bit: wet and dry states, waves from round-off to bores, states
at rest, triangles and squares, meshes from one block of cells to several,
with a remainder.
"""
import ctypes as C

import numpy as np
import pytest

import braids_hkt_gb300.scenarios as S

pytestmark = pytest.mark.gpu


def closed(case):
    m = case["mesh"]
    m.bid[:] = -1
    m.boundary_offset = np.zeros(1, np.int32)
    m.boundary_faces = np.zeros(0, np.int32)
    return dict(case, mesh=m, seg_mode=np.zeros(0, np.int32), stage_policy=np.zeros(0, np.int32),
                forcing=np.zeros((2, 1)), exterior_bed=np.zeros(m.nf))


CASES = {
    "islands": lambda: S.lake_at_rest(seed=17),
    "channel": lambda: closed(S.channel(300.0, 60.0, 3.1, 0.8, seed=5)),
    "squares": lambda: closed(S.cartesian_channel(length=120.0, width=39.0, spacing=3.0)),
    "strip": lambda: closed(S.cartesian_channel(length=99.0, width=3.0, spacing=3.0)),
}
# wave amplitude [m], current [m/s], share of dry cells
STATES = [(0.0, 0.0, 0.0), (1e-13, 1e-13, 0.0), (1e-3, 1e-2, 0.0), (0.3, 0.6, 0.0), (0.5, 0.6, 0.3), (2.5, 4.0, 0.1)]


@pytest.mark.parametrize("name", sorted(CASES))
def test_residual_equals_the_general_sweep_bit_for_bit(name):
    import torch
    import braids_hkt_gb300._lib as L
    from braids_hkt_gb300.solver import RiverSolver
    lib = L.load()
    case = CASES[name]()
    m, r, ctl = case["mesh"], case["mesh"].records, case["controls"]
    assert m.nc <= 16384
    solver = RiverSolver(case)
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in dict(
        owner=m.owner, neighbour=m.neighbour, offset=m.offset, faces=m.faces, signs=m.signs, normal=m.normal,
        length=m.length, area=m.area, ls_matrix=r["ls_matrix"], ls_weight=r["ls_weight"], ls_delta=r["ls_delta"],
        disp=r["disp"], disp_len=r["disp_len"], distance=r["distance"], z=np.asarray(case["z"], float)).items()}
    p = lambda t: C.c_void_p(t.data_ptr())
    for seed, (amplitude, velocity, dry) in enumerate(STATES):
        q = S.perturbed_state(case, 40 + seed, amplitude, velocity, dry)
        solver.set_state(q)
        rate, water, status, freq = solver.rate(0.01)
        qd = torch.from_numpy(q).cuda()
        rate2, water2 = torch.empty_like(rate), torch.empty_like(water)
        st, fr = C.c_uint(), C.c_double()
        assert lib.brx_rate_noalloc(
            m.nc, m.nf, m.nadj, p(dev["owner"]), p(dev["neighbour"]), p(dev["offset"]), p(dev["faces"]),
            p(dev["signs"]), p(dev["normal"]), p(dev["length"]), p(dev["area"]), p(dev["ls_matrix"]),
            p(dev["ls_weight"]), p(dev["ls_delta"]), p(dev["disp"]), p(dev["disp_len"]), p(dev["distance"]), p(qd),
            p(dev["z"]), ctl["grav"], ctl["dry"], ctl["cfl"], 0.01, p(rate2), p(water2), C.byref(st), C.byref(fr),
            None) == 0, lib.brx_last_error()
        assert (status, freq) == (st.value, fr.value)
        np.testing.assert_array_equal(rate.cpu().numpy(), rate2.cpu().numpy())
        np.testing.assert_array_equal(water.cpu().numpy(), water2.cpu().numpy())


@pytest.mark.parametrize("momentum", [1e140, 1e160, 1e200, 1e300])
def test_drag_of_a_momentum_whose_square_overflows(momentum):
    """A wet cell's momentum whose square is infinite: the drag's factor is zero
    and the trial accepted, as in the oracle; one below that is refused by both.
    The same steps of FP64 arithmetic: 1e-12 of each row's largest value."""
    from braids_hkt_gb300.solver import RiverSolver
    from oracle import Oracle
    case = S.small_channel()
    q = case["q"].copy()
    q[1, case["mesh"].nc // 2] = momentum
    s = RiverSolver(case, precision="fp64")
    s.set_state(q)
    status, _ = s.substep(0.004, 0.0)
    code, _, _ = Oracle(case, threads=4).advance(q, 0.004, 0.0)
    assert (status == 0) == (code == 0) == (momentum > 1e154)
    if code == 0:
        scale = np.abs(q).max(axis=1, keepdims=True)
        assert (np.abs(s.state() - q) / scale).max() <= 1e-12


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("row", [0, 1])
def test_hllc_ends_a_nonfinite_state_at_its_first_trial(row, value):
    """A nonfinite state gives an infinite CFL peak: the trial is rejected with a
    zero hint and the interval fails, not after halving down to the floor."""
    from braids_hkt_gb300.solver import RiverSolver
    if row == 0 and value == -np.inf:
        pytest.skip("a negative depth is refused by its own status")
    case = S.small_channel()
    q = case["q"].copy()
    q[row, case["mesh"].nc // 2] = value
    s = RiverSolver(case, precision="fp64", method="hllc")
    s.set_state(q)
    d = s.advance(0.05, 0.0, raise_on_failure=False)
    assert (d["failed"], d["hydraulic_substeps"], d["hydraulic_rejections"]) == (1, 0, 1)
