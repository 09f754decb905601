"""Cells of more than four faces: squares of the Cartesian channel merged into
bricks of two (six faces), a block of sixteen (sixteen faces) and the largest
accepted, a strip of 32 faces, beside squares that stay.

FP64: one residual of the closed domain equals the oracle's bit for bit, with
step lengths that drain no cell and many, and so does the allocation-free
residual's; intervals of the open channel follow the oracle to 1e-10 with its
substeps, f-wave and HLLC, as on narrower cells. Mixed: depths within 1e-4 of
FP64's, the mass of draining cells to FP64 rounding, and batched as alone."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import braids_hkt_gb300.mesh as M
import braids_hkt_gb300.scenarios as S
from oracle import Oracle

pytestmark = pytest.mark.gpu


def merged(mesh, group):
    """The mesh of the unions of cells of one group; faces inside a union go."""
    _, group = np.unique(group, return_inverse=True)
    nc = group.max() + 1
    owner = group[mesh.owner]
    neighbour = np.where(mesh.neighbour >= 0, group[mesh.neighbour], -1)
    keep = np.flatnonzero(owner != neighbour)
    number = np.full(mesh.nf, -1)
    number[keep] = np.arange(len(keep))
    area = np.bincount(group, mesh.area, nc)
    xy = np.stack([np.bincount(group, mesh.area * mesh.xy[k], nc) / area for k in range(2)])
    cell_of = np.repeat(group, np.diff(mesh.offset))
    entries = [np.flatnonzero((cell_of == c) & (number[mesh.faces] >= 0)) for c in range(nc)]
    order = np.concatenate(entries)
    i32 = lambda a: np.ascontiguousarray(a, dtype=np.int32)
    out = dataclasses.replace(
        mesh, owner=i32(owner[keep]), neighbour=i32(neighbour[keep]), bid=i32(mesh.bid[keep]),
        normal=np.ascontiguousarray(mesh.normal[:, keep]), length=mesh.length[keep].copy(),
        mid=np.ascontiguousarray(mesh.mid[:, keep]), area=area, xy=np.ascontiguousarray(xy),
        offset=i32(np.concatenate([[0], np.cumsum([len(e) for e in entries])])), faces=i32(number[mesh.faces[order]]),
        signs=i32(mesh.signs[order]), boundary_faces=i32(number[mesh.boundary_faces]), records={})
    M.geometry_records(out)
    return out, group


def bricks():
    """Open channel of 40 x 8 squares: most in bricks, a 4 x 4 block, a strip of 15 (32 faces), squares between."""
    case = S.cartesian_channel()
    mesh = case["mesh"]
    i, j = (np.floor(mesh.xy[k] / 3.0).astype(int) for k in range(2))
    assert i.max() == 39 and j.max() == 7
    group = 1000 + 100 * ((i + j % 2) // 2) + j
    group = np.where(i >= 33, 100_000 + 100 * i + j, group)                 # squares at the outlet
    group = np.where((i >= 8) & (i < 12) & (j >= 2) & (j < 6), 1, group)
    group = np.where((i >= 14) & (i < 29) & (j == 3), 2, group)
    out, group = merged(mesh, group)
    weights = np.bincount(group)
    mean = lambda v: np.ascontiguousarray(np.bincount(group, v) / weights)
    z = mean(case["z"])
    q = np.stack([mean(v) for v in case["q"]])
    degree = np.diff(out.offset)
    assert degree.max() == 32 and (degree == 16).any() and (degree == 6).any() and (degree == 4).any()
    return dict(case, mesh=out, z=z, q=np.ascontiguousarray(q), exterior_bed=S._exterior_bed(out, z))


def closed(case):
    m = case["mesh"]
    m.bid[:] = -1
    m.boundary_offset = np.zeros(1, np.int32)
    m.boundary_faces = np.zeros(0, np.int32)
    return dict(case, seg_mode=np.zeros(0, np.int32), stage_policy=np.zeros(0, np.int32), forcing=np.zeros((2, 1)),
                exterior_bed=np.zeros(m.nf))


@pytest.mark.parametrize("dt", [1e-3, 3.0])
@pytest.mark.parametrize("amplitude,speed,dry", [(0.0, 0.0, 0.0), (0.3, 0.6, 0.0), (0.5, 1.5, 0.3)])
def test_fp64_residual(amplitude, speed, dry, dt):
    import torch

    import braids_hkt_gb300._lib as L
    from braids_hkt_gb300.solver import RiverSolver
    case = closed(bricks())
    case["q"] = S.perturbed_state(case, 8, amplitude, speed, dry)
    rate, water, status, freq = RiverSolver(case).rate(dt)
    st, rate_o, water_o, freq_o = Oracle(case).rate(case["q"].copy(), dt, 0.0)
    np.testing.assert_array_equal(rate.cpu().numpy(), rate_o)
    np.testing.assert_array_equal(water.cpu().numpy(), water_o)
    assert freq == freq_o and (int(status) == 0) == (st == 0)
    lib, m, r, ctl = L.load(), case["mesh"], case["mesh"].records, case["controls"]
    dev = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (
        m.owner, m.neighbour, m.offset, m.faces, m.signs, m.normal, m.length, m.area, r["ls_matrix"], r["ls_weight"],
        r["ls_delta"], r["disp"], r["disp_len"], r["distance"], case["q"], case["z"])]
    p = lambda t: C.c_void_p(t.data_ptr())
    rate2, water2, st2, fr2 = torch.empty_like(rate), torch.empty_like(water), C.c_uint(), C.c_double()
    assert lib.brx_rate_noalloc(m.nc, m.nf, m.nadj, *(p(t) for t in dev), ctl["grav"], ctl["dry"], ctl["cfl"], dt,
                                p(rate2), p(water2), C.byref(st2), C.byref(fr2), None) == 0
    np.testing.assert_array_equal(rate2.cpu().numpy(), rate_o)
    np.testing.assert_array_equal(water2.cpu().numpy(), water_o)


@pytest.mark.parametrize("method", ["fwave", "hllc"])
def test_intervals(method):
    from braids_hkt_gb300.solver import RiverSolver
    case = bricks()
    a, b = (RiverSolver(case, precision=p, method=method) for p in ("fp64", "mixed"))
    batch = RiverSolver([S.small_channel(), case], precision="mixed", method=method)
    o = Oracle(case, threads=4)
    q = case["q"].copy()
    for k in range(3):
        da, db, dc = (s.advance(1.0, float(k)) for s in (a, b, batch))
        st, _, stats = (o.advance if method == "fwave" else o.hllc_advance)(q, 1.0, float(k))
        assert st == 0 and da["failed"] == 0 and db == dc[1]
        assert da["hydraulic_substeps"] == stats["substeps"]
    scale = np.maximum(np.abs(q).max(axis=1, keepdims=True), 1e-3)
    assert (np.abs(a.state() - q) / scale).max() <= 1e-10
    ha, hb = a.state()[0], b.state()[0]
    assert (np.abs(hb - ha) / np.maximum(ha, 1e-3)).max() <= 1e-4
    np.testing.assert_array_equal(batch.state(1), b.state())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_draining_cells_keep_the_water(precision):
    """A residual whose step drains cells: the limited rates sum to nothing over
    the closed domain (a face's flux enters two sums of at most 32, 64 roundings
    of it in all) and no cell goes below zero by more than the limiter's roundings."""
    from braids_hkt_gb300.solver import RiverSolver
    case = closed(bricks())
    case["q"] = S.perturbed_state(case, 8, 0.5, 1.5, 0.3)
    m, dt = case["mesh"], 3.0
    rate, water = (t.cpu().numpy() for t in RiverSolver(case, precision=precision).rate(dt)[:2])
    assert abs((rate[0] * m.area).sum()) <= 64 * np.finfo(float).eps * 2 * (np.abs(water) * m.length).sum()
    depth = case["q"][0] + dt * rate[0]
    assert depth.min() >= -1e-12 and (depth < 1e-3 * case["q"][0].max()).any()
