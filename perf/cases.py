"""Performance cases of the river solver: what a program asks of RiverSolver.

Every case is one call (or the loop body) that a program makes again and
again through the public owner: a spatial residual, a substep, an adaptive
interval, the owner's budget-checked step, the step with its bed update. The
families cover both arithmetic forms, both hydraulic methods, triangles and
quadrilaterals, single scenarios and batches, rotor arrays, wet/dry braided
reaches and the section solvers of the open boundaries, from a few hundred
cells, where launches and latency count, to meshes far beyond the L2 cache.

Meshes are the package's own synthetic channels at the sizes named in a case
and do not depend on the seed; the seed sets the flow state. A pass starts
from the same state each time (a restored snapshot, as an ensemble or a
serving slot restores one), so every pass does the same work.

The mixed form computes in FP32 (FP64 depth and mass); its fields are read
out as FP32, as a program that picked that form keeps them. The FP64 form's
fields are returned as they are.

exact() restates the fixed-length operations (residual, f-wave substep, HLLC
substep) in 64 bits with plain torch tensor operations; adaptive intervals,
rotor arrays, section solvers and bed updates have no value there.
"""
import functools
import math

import numpy as np
import torch

from braids_hkt_gb300 import scenarios as S
from braids_hkt_gb300 import turbines as TB
from braids_hkt_gb300.solver import RiverSolver

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _case(kind, family, cells, precision="fp64", method="fwave", **more):
    return dict(kind=kind, family=family, cells=cells, precision=precision, method=method, **more)


def listed():
    return [
        # the owner's step on a model of a few hundred cells: calibration loops,
        # tests and teaching models; bound by launches and serial latency
        dict(_case("step", "channel", 360, dt=1.0), name="fp64-step-360"),
        # the same owner with an exact-discharge inlet and a weir: section solves
        # of the boundary CTA at every stage
        dict(_case("step", "inlet-weir", 1500, dt=0.5), name="fp64-step-inlet-weir-1k5"),
        # one residual on Cartesian cells (four faces): implicit or coupled
        # programs that integrate the residual themselves
        dict(_case("rate", "quads", 4030), name="fp64-rate-quads-4k"),
        # the plain method's own configuration (2000 m x 200 m channel, 4 m grid)
        dict(_case("step", "channel", 50000, dt=0.25), name="fp64-step-50k"),
        # a residual on a large ragged reach, out of cache
        dict(_case("rate", "channel", 301777), name="fp64-rate-302k"),
        # three tandem rotors with their refined wakes (one fixed-length trial)
        dict(_case("substep", "rotors", 124041), name="fp64-substep-rotors-124k"),
        # the HLLC / MUSCL-Hancock option in FP64
        dict(_case("substep", "channel", 101003, method="hllc"), name="fp64-hllc-substep-101k"),
        # a short mixed interval on a rotor channel of a few thousand cells: the
        # small request of a serving loop
        dict(_case("advance", "small-rotors", 4000, precision="mixed", dt=0.25), name="mixed-advance-rotors-4k"),
        # the mixed form's substep on one reach beyond the L2 cache
        dict(_case("substep", "channel", 900001, precision="mixed"), name="mixed-substep-900k"),
        # the mixed HLLC form, half that size
        dict(_case("substep", "channel", 450011, precision="mixed", method="hllc"), name="mixed-hllc-substep-450k"),
        # a batch of channels of mixed size with 0 to 8 rotors each, one interval
        dict(_case("advance", "batch", 800000, precision="mixed", dt=0.125, scenarios=12), name="mixed-batch-12"),
        # a braided reach with banks and bars wetting and drying: interval and bed update
        dict(_case("river", "braided", 190000, precision="mixed", dt=0.25), name="mixed-river-braided-190k"),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    family = rng.choice(["channel", "channel", "channel", "quads", "inlet-weir", "rotors", "small-rotors", "batch",
                         "braided"])
    # a program that integrates the residual itself asks for it in FP64
    form = rng.choice(["fp64", "mixed"])
    if family == "channel":
        kind = rng.choice(["step", "rate", "substep", "substep"])
        if kind == "step":
            return _case("step", family, log(300, 60000), dt=rng.choice([0.125, 0.25]))
        form = "fp64" if kind == "rate" else form
        method = rng.choice(["fwave", "hllc"]) if kind == "substep" else "fwave"
        return _case(kind, family, log(600, 300000 if form == "fp64" else 900000), precision=form, method=method)
    if family == "quads":
        kind = rng.choice(["rate", "substep"])
        return _case(kind, family, log(500, 30000), precision="fp64" if kind == "rate" else form)
    if family == "inlet-weir":
        return _case("step", family, log(600, 6000), dt=0.25)
    if family == "rotors":
        return _case("substep", family, log(30000, 124000), precision=form)
    if family == "small-rotors":
        return _case("advance", family, log(3500, 8000), precision="mixed", dt=rng.choice([0.125, 0.25]))
    if family == "batch":
        n = rng.randint(2, 12)
        return _case("advance", family, log(20000, 60000) * n, precision="mixed", dt=0.0625, scenarios=n)
    return _case("river", family, log(20000, 190000), precision=form, dt=0.125 if form == "mixed" else 0.0625)


# ---------------------------------------------------------------------------
# Scenarios of a case (no seed: geometry, bed, boundaries, the base state)
# ---------------------------------------------------------------------------
def _channel(cells, rotors=0):
    """The 10:1 channel of the plain configuration with the grid spacing that
    gives about ``cells`` triangles; small models keep a 24 m wide reach."""
    if cells < 3000:
        width, discharge = 24.0, 20.0
        spacing = 4.0
        length = cells * spacing * spacing / (2.0 * width)
        case = S.small_channel(length=length, width=width, spacing=spacing)
    else:
        width, length, discharge = 200.0, 2000.0, 400.0
        spacing = math.sqrt(2.0 * length * width / cells)
        case = S.channel(length, width, spacing, 0.25 * spacing, seed=1)
    case["q"][1] = np.where(case["q"][0] > 0.0, discharge / width, 0.0)
    return case, spacing


@functools.lru_cache(maxsize=24)
def _scenarios(family, cells, count):
    """(list of base cases, shortest grid spacing)."""
    if family == "channel":
        case, spacing = _channel(cells)
        return [case], spacing
    if family == "quads":
        spacing = 3.0
        width = 24.0 if cells < 3000 else 60.0
        case = S.cartesian_channel(length=spacing * round(cells * spacing / width), width=width, spacing=spacing)
        case["q"][1] = np.where(case["q"][0] > 0.0, 20.0 / width, 0.0)
        return [case], spacing
    if family == "inlet-weir":
        width, spacing, discharge = 40.0, 2.5, 60.0
        length = cells * spacing * spacing / (2.0 * width)
        case = S.stage_discharge_channel(discharge=discharge, reference_stage=3.05, length=length, width=width,
                                         spacing=spacing)
        case["seg_mode"] = np.array([9, 5], np.int32)
        case["outlet"] = {1: {"crest_m": 2.0, "coefficient_m_half_s": 1.7, "effective_width_m": width}}
        case["q"][1] = np.where(case["q"][0] > 0.0, discharge / width, 0.0)
        return [case], spacing
    if family == "rotors":
        # the tandem-rotor configuration; fewer cells: a coarser wake grid
        fine = math.sqrt(84000.0 / max(cells - 40000.0, 20000.0))
        case = S.config2(refine_spacing=fine)
        case["q"][1] = np.where(case["q"][0] > 0.0, 2.0, 0.0)
        return [case], fine
    if family == "small-rotors":
        spacing = math.sqrt(2.0 * 150.0 * 30.0 / cells)
        return [S.small_rotor_channel(spacing=spacing)], spacing
    if family == "batch":
        params = S.config4_params(count, seed=4)
        scale = cells / sum(p["cells"] for p in params)
        for p in params:
            p["cells"] *= scale
            p["spacing"] = math.sqrt(2.0 * p["length"] * p["width"] / p["cells"])
        return [S.config4_case(p) for p in params], min(1.5, min(p["spacing"] for p in params))
    if family == "braided":
        spacing = math.sqrt(2.0 * 2000.0 * 300.0 / cells)
        case = S.config3(length=2000.0, width=300.0, spacing=spacing, rotors=4)
        case["exner"] = S.exner_params(case, diameter=0.003, chezy=40.0)
        case["_flow"] = TB.flow_geometry(case["mesh"])
        return [case], spacing
    raise ValueError(family)


def _base(case):
    return _scenarios(case["family"], int(case["cells"]), int(case.get("scenarios", 1)))


def _state(case, base, rng):
    """The base state with a dozen travelling surface waves of 2 mm to 3 cm
    and currents to match: smooth flow with fronts at the banks, as a running
    model has."""
    q, z = base["q"].copy(), base["z"]
    x, y = base["mesh"].xy
    wide = float(y.max() - y.min())
    amplitude = 0.005 if case["family"] == "braided" else 0.03
    rise, u, v = np.zeros_like(x), np.zeros_like(x), np.zeros_like(x)
    for _ in range(12):
        k = 2 * np.pi / (wide * rng.uniform(0.15, 1.5))
        angle, phase = rng.uniform(0, 2 * np.pi), rng.uniform(0, 2 * np.pi)
        a = amplitude * 10 ** rng.uniform(-1, 0)
        wave = a * np.sin(k * (x * np.cos(angle) + y * np.sin(angle)) + phase)
        rise += wave
        u += 1.5 * wave * np.cos(angle)
        v += 1.5 * wave * np.sin(angle)
    wet = q[0] > 0.0
    h = np.where(wet, np.maximum(q[0] + rise, 0.0), 0.0)
    keep = h / np.where(wet, q[0], 1.0)
    return np.ascontiguousarray(np.stack((h, q[1] * keep + h * u, q[2] * keep + h * v)))


def _trial(base, q):
    """A fixed trial length well inside the CFL limit (0.6 of the bound from
    the largest perimeter / area and the fastest characteristic)."""
    m = base["mesh"]
    per = np.add.reduceat(m.length[m.faces], m.offset[:-1]) / m.area
    h = q[0]
    wet = h > 1e-3
    speed = np.hypot(q[1], q[2])[wet] / h[wet] + np.sqrt(9.81 * h[wet])
    return float(0.6 * 0.9 / (per[wet] * speed).max())


def _states(case, seed):
    rng = np.random.default_rng([int(seed), 0xB1])
    bases, _ = _base(case)
    return [dict(b, q=_state(case, b, rng)) for b in bases]


# ---------------------------------------------------------------------------
# Preparation and one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    cases = _states(case, seed)
    solver = RiverSolver(cases if len(cases) > 1 else cases[0], precision=case["precision"], method=case["method"])
    state = dict(case=case, solver=solver, q0=solver.q.clone(), z0=solver.z.clone(), hints=None)
    if case["family"] == "braided":
        solver.set_forcing_table(cases[0]["table_time"], cases[0]["table_value"])
    if case["kind"] in ("rate", "substep"):
        state["dt"] = _trial(cases[0], cases[0]["q"])
    else:
        # a running program carries the step hint of the interval before
        solver.advance(float(case["dt"]), 0.0)
        state["hints"] = solver.hints()
        solver.q.copy_(state["q0"])
    return state


def _restore(state):
    solver = state["solver"]
    solver.q.copy_(state["q0"])
    if state["hints"] is not None:
        solver.set_hints(state["hints"])
        solver.time[:] = 0.0
    return solver


def _read(case, field):
    return field.float() if case["precision"] == "mixed" else field


def run(state):
    case = state["case"]
    if case["kind"] == "rate":
        rate, water, status, frequency = state["solver"].rate(state["dt"])
        return dict(rate=_read(case, rate), water=_read(case, water), status=int(status))
    solver = _restore(state)
    if case["kind"] == "substep":
        status, _ = solver.substep(state["dt"])
        return dict(q=_read(case, solver.q), status=int(status))
    if case["kind"] == "step":
        out = solver.step(float(case["dt"]))
        return dict(q=out["q"], substeps=out["diagnostics"]["hydraulic_substeps"])
    if case["kind"] == "advance":
        rows = solver.advance(float(case["dt"]), 0.0)
        rows = rows if isinstance(rows, list) else [rows]
        out = dict(q=_read(case, solver.q), substeps=np.array([r["hydraulic_substeps"] for r in rows]))
        if solver.rotors is not None:
            out["rotors"] = solver.turbine_record().astype(np.float32)
        return out
    # "river": the interval, then the bed over it (the bed is restored too)
    solver.z.copy_(state["z0"])
    row = solver.advance(float(case["dt"]), 0.0)
    bed = solver.morphology(float(case["dt"]))
    return dict(q=_read(case, solver.q), z=_read(case, solver.z), substeps=row["hydraulic_substeps"],
                moved=int(bed["ok"]))


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: every geometry record, the bed and the state read once and the
    state (for a residual: rates and fluxes) written once per evaluation
    pass over the mesh, i.e. per substep; flops: the arithmetic of the method
    (counted for the f-wave from executed FP64 instructions, 3110 per cell and
    residual; the Hancock step about half)."""
    cells = float(case["cells"])
    real = 8.0 if case["precision"] == "fp64" else 4.0
    entries, faces = (4.0, 2.0) if case["family"] == "quads" else (3.0, 1.5)
    geometry = entries * (8 + 3 * real) + faces * (8 + 8 * real) + 5 * real
    flow = (4 + 3) * 8.0
    if case["kind"] == "rate":
        return dict(bytes=cells * (geometry + flow + 8.0 * faces), flops=3110.0 * cells)
    substeps = 1.0
    if case["kind"] != "substep":
        # dt = 0.9 / (perimeter / area x speed), 8 m/s on channels, 4 m/s on the braided reach
        spacing = {"channel": 4.0 if cells < 3000 else math.sqrt(8e5 / cells), "inlet-weir": 2.5, "batch": 1.5,
                   "small-rotors": math.sqrt(9000.0 / cells), "braided": math.sqrt(1.2e6 / cells)}[case["family"]]
        speed = 4.0 if case["family"] == "braided" else 8.0
        substeps = max(1.0, case["dt"] * 6.83 / spacing * speed / 0.9)
    per = 3110.0 if case["method"] == "hllc" else 6220.0
    return dict(bytes=substeps * cells * (geometry + flow), flops=substeps * cells * per)


# ---------------------------------------------------------------------------
# The fixed-length operations in 64 bits, in plain tensor operations
# ---------------------------------------------------------------------------
EPS = 2.0 ** -52


def exact(case, seed):
    if case["kind"] not in ("rate", "substep") or case["family"] not in ("channel", "quads"):
        return None
    base = _states(case, seed)[0]
    dt = _trial(base, base["q"])
    R = _Reference(base)
    q = R.tensor(base["q"])
    if case["kind"] == "rate":
        rate, water = R.residual(q, q, dt)
        return dict(rate=rate, water=water, status=None)
    step = R.hancock if case["method"] == "hllc" else R.ssprk
    return dict(q=step(q, dt), status=None)


class _Reference:
    """One scenario with a conveyance inlet (total discharge) and a stage
    outlet, every cell with the same number of faces."""

    def __init__(self, case):
        m, r, ctl = case["mesh"], case["mesh"].records, case["controls"]
        self.g, self.dry, self.manning = ctl["grav"], ctl["dry"], ctl["roughness_value"]
        deg = m.nadj // m.nc
        t, i = self.tensor, lambda a: torch.as_tensor(np.asarray(a, np.int64), device=DEVICE)
        self.nc, self.nf, self.deg = m.nc, m.nf, deg
        self.owner, self.nb, self.bid = i(m.owner), i(m.neighbour), i(m.bid)
        self.faces, self.signs = i(m.faces).view(-1, deg), t(m.signs).view(-1, deg)
        self.inner = self.nb >= 0
        self.nbs = self.nb.clamp(min=0)
        self.wall = ~self.inner & (self.bid < 0)
        self.open = ~self.inner & (self.bid >= 0)
        self.n = t(m.normal)
        self.length, self.area = t(m.length), t(m.area)
        self.other = torch.where(self.signs < 0, self.owner[self.faces], self.nb[self.faces])
        self.has = self.other >= 0
        self.others = self.other.clamp(min=0)
        self.side = (self.signs < 0).long()
        self.disp = t(r["disp"])                                     # [component, side, face]
        self.ls_delta, self.ls_weight = t(r["ls_delta"]).view(2, -1, deg), t(r["ls_weight"]).view(-1, deg)
        self.distance = t(r["distance"])
        self.xy, self.mid = t(m.xy), t(m.mid)
        self.z, self.ext = t(case["z"]), t(case["exterior_bed"])
        self.Q, self.stage = float(case["forcing"][0, 0]), float(case["forcing"][1, 1])

    @staticmethod
    def tensor(a):
        return torch.as_tensor(np.ascontiguousarray(a, np.float64), device=DEVICE)

    # --- shared pieces ------------------------------------------------------
    def velocity(self, q):
        wet = q[0] > self.dry
        h = torch.where(wet, q[0], torch.ones_like(q[0]))
        zero = torch.zeros_like(h)
        return wet, torch.where(wet, q[1] / h, zero), torch.where(wet, q[2] / h, zero)

    def drag(self, q, dt):
        wet, u, v = self.velocity(q)
        h = torch.where(wet, q[0], torch.ones_like(q[0]))
        chezy = h ** (1.0 / 6.0) / self.manning
        factor = 1.0 / (1.0 + dt * self.g * torch.sqrt(u * u + v * v) / (chezy * chezy * h))
        factor = torch.where(wet, factor, torch.zeros_like(h))
        return torch.stack((q[0], q[1] * factor, q[2] * factor))

    def boundary(self, q):
        """Fluxes (3, nf) of the open faces (0 elsewhere) and their water."""
        f = torch.nonzero(self.open).flatten()
        c = self.owner[f]
        h0, bed, (nx, ny), ln = q[0][c], self.ext[f], self.n[:, f], self.length[f]
        _, uc, vc = self.velocity(q)
        geom = (h0 + self.z[c] - bed).clamp(min=0.0)
        h = geom.clone()
        un, inlet = uc[c] * nx + vc[c] * ny, self.bid[f] == 0
        tx, ty = uc[c] - un * nx, vc[c] - un * ny
        # total discharge by conveyance
        wt = torch.where(inlet & (h0 > self.dry), ln, torch.zeros_like(ln))
        section = ((self.z[c] + h0) * wt).sum() / wt.sum()
        w = (section - bed).clamp(min=0.0) ** 1.5 * h.clamp(min=self.dry) ** (1.0 / 6.0) / self.manning * ln
        w = torch.where(inlet & (h > self.dry), w, torch.zeros_like(w))
        speed = -self.Q * w / (w.sum() * h.clamp(min=self.dry) * ln)
        # prescribed stage, half-Riemann outflow
        target, cc = (self.stage - bed).clamp(min=0.0), torch.sqrt(self.g * h)
        k = torch.sqrt(0.5 * self.g * (1.0 / target.clamp(min=1e-9) + 1.0 / h.clamp(min=1e-9)))
        shock = un - target * k < 0.0
        cb = torch.sqrt(self.g * target)
        ub = un + 2.0 * (cc - cb)
        sonic = (un + 2.0 * cc) / 3.0
        rise = target > h
        hb = torch.where(rise, torch.where(shock, target, h), torch.where(
            un - cc >= 0.0, h, torch.where((ub - cb > 0.0) | (target == 0.0), sonic * sonic / self.g, target)))
        vb = torch.where(rise, torch.where(shock, un - (target - h) * k, un), torch.where(
            un - cc >= 0.0, un, torch.where((ub - cb > 0.0) | (target == 0.0), sonic, ub)))
        stop = (un <= -cc) | (vb < 0.0)
        speed = torch.where(inlet, speed, torch.where(stop, torch.zeros_like(vb), vb))
        h = torch.where(inlet | stop, h, hb)
        tx = torch.where(~inlet & stop, torch.zeros_like(tx), tx)
        ty = torch.where(~inlet & stop, torch.zeros_like(ty), ty)
        water, half = h * speed, 0.5 * self.g * h * h
        pressure = 0.5 * self.g * (h0 * h0 - geom * geom)
        flux = torch.zeros((3, self.nf), dtype=torch.float64, device=q.device)
        flux[:, f] = torch.stack((water, water * (speed * nx + tx) + (half + pressure) * nx,
                                  water * (speed * ny + ty) + (half + pressure) * ny))
        return flux

    def limited(self, water, base, q, dt):
        """Donor-limited water, the momentum it no longer carries."""
        out = torch.clamp(self.signs * water[self.faces], min=0.0) * self.length[self.faces]
        is_open = self.open[self.faces]
        prescribed, free = (out * is_open).sum(1), (out * ~is_open).sum(1)
        stock = base[0] * self.area / dt - prescribed
        theta = torch.where((free > 0.0) & (free >= stock),
                            torch.clamp(stock / free.clamp(min=1e-300), max=1.0) * (1.0 - 32.0 * EPS),
                            torch.ones_like(free))
        donor = torch.where(water < 0.0, self.nbs, self.owner)
        factor = torch.where(self.open | (water == 0.0), torch.ones_like(water), theta[donor])
        _, u, v = self.velocity(q)
        lost = (factor - 1.0) * water
        return water * factor, lost * u[donor], lost * v[donor]

    def gather(self, per_owner, per_other):
        """sum(s length flux) / area with each side's own face value."""
        own = per_owner[self.faces]
        value = torch.where(self.signs > 0, own, per_other[self.faces])
        return (self.signs * self.length[self.faces] * value).sum(1) / self.area

    # --- augmented f-wave residual -----------------------------------------
    def reconstruct(self, q):
        """Limited gradients (2, 4, nc) of eta, u, v, b; flatten and active flags."""
        dry, deg = self.dry, self.deg
        wet, u, v = self.velocity(q)
        p = torch.stack((q[0] + self.z, u, v, self.z))               # (4, nc)
        adj = p[:, self.others]                                      # (4, nc, deg)
        nwet = wet[self.others]
        lift = (wet[:, None] & ~nwet & (adj[3] >= p[0][:, None]))
        adj[0] = torch.where(lift, p[0][:, None].expand_as(adj[0]), adj[0])
        adj = torch.where(self.has, adj, p[:, :, None])
        wd = self.ls_weight * self.ls_delta
        b = torch.stack(((wd[0] * (adj - p[:, :, None])).sum(2), (wd[1] * (adj - p[:, :, None])).sum(2)))
        rr = (self.ls_weight * self.ls_delta[0] ** 2).sum(1), (self.ls_weight * self.ls_delta[0] * self.ls_delta[1]).sum(1), \
             (self.ls_weight * self.ls_delta[1] ** 2).sum(1)
        a11, a12, a22 = rr
        det, tr = a11 * a22 - a12 * a12, a11 + a22
        full = det > 1e-12 * tr * tr
        dd, t2 = torch.where(full, det, torch.ones_like(det)), torch.where(tr > 0, tr * tr, torch.ones_like(tr))
        gx = torch.where(full, (a22 * b[0] - a12 * b[1]) / dd, (a11 * b[0] + a12 * b[1]) / t2)
        gy = torch.where(full, (a11 * b[1] - a12 * b[0]) / dd, (a12 * b[0] + a22 * b[1]) / t2)
        active = wet | (self.has & nwet).any(1) | self.open[self.faces].any(1)
        on = active & (tr > 0)
        gx, gy = torch.where(on, gx, torch.zeros_like(gx)), torch.where(on, gy, torch.zeros_like(gy))
        lo, hi = torch.minimum(p, adj.amin(2)), torch.maximum(p, adj.amax(2))
        # a wall bounds the velocities by the mirrored velocity
        for e in range(deg):
            f = self.faces[:, e]
            nx, ny = self.n[0, f], self.n[1, f]
            un = u * nx + v * ny
            use = self.wall[f] & wet & on
            for k, mirror in ((1, u - 2 * un * nx), (2, v - 2 * un * ny)):
                lo[k] = torch.where(use, torch.minimum(lo[k], mirror), lo[k])
                hi[k] = torch.where(use, torch.maximum(hi[k], mirror), hi[k])
        dx = self.disp[0][self.side, self.faces]
        dy = self.disp[1][self.side, self.faces]
        ln = torch.sqrt(dx * dx + dy * dy)
        keep = torch.ones_like(self.has)
        if self.open.any():
            f = self.faces
            un = (u[:, None] * self.n[0, f] + v[:, None] * self.n[1, f]).abs()
            slope = (gx[3][:, None] * dx + gy[3][:, None] * dy).abs()
            keep = ~(self.open[f] & (self.bid[f] == 1) & wet[:, None] & (un < torch.sqrt(self.g * q[0])[:, None]) &
                     (slope > 64 * EPS * self.z.abs().clamp(min=1.0)[:, None]))
        for k in (1, 2):
            d = gx[k][:, None] * dx + gy[k][:, None] * dy
            scale = torch.maximum(p[k].abs(), torch.maximum(lo[k].abs(), hi[k].abs())).clamp(min=1.0)
            use = keep & (d.abs() > 64 * EPS * scale[:, None])
            room = torch.where(d > 0, (hi[k] - p[k])[:, None], (lo[k] - p[k])[:, None])
            th = torch.where(use, room / torch.where(use, d, torch.ones_like(d)), torch.ones_like(d)).amin(1)
            th = th.clamp(min=0.0, max=1.0)
            gx[k], gy[k] = gx[k] * th, gy[k] * th
        none = torch.full_like(ln, math.inf)
        for k, use in ((0, keep), (3, keep & ~self.wall[self.faces])):
            up = torch.where(use, (hi[k] - p[k]).clamp(min=0.0)[:, None] / ln, none)
            down = torch.where(use, (p[k] - lo[k]).clamp(min=0.0)[:, None] / ln, none)
            gx[k], gy[k] = self.project(gx[k], gy[k], torch.cat((dx / ln, -dx / ln), 1),
                                        torch.cat((dy / ln, -dy / ln), 1), torch.cat((up, down), 1))
        de = gx[0][:, None] * dx + gy[0][:, None] * dy
        db = gx[3][:, None] * dx + gy[3][:, None] * dy
        bad = (q[0][:, None] + de - db <= dry) | (db.abs() >= q[0][:, None])
        return p, torch.stack((gx, gy)), ~wet | bad.any(1), active, wet

    @staticmethod
    def project(gx, gy, ax, ay, b):
        """Nearest point of the polygon a . g <= b (the origin is inside)."""
        def feasible(x, y):
            return (ax * x[:, None] + ay * y[:, None] <= b + 2e-14).all(1)

        bx, by, best = torch.zeros_like(gx), torch.zeros_like(gy), gx * gx + gy * gy

        def take(x, y, ok):
            nonlocal bx, by, best
            d = (x - gx) ** 2 + (y - gy) ** 2
            ok = ok & (d < best) & feasible(x, y)
            bx, by, best = torch.where(ok, x, bx), torch.where(ok, y, by), torch.where(ok, d, best)

        inside = feasible(gx, gy)
        for i in range(ax.shape[1]):
            bounded = torch.isfinite(b[:, i])
            bi = torch.where(bounded, b[:, i], torch.zeros_like(gx))
            dot = ax[:, i] * gx + ay[:, i] * gy - bi
            take(gx - dot * ax[:, i], gy - dot * ay[:, i], bounded)
            for j in range(i):
                det = ax[:, i] * ay[:, j] - ay[:, i] * ax[:, j]
                ok = bounded & torch.isfinite(b[:, j]) & (det.abs() >= 1e-12)
                d, bj = torch.where(ok, det, torch.ones_like(det)), torch.where(ok, b[:, j], torch.zeros_like(det))
                take((bi * ay[:, j] - ay[:, i] * bj) / d, (ax[:, i] * bj - bi * ax[:, j]) / d, ok)
        return torch.where(inside, gx, bx), torch.where(inside, gy, by)

    def trace(self, p, grad, flat, wet, q, cell, side):
        dx, dy = self.disp[0, side], self.disp[1, side]
        val = p[:, cell] + grad[0][:, cell] * dx + grad[1][:, cell] * dy
        constant, dry_cell = flat[cell], q[0][cell] <= self.dry
        val[:3] = torch.where(constant, p[:3, cell], val[:3])
        val[3] = torch.where(constant & dry_cell, p[3, cell], val[3])
        raw = (val[0] - val[3]).clamp(min=0.0)
        h = torch.where(dry_cell | (constant & (raw <= self.dry)), torch.zeros_like(raw), raw)
        return h, h * val[1], h * val[2], val[3], raw

    def residual(self, q, base, dt):
        g, dry = self.g, self.dry
        p, grad, flat, active, wet = self.reconstruct(q)
        o, n, inner, (nx, ny) = self.owner, self.nbs, self.inner, self.n
        hL, xL, yL, bL, rawL = self.trace(p, grad, flat, wet, q, o, 0)
        hR, xR, yR, bR, rawR = self.trace(p, grad, flat, wet, q, n, 1)
        dot = xL * nx + yL * ny
        hR, bR, rawR = (torch.where(inner, a, b) for a, b in ((hR, hL), (bR, bL), (rawR, rawL)))
        xR = torch.where(inner, xR, xL - 2 * dot * nx)
        yR = torch.where(inner, yR, yL - 2 * dot * ny)
        unL, utL, unR, utR = dot, -xL * ny + yL * nx, xR * nx + yR * ny, -xR * ny + yR * nx
        top = torch.maximum(bL, bR)
        tol = 16 * EPS * torch.maximum(top.abs(), torch.maximum((hL + bL).abs(), (hR + bR).abs())).clamp(min=dry)
        sl, sr = (hL + bL - top).clamp(min=0.0), (hR + bR - top).clamp(min=0.0)
        sl, sr = torch.where(sl <= dry + tol, 0 * sl, sl), torch.where(sr <= dry + tol, 0 * sr, sr)
        sl, sr = torch.where(inner, sl, hL), torch.where(inner, sr, hR)
        kl = torch.where(hL > dry, sl / hL.clamp(min=dry), 0 * hL)
        kr = torch.where(hR > dry, sr / hR.clamp(min=dry), 0 * hR)
        kl, kr = torch.where(inner, kl, torch.ones_like(kl)), torch.where(inner, kr, torch.ones_like(kr))
        loc = [sl, unL * kl, utL * kl, torch.where(inner, top, bL), sr, unR * kr, utR * kr, torch.where(inner, top, bR)]
        # wet/dry faces whose shared surface stays below the higher bed are closed
        hc, hn, zc, zn = q[0][o], q[0][n], self.z[o], self.z[n]
        dc, dn = self.distance
        shared = (dn * (zc + hc) + dc * (zn + hn)) / (dc + dn).clamp(min=1e-300) - torch.maximum(zc, zn)
        closed = inner & ~(torch.minimum(hc, hn) > dry) & (shared <= dry)
        wl, wr = hL > dry, hR > dry
        vl, vr = unL / hL.clamp(min=dry), unR / hR.clamp(min=dry)
        ml = self.riemann(hL.clamp(min=dry * 2), hL.clamp(min=dry * 2), vl, -vl)[0]
        mr = self.riemann(hR.clamp(min=dry * 2), hR.clamp(min=dry * 2), -vr, vr)[0]
        opens = torch.where(wl & ~wr & (vl > 0), (ml > hL + dry) & (ml + bL > bR + dry),
                            torch.where(wr & ~wl & (-vr > 0), (mr > hR + dry) & (mr + bR > bL + dry),
                                        torch.zeros_like(wl)))
        closed = closed & ~opens
        am, ap = self.fwave(loc)
        half = 0.5 * g

        def flux(s, un, ut):
            on = s > dry
            d = torch.where(on, s, torch.ones_like(s))
            zero = torch.zeros_like(s)
            return [torch.where(on, un, zero), torch.where(on, un * un / d + half * s * s, zero),
                    torch.where(on, un * ut / d, zero)]

        fl, fr = flux(loc[0], loc[1], loc[2]), flux(loc[4], loc[5], loc[6])
        fl = [a + b for a, b in zip(fl, am)]
        fr = [a - b for a, b in zip(fr, ap)]
        water = 0.5 * (fl[0] + fr[0])
        cl = torch.where(inner, half * (hL * hL - loc[0] ** 2), 0 * hL)
        cr = torch.where(inner, half * (hR * hR - loc[4] ** 2), 0 * hR)
        l1, l2 = (fl[1] + cl) * nx - fl[2] * ny, (fl[1] + cl) * ny + fl[2] * nx
        r1, r2 = (fr[1] + cr) * nx - fr[2] * ny, (fr[1] + cr) * ny + fr[2] * nx
        wallp = self.wall_pressure(hL, unL)
        l1, l2 = torch.where(inner, l1, wallp * nx), torch.where(inner, l2, wallp * ny)
        water = torch.where(closed | ~inner, 0 * water, water)
        l1, l2 = torch.where(closed, half * hL * hL * nx, l1), torch.where(closed, half * hL * hL * ny, l2)
        r1, r2 = torch.where(closed, half * hR * hR * nx, r1), torch.where(closed, half * hR * hR * ny, r2)
        kL = torch.where(flat[o], half * (hc * hc - hL * hL), half * (hc + rawL) * (bL - zc))
        kR = torch.where(flat[n], half * (hn * hn - hR * hR), half * (hn + rawR) * (bR - zn))
        kL, kR = torch.where(hc > dry, kL, 0 * kL), torch.where(hn > dry, kR, 0 * kR)
        l1, l2, r1, r2 = l1 + kL * nx, l2 + kL * ny, r1 + kR * nx, r2 + kR * ny
        idle = (hc <= dry) & (~inner | (hn <= dry))
        water, l1, l2, r1, r2 = (torch.where(idle, 0 * a, a) for a in (water, l1, l2, r1, r2))
        ext = self.boundary(q)
        water, l1, l2 = (torch.where(self.open, e, a) for e, a in zip(ext, (water, l1, l2)))
        # each cell gathers the flux above its own pressure
        pc, pn = half * hc * hc, half * hn * hn
        m1 = self.gather(l1 - pc * nx, r1 - pn * nx)
        m2 = self.gather(l2 - pc * ny, r2 - pn * ny)
        m1, m2 = torch.where(active, m1, 0 * m1), torch.where(active, m2, 0 * m2)
        water, cx, cy = self.limited(water, base, q, dt)
        return torch.stack((-self.gather(water, water), -m1 - self.gather(cx, cx), -m2 - self.gather(cy, cy))), water

    def riemann(self, hL, hR, uL, uR):
        """Middle depth and speeds of the approximate Riemann state (one step)."""
        g, dry = self.g, self.dry
        rt = lambda a: torch.sqrt(a.clamp(min=0.0))                  # noqa: E731
        lo, hi, du = torch.minimum(hL, hR), torch.maximum(hL, hR), uR - uL
        los, his = lo.clamp(min=dry), hi.clamp(min=dry)
        fmn = du + 2 * (rt(g * lo) - rt(g * hi))
        fmx = du + (hi - lo) * rt(0.5 * g * (hi + lo) / (his * los))
        rar = (-du + 2 * (rt(g * hL) + rt(g * hR))).clamp(min=0.0) ** 2 / (16 * g)
        a = uL + 2 * rt(g * hL), uR - 2 * rt(g * hR)
        h0 = his
        gL, gR = rt(0.5 * g * (1 / h0 + 1 / hL.clamp(min=dry))), rt(0.5 * g * (1 / h0 + 1 / hR.clamp(min=dry)))
        F0 = du + (h0 - hL) * gL + (h0 - hR) * gR
        slope = 2 * rt(h0) * (gL - g * (h0 - hL) / (4 * h0 * h0 * gL) + gR - g * (h0 - hR) / (4 * h0 * h0 * gR))
        two = (rt(h0) - F0 / slope) ** 2
        twos = two.clamp(min=1e-300)
        s1 = uL - (two - hL) * rt(0.5 * g * (1 / twos + 1 / hL.clamp(min=dry))) - rt(g * two)
        s2 = uR + (two - hR) * rt(0.5 * g * (1 / twos + 1 / hR.clamp(min=dry))) + rt(g * two)
        F1 = du + 2 * (rt(g * lo) - rt(g * hi))
        gap = hi - lo
        slope1 = (fmx - F1) / torch.where(gap > 0, gap, torch.ones_like(gap))
        mix = lo - F1 / torch.where(slope1 != 0, slope1, torch.ones_like(slope1))
        left = hL > hR
        m1 = torch.where(left, a[0] - 3 * rt(g * mix), a[1] + rt(g * mix))
        m2 = torch.where(left, a[0] - rt(g * mix), a[1] + 3 * rt(g * mix))
        pick = lambda r, s, m: torch.where(fmn > 0, r, torch.where(fmx <= 0, s, m))   # noqa: E731
        hm, s1m, s2m = pick(rar, two, mix), pick(a[0] - 3 * rt(g * rar), s1, m1), pick(a[1] + 3 * rt(g * rar), s2, m2)
        dryside = lo <= dry
        edge = uR + uL - 2 * rt(g * hR) + 2 * rt(g * hL)
        return torch.where(dryside, 0 * hm, hm), torch.where(dryside, edge, s1m), torch.where(dryside, edge, s2m)

    def fwave(self, loc):
        """Left- and right-going fluctuations of the augmented solver."""
        g, dry = self.g, self.dry
        hL, qL, tL, bL, hR, qR, tR, bR = (a.clone() for a in loc)
        dl, dr = hL <= dry, hR <= dry
        zero, one = torch.zeros_like(hL), torch.ones_like(hL)
        hL, qL, tL = (torch.where(dl, zero, a) for a in (hL, qL, tL))
        hR, qR, tR = (torch.where(dr, zero, a) for a in (hR, qR, tR))
        dL, dR = torch.where(dl, one, hL), torch.where(dr, one, hR)
        uL, vL, uR, vR = qL / dL, tL / dL, qR / dR, tR / dR
        pL, pR = 0.5 * g * hL * hL + qL * uL, 0.5 * g * hR * hR + qR * uR
        # a dry side reflects where the wet side's stagnation depth stays below its bed
        starR = torch.maximum(hL, self.riemann(dL, dL, uL, -uL)[0])
        refl = dr & ~dl & (starR + bL < bR)
        lift = dr & ~dl & ~refl & (hL + bL < bR)
        starL = torch.maximum(hR, self.riemann(dR, dR, -uR, uR)[0])
        refr = dl & ~dr & (starL + bR < bL)
        lifr = dl & ~dr & ~refr & (hR + bR < bL)
        w = [torch.where(refr, zero, one), torch.where(refl | refr, zero, one), torch.where(refl, zero, one)]
        bR, bL = torch.where(lift, hL + bL, bR), torch.where(lifr, hR + bR, bL)
        nhR, nqR, nbR, npR, nuR, nvR = hL, -qL, bL, pL, -uL, vL
        nhL, nqL, nbL, npL, nuL, nvL = hR, -qR, bR, pR, -uR, vR
        pick = torch.where
        hR, qR, bR, pR, uR, vR = (pick(refl, a, b) for a, b in zip((nhR, nqR, nbR, npR, nuR, nvR), (hR, qR, bR, pR, uR, vR)))
        hL, qL, bL, pL, uL, vL = (pick(refr, a, b) for a, b in zip((nhL, nqL, nbL, npL, nuL, nvL), (hL, qL, bL, pL, uL, vL)))
        cL, cR = torch.sqrt(g * hL), torch.sqrt(g * hR)
        both = (cL + cR).clamp(min=1e-300)
        uh, ch = (cL * uL + cR * uR) / both, torch.sqrt(0.5 * g * (hL + hR))
        _, s1m, s2m = self.riemann(hL, hR, uL, uR)
        e1 = torch.minimum(torch.minimum(uL - cL, uh - ch), s2m)
        e2 = torch.maximum(torch.maximum(uR + cR, uh + ch), s1m)
        gap = torch.where(e2 - e1 != 0, e2 - e1, one)
        hll = ((qL - qR + e2 * hR - e1 * hL) / gap).clamp(min=0.0)
        crit = max(dry * g, 1e-6)
        root = math.sqrt(crit)
        hbar, db = 0.5 * (hL + hR), bR - bL
        sbar = 0.25 * (uL + uR) ** 2 - g * hbar
        stil = (uL * uR).clamp(min=0.0) - g * hbar
        sonic = (sbar.abs() <= crit) | (sbar * stil <= crit * crit) | (sbar * e1 * e2 <= crit * crit) | \
                (torch.minimum(e1.abs(), e2.abs()) < root) | ((e1 < root) & (s1m > -root)) | \
                ((e2 > -root) & (s2m < root)) | ((uL + cL) * (uR + cR) < 0) | ((uL - cL) * (uR - cR) < 0)
        sb = torch.where(sonic, one, sbar)
        dh = torch.where(sonic, -db, db * g * hbar / sb)
        n1, n2 = torch.where(e1 != 0, e1, one), torch.where(e2 != 0, e2, one)
        span = hll * (e2 - e1)
        mid = (e1 < -crit) & (e2 > crit)
        right, left = ~mid & (e1 >= crit), ~mid & ~(e1 >= crit) & (e2 <= -crit)
        dh = torch.where(mid, torch.maximum(torch.minimum(dh, span / n2), span / n1), dh)
        dh = torch.where(right, torch.maximum(torch.minimum(dh, span / n1), -hL), dh)
        dh = torch.where(left, torch.maximum(torch.minimum(dh, hR), span / n2), dh)
        dp = torch.where(sonic, -g * hbar * db, -db * g * hbar * stil / sb)
        dp = torch.minimum(dp, g * torch.maximum(-hL * db, -hR * db))
        dp = torch.maximum(dp, g * torch.minimum(-hL * db, -hR * db))
        d0, d1, d2 = hR - hL - dh, qR - qL, pR - pL - dp
        det = torch.where(e1 - e2 != 0, e2 - e1, one)
        b0, b2 = (d0 * e2 - d1) / det, (d1 - d0 * e1) / det
        b1 = d2 - b0 * e1 * e1 - b2 * e2 * e2
        f = [[b0 * e1, b0 * e1 * e1, b0 * e1 * vL], [zero, b1, zero], [b2 * e2, b2 * e2 * e2, b2 * e2 * vR]]
        rest = hR * uR * vR - hL * uL * vL - f[0][2] - f[2][2]
        to_left = qL + f[0][0] <= 0
        f[0][2] = f[0][2] + torch.where(to_left, rest, zero)
        f[2][2] = f[2][2] + torch.where(to_left, zero, rest)
        s = [e1 * w[0], 0.5 * (e1 + e2) * w[1], e2 * w[2]]
        am, ap = [zero] * 3, [zero] * 3
        for k in range(3):
            share = torch.where(s[k] < -1e-14, one, torch.where(s[k] > 1e-14, zero, 0.5 * one))
            for c in range(3):
                am[c] = am[c] + share * w[k] * f[k][c]
                ap[c] = ap[c] + (1 - share) * w[k] * f[k][c]
        idle = dl & dr
        return [torch.where(idle, zero, a) for a in am], [torch.where(idle, zero, a) for a in ap]

    def wall_pressure(self, h, un):
        wet = h > self.dry
        d = torch.where(wet, h, torch.ones_like(h))
        v = un / d / torch.sqrt(self.g * d)
        r = 1.0 + v.clamp(min=0.0)
        for _ in range(40):                                          # (r - 1) sqrt((1 + 1/r) / 2) = v
            s = torch.sqrt(0.5 * (1 + 1 / r))
            r = (r - ((r - 1) * s - v.clamp(min=0.0)) / (s - (r - 1) / (4 * s * r * r))).clamp(min=1.0)
        ratio = torch.where(v <= 0, (1 + 0.5 * v).clamp(min=0.0) ** 2, r)
        return torch.where(wet, 0.5 * self.g * (h * ratio) ** 2, torch.zeros_like(h))

    def settled(self, q):
        wet = q[0] > self.dry
        return torch.stack((q[0], torch.where(wet, q[1], 0 * q[1]), torch.where(wet, q[2], 0 * q[2])))

    def ssprk(self, q, dt):
        a = self.drag(q, 0.5 * dt)
        b = self.settled(a + dt * self.residual(a, a, dt)[0])
        return self.drag(self.settled(0.5 * a + 0.5 * (b + dt * self.residual(b, b, dt)[0])), 0.5 * dt)

    # --- HLLC / MUSCL-Hancock step ------------------------------------------
    def hancock(self, q, dt):
        g, dry, z = self.g, self.dry, self.z
        q = self.drag(q, 0.5 * dt)
        wet, u, v = self.velocity(q)
        p = torch.stack((q[0] + z, u, v, z))
        f = self.faces
        o = p[:, self.others]
        lift = ~wet[self.others] & (o[3] >= p[0][:, None])
        o[0] = torch.where(lift, p[0][:, None].expand_as(o[0]), o[0])
        nx, ny = self.n[0, f], self.n[1, f]
        un = u[:, None] * nx + v[:, None] * ny
        mirror = torch.stack((p[0][:, None].expand_as(un), u[:, None] - 2 * un * nx, v[:, None] - 2 * un * ny,
                              p[3][:, None].expand_as(un)))
        o = torch.where(self.has, o, mirror)
        mx, my = self.mid[0][f] - self.xy[0][:, None], self.mid[1][f] - self.xy[1][:, None]
        dist = 2 * (mx * nx + my * ny)
        dx = torch.where(self.has, self.xy[0][self.others] - self.xy[0][:, None], dist * nx)
        dy = torch.where(self.has, self.xy[1][self.others] - self.xy[1][:, None], dist * ny)
        use = ~self.open[f]
        d2 = dx * dx + dy * dy
        zero = torch.zeros_like(dx)
        wx, wy = torch.where(use, dx / d2, zero), torch.where(use, dy / d2, zero)
        a11, a12, a22 = (wx * dx).sum(1), (wx * dy).sum(1), (wy * dy).sum(1)
        det = a11 * a22 - a12 * a12
        jump = torch.where(use, o - p[:, :, None], torch.zeros_like(o))
        bx, by = (jump * wx).sum(2), (jump * wy).sum(2)
        gx, gy = (a22 * bx - a12 * by) / det, (a11 * by - a12 * bx) / det
        lo, hi = jump.amin(2).clamp(max=0.0), jump.amax(2).clamp(min=0.0)
        d = gx[:, :, None] * mx + gy[:, :, None] * my
        room = torch.where(d > 0, hi[:, :, None], lo[:, :, None])
        lim = torch.where(d != 0, room / torch.where(d != 0, d, torch.ones_like(d)), torch.ones_like(d))
        lim = lim.amin(2).clamp(max=1.0)
        gx, gy = gx * lim, gy * lim
        gx[:3], gy[:3] = torch.where(wet, gx[:3], 0 * gx[:3]), torch.where(wet, gy[:3], 0 * gy[:3])
        hc = q[0]
        eta = p[0] - 0.5 * dt * (u * (gx[0] - gx[3]) + v * (gy[0] - gy[3]) + hc * (gx[1] + gy[2]))
        uh = u - 0.5 * dt * (u * gx[1] + v * gy[1] + g * gx[0])
        vh = v - 0.5 * dt * (u * gx[2] + v * gy[2] + g * gy[0])
        under = eta < z
        eta, uh, vh = torch.where(under | ~wet, p[0], eta), torch.where(under, u, uh), torch.where(under, v, vh)
        uh, vh = torch.where(wet, uh, 0 * uh), torch.where(wet, vh, 0 * vh)
        P = torch.stack((eta, uh, vh, z))
        hh = (eta - z).clamp(min=0.0)
        ext = self.boundary(torch.stack((hh, hh * uh, hh * vh)))
        # faces
        l, r, inner = self.owner, self.nbs, self.inner
        nx, ny = self.n
        L = P[:, l] + gx[:, l] * self.disp[0, 0] + gy[:, l] * self.disp[1, 0]
        R = P[:, r] + gx[:, r] * self.disp[0, 1] + gy[:, r] * self.disp[1, 1]
        R = torch.where(inner, R, L)
        ldry, rdry = P[0][l] - z[l] <= dry, inner & (P[0][r] - z[r] <= dry)
        either = ldry | rdry
        L[3] = torch.where(either, z[l], L[3])
        R[3] = torch.where(either, torch.where(inner, z[r], L[3]), R[3])
        for side, off in ((L, ldry), (R, rdry)):
            side[0] = torch.where(off, side[3], side[0])
            side[1], side[2] = torch.where(off, 0 * side[1], side[1]), torch.where(off, 0 * side[2], side[2])
        un = R[1] * nx + R[2] * ny
        R[1] = torch.where(inner, R[1], R[1] - 2 * un * nx)
        R[2] = torch.where(inner, R[2], R[2] - 2 * un * ny)
        top = torch.maximum(L[3], R[3])
        hl, hr = (L[0] - L[3]).clamp(min=0.0), (R[0] - R[3]).clamp(min=0.0)
        sl, sr = (L[0] - top).clamp(min=0.0), (R[0] - top).clamp(min=0.0)
        out = self.hllc(sl, L[1] * nx + L[2] * ny, -L[1] * ny + L[2] * nx, sr, R[1] * nx + R[2] * ny,
                        -R[1] * ny + R[2] * nx)
        el = (P[0][l] - L[3]).clamp(min=0.0)
        er = torch.where(inner, (P[0][r] - R[3]).clamp(min=0.0), el)
        pl, pr = 0.5 * g * (hl * hl - sl * sl - el * el), 0.5 * g * (hr * hr - sr * sr - er * er)
        l1, l2 = (out[1] + pl) * nx - out[2] * ny, (out[1] + pl) * ny + out[2] * nx
        r1, r2 = (out[1] + pr) * nx - out[2] * ny, (out[1] + pr) * ny + out[2] * nx
        water = torch.where(inner, out[0], 0 * out[0])
        own = 0.5 * g * hh[l] ** 2
        water, l1, l2 = (torch.where(self.open, e, a) for e, a in
                         zip((ext[0], ext[1] - own * nx, ext[2] - own * ny), (water, l1, l2)))
        water, cx, cy = self.limited(water, q, q, dt)
        new = torch.stack((q[0] - dt * self.gather(water, water), q[1] - dt * self.gather(l1 + cx, r1 + cx),
                           q[2] - dt * self.gather(l2 + cy, r2 + cy)))
        return self.drag(self.settled(new), 0.5 * dt)

    def hllc(self, hl, ul, vl, hr, ur, vr):
        g, dry = self.g, self.dry
        cl, cr = torch.sqrt(g * hl), torch.sqrt(g * hr)
        sl, sr = torch.minimum(ul - cl, ur - cr), torch.maximum(ul + cl, ur + cr)
        dl, dr = hl <= dry, hr <= dry
        sl, sr = torch.where(dl, ur - 2 * cr, sl), torch.where(dr, ul + 2 * cl, sr)
        fl = [hl * ul, hl * ul * ul + 0.5 * g * hl * hl, hl * ul * vl]
        fr = [hr * ur, hr * ur * ur + 0.5 * g * hr * hr, hr * ur * vr]
        a, b = hl * (sl - ul), hr * (sr - ur)
        some = (a - b).abs() > 1e-30
        den = torch.where(some, a - b, torch.ones_like(a))
        sm = torch.where(some, (0.5 * g * (hr * hr - hl * hl) + a * ul - b * ur) / den, 0 * a)
        contact = ~dl & ~dr & (sl < sm) & (sm < sr)
        gl, gr = torch.where(contact, sl - sm, -torch.ones_like(a)), torch.where(contact, sr - sm, torch.ones_like(a))
        hs = torch.where(sm >= 0, a / gl, b / gr)
        contact = contact & (hs >= 0)
        left = [fl[0] + sl * (hs - hl), fl[1] + sl * (hs * sm - hl * ul), fl[2] + sl * (hs * vl - hl * vl)]
        right = [fr[0] + sr * (hs - hr), fr[1] + sr * (hs * sm - hr * ur), fr[2] + sr * (hs * vr - hr * vr)]
        w = torch.where(sr - sl != 0, sr - sl, torch.ones_like(sl))
        U = ((hl, hl * ul, hl * vl), (hr, hr * ur, hr * vr))
        out = []
        for k in range(3):
            hlle = (sr * fl[k] - sl * fr[k] + sl * sr * (U[1][k] - U[0][k])) / w
            x = torch.where(contact, torch.where(sm >= 0, left[k], right[k]), hlle)
            x = torch.where(sl >= 0, fl[k], torch.where(sr <= 0, fr[k], x))
            out.append(torch.where(dl & dr, 0 * x, x))
        return out
