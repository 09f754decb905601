// FP64 update of the f-wave step: gather, donor limiter, CFL frequency, stage
// combination and closing drag in one sweep over the cells.
//
// The donor factor of a cell needs all of its outflow, and the fluxes a cell
// receives need its neighbours' factors, so this was two sweeps with the
// rates in memory between them. But a factor differs from one only where a
// cell would run dry within the substep. The sweep therefore updates every
// cell with the unlimited fluxes, forms its own factor, and lists the cells
// whose factor is not one; k_limited then redoes those cells and the
// neighbours they drain into with the limited fluxes. Both write what the two
// sweeps wrote: the unlimited update of a cell no limited donor feeds is the
// limited one, operation for operation.
//
// Bound by FP64 instructions (brx_num64.cuh): length / area per entry and
// 1 / area per cell are tables, the donor test and the sign and threshold
// tests run on the integer pipe.
// Gather + update per stage, before -> after (k_limited included): 302k cells
// 69 + 94 -> 78 us, 50k 23 + 29 -> 29 us, 360 cells 15 + 18 -> 21 us.
#pragma once
#include "brx_num64.cuh"

namespace brx {

// Entry and cell tables; cw may be null (the HLLC method reads the cells' alone).
__global__ void __launch_bounds__(256) k64_weights(MeshDev m, double2 *cw, double *rarea)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < m.nc; c += gridDim.x * blockDim.x) {
        const double area = m.area[c];
        rarea[c] = 1. / area;
        if (!cw) continue;
        for (int k = m.offset[c]; k < m.offset[c + 1]; ++k) {
            const double len = m.length[m.faces[k]];
            cw[k] = make_double2(m.signs[k] * len / area, len);
        }
    }
}

__device__ __forceinline__ double2 entry_weight(const MeshDev &m, const Work &w, int c, int k)
{
    if (w.cw) return w.cw[k];
    const double len = m.length[m.faces[k]];
    return make_double2(m.signs[k] * len / m.area[c], len);
}

// Rotor, viscosity and stage terms of one cell whose hydraulic rates are r0,
// r1, r2; result into the stage's target. Status is raised unless quiet.
__device__ __forceinline__ void finish_cell(const MeshDev &m, const StateDev &s, Ctrl &ct, const Work &w, int stage,
                                            int sid, int c, double r0, double r1, double r2, double *rate_out,
                                            const TurbDev &t, int turb, Prim64 *prim, bool quiet)
{
    const int nc = m.nc;
    if (turb && t.hkt[sid]) add_rotor_momentum(m, t, sid, c, m.area[c], r1, r2, true, w.rarea[c]);
    if (w.visc.nu && w.visc.nu[sid] > 0.) add_viscosity(m, w.visc, c, m.area[c], r1, r2);
    if (!finite_bits(r0) || !finite_bits(r1) || !finite_bits(r2)) raise_status(ct, stage, ST_RATE);
    if (rate_out) { rate_out[c] = r0; rate_out[nc + c] = r1; rate_out[2 * nc + c] = r2; return; }
    const double dt = ct.trial, dry = ct.dry;
    if (stage == 1) {
        const double h = s.work[c] + dt * r0;
        double hu = s.work[nc + c] + dt * r1, hv = s.work[2 * nc + c] + dt * r2;
        if (!quiet && negative(h)) raise_status(ct, 1, ST_ENDPOINT);
        if (!greater(h, dry)) { hu = 0.; hv = 0.; }
        s.q1[c] = h; s.q1[nc + c] = hu; s.q1[2 * nc + c] = hv;
        if (prim) put_prim64(prim, c, h, hu, hv, s.z[c], dry);       // the second stage's
    } else {
        double h = .5 * s.work[c] + .5 * (s.q1[c] + dt * r0);
        double hu = .5 * s.work[nc + c] + .5 * (s.q1[nc + c] + dt * r1);
        double hv = .5 * s.work[2 * nc + c] + .5 * (s.q1[2 * nc + c] + dt * r2);
        if (!quiet && (!finite_bits(h) || !finite_bits(hu) || !finite_bits(hv) || negative(h)))
            raise_status(ct, 2, ST_ENDPOINT);
        if (!greater(h, dry)) { hu = 0.; hv = 0.; }
        drag_cell(ct, .5 * dt, h, hu, hv);
        double *qn = ct.cur ? s.q[0] : s.q[1];
        qn[c] = h; qn[nc + c] = hu; qn[2 * nc + c] = hv;
    }
}

// With rate_out set, the rate is stored there and no state is written.
__global__ void __launch_bounds__(256) k64_update(MeshDev m, StateDev s, Ctrl *ctrl, Work w, int stage,
                                                  double *rate_out, TurbDev t, int turb, Prim64 *prim)
{
    const int nc = m.nc;
    const int stride = gridDim.x * blockDim.x;
    const int na = m.act.count[1];
    for (int first = blockIdx.x * blockDim.x; first < na; first += stride) {   // warp-uniform trip count
        const int c = first + (int)threadIdx.x < na ? active_cell(m.act, first + threadIdx.x) : nc;
        bool have = false;
        double fr = 0.;
        int sid = 0;
        if (c < nc) {
            sid = m.cell_sid[c];
            Ctrl &ct = ctrl[sid];
            if (!skip_stage(ct, stage)) {
                const double *base = stage == 1 ? s.work : s.q1;
                const double dt = ct.trial, area = m.area[c];
                const bool owns_open = m.cflags[c] & 1;
                double sum0 = 0., sum1 = 0., sum2 = 0., out = 0., freq = 0., ext = 0., interior = 0.;
                for (int k = m.offset[c]; k < m.offset[c + 1]; ++k) {
                    const int f = m.faces[k];
                    const double2 wl = entry_weight(m, w, c, k);
                    const double2 ws = w.ws[f];
                    const double4_32a gf = w.gf[f];
                    const bool own = __double_as_longlong(wl.x) >= 0;
                    sum0 += wl.x * ws.x;
                    sum1 += wl.x * (own ? gf.x : gf.z);
                    sum2 += wl.x * (own ? gf.y : gf.w);
                    freq += wl.y * ws.y;
                    const double debit = (__double_as_longlong(ws.x) >= 0) == own ? fabs(ws.x) * wl.y : 0.;
                    out += debit;
                    if (owns_open) { if (m.bslot[f] >= 0) ext += debit; else interior += debit; }
                }
                const double stock = base[c] * area;
                double theta = 1.;
                if (greater(out, 0.) && !greater(stock, dt * out)) theta = fmin(1., stock / (dt * out)) * (1. - 32. * EPS);
                if (owns_open) {
                    const double available = stock / dt;
                    if (ext > available) raise_status(ct, stage, ST_BUDGET);
                    const double factor = fmin(1., (available - ext) / fmax(interior, 1e-300)) * (1. - 32. * EPS);
                    theta = (interior > 0. && interior >= available - ext) ? factor : 1.;
                }
                w.theta[c] = theta;
                const bool limits = theta != 1.;
                if (limits) w.limited[atomicAdd(&m.act.count[2 + stage], 1)] = c;
                fr = w.rarea && finite_bits(freq) ? quotient(freq, area, w.rarea[c]) : freq / area;
                if (isnan(fr)) raise_status(ct, stage, ST_FREQ);
                else have = true;
                const bool active = w.rec[c].flags & 2;
                // (0 - 0 is 0: the rate of a cell at rest has no sign)
                finish_cell(m, s, ct, w, stage, sid, c, 0. - sum0, active ? -sum1 : 0., active ? -sum2 : 0., rate_out, t,
                            turb, prim, limits);
            }
        }
        unsigned long long *peak0 = stage == 1 ? &ctrl[0].peak1 : &ctrl[0].peak2;
        warp_max_peak(peak0, sizeof(Ctrl), sid, have, fr);
    }
}

// One cell with the donor-limited fluxes of its faces (midpoint_faces and
// midpoint_gather, river_midpoint.h:30-49): the same values k_limit stores.
__device__ void limited_cell(const MeshDev &m, const StateDev &s, Ctrl *ctrl, const Work &w, int stage, int c,
                             double *rate_out, const TurbDev &t, int turb, Prim64 *prim)
{
    const int nc = m.nc, sid = m.cell_sid[c];
    Ctrl &ct = ctrl[sid];
    const double *q = stage == 1 ? s.work : s.q1;
    double mass = 0., mx = 0., my = 0., sum1 = 0., sum2 = 0.;
    for (int k = m.offset[c]; k < m.offset[c + 1]; ++k) {
        const int f = m.faces[k];
        const double wt = entry_weight(m, w, c, k).x;
        const double4_32a gf = w.gf[f];
        double water = w.ws[f].x;
        sum1 += wt * (wt > 0. ? gf.x : gf.z);
        sum2 += wt * (wt > 0. ? gf.y : gf.w);
        if (water != 0. && m.bslot[f] < 0) {
            const int donor = water < 0. ? m.neighbour[f] : m.owner[f];
            if (donor >= 0) {
                const double th = w.theta[donor];
                if (th != 1.) {
                    const double delta = (th - 1.) * water;
                    water *= th;
                    const double hd = q[donor];
                    if (hd > ct.dry) {
                        mx -= wt * (delta * q[nc + donor] / hd);
                        my -= wt * (delta * q[2 * nc + donor] / hd);
                    }
                }
            }
        }
        mass -= wt * water;
    }
    const bool active = w.rec[c].flags & 2;
    finish_cell(m, s, ct, w, stage, sid, c, mass, (active ? -sum1 : 0.) + mx, (active ? -sum2 : 0.) + my, rate_out, t,
                turb, prim, false);
}

// Redo the listed cells and the neighbours they drain into. A cell reached
// from several list entries is redone by each with the same result; nothing
// read here is written here (stage 1 reads work and writes q1, stage 2 reads
// both and writes the inactive buffer).
__global__ void __launch_bounds__(64) k_limited(MeshDev m, StateDev s, Ctrl *ctrl, Work w, int stage, double *rate_out,
                                                TurbDev t, int turb, Prim64 *prim)
{
    // four threads per listed cell: itself, then its entries in turn; a
    // neighbour that is listed too is left to its own entry
    const int n = 4 * m.act.count[2 + stage];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = w.limited[i >> 2], part = i & 3;
        if (part == 0) limited_cell(m, s, ctrl, w, stage, c, rate_out, t, turb, prim);
        for (int k = m.offset[c] + (part + 3) % 4; k < m.offset[c + 1]; k += 4) {
            const int f = m.faces[k];
            const double water = w.ws[f].x;
            const int o = m.signs[k] > 0 ? m.neighbour[f] : m.owner[f];
            if (o >= 0 && (m.signs[k] > 0 ? water > 0. : water < 0.) && w.theta[o] == 1.)
                limited_cell(m, s, ctrl, w, stage, o, rate_out, t, turb, prim);
        }
    }
}

}  // namespace brx
