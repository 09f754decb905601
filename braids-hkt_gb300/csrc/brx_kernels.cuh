// Kernels of one SSPRK(2,2) substep of the augmented f-wave river step.
//
// Included by one translation unit per arithmetic form. Each includer
// defines BRX_NS (the namespace its kernel copies live in) so the FP64
// unit (-fmad=false, reference operation order) and the mixed unit (FP32
// fluxes, FMA on) never share a symbol. The boundary kernels, whose arithmetic
// differs between the forms, are templates on the flux type F; the others are
// the FP64 form's and evaluate the FP64 expressions of the reference.
#pragma once
#include "brx_common.cuh"
#include <cooperative_groups.h>
#include "brx_num64.cuh"

#ifndef BRX_NS
#error "define BRX_NS before including brx_kernels.cuh"
#endif

namespace BRX_NS {
using namespace brx;
// ---------------------------------------------------------------------------
// Drag: cell-local implicit Manning/Chezy friction over dt_scale * trial.
// src/braids_core/sediment/river_hydraulic_drag.h:3-16
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ F chezy(int method, F depth, F value)
{
    if (method == 1) return value;
    if (method == 2) return pow(depth, F(1.) / F(6.)) / value;
    if (method == 3) return sqrt(F(9.81)) / F(.41) * log1p(F(30.) * depth / (exp(F(1.)) * value));
    return F(18.) * log10(F(12.) * fmax(F(.5), depth / value));
}

// The drag factor by plain divisions, where quotient() leaves its domain: a
// momentum whose square is infinite (factor 0: the cell stops), a roughness whose
// squared Chezy coefficient is (factor 1: no friction) or vanishes (factor 0).
static __device__ __noinline__ double drag_factor_far(const Ctrl &ct, double square, double h, double dt)
{
    const double c = ct.roughness_mode == 2 ? cbrt(sqrt(h)) / ct.roughness_value
                                            : chezy<double>(ct.roughness_mode, h, ct.roughness_value);
    const double speed = sqrt(square) / h;
    return 1. / (1. + dt * ct.grav * speed / (c * c * h));
}

// The depth's sixth root of Manning's law is cbrt(sqrt(h)) (25 FP64
// instructions, good to about one ulp) instead of pow (88, two ulp), and the
// quotients go through quotient(): 61 instructions instead of 145. Error of the
// factor over depths 1e-6 to 20 m: rms 1.2e-16, largest 7.5e-16 (with pow 1.8e-16
// and 1.1e-15). The opening half-step takes 57 us instead of 97 on 302k cells, 13
// instead of 18 on 360.
__device__ __forceinline__ void drag_cell(const Ctrl &ct, double dt, double &h, double &hu, double &hv)
{
    if (!greater(h, ct.dry)) { hu = 0.; hv = 0.; return; }
    const double c = ct.roughness_mode == 2 ? quotient(cbrt(sqrt(h)), ct.roughness_value, ct.rrough)
                                            : chezy<double>(ct.roughness_mode, h, ct.roughness_value);
    const double square = hu * hu + hv * hv, stiff = c * c * h;
    const double speed = quotient(sqrt(square), h, reciprocal(h));
    const double y = 1. + quotient(dt * ct.grav * speed, stiff, reciprocal(stiff));
    double factor = quotient(1., y, reciprocal(y));
    if (!finite_bits(factor)) factor = drag_factor_far(ct, square, h, dt);
    hu *= factor;
    hv *= factor;
}

// work = drag(accepted, trial/2); prim (may be null): the first stage's primitives
__global__ void k_open_drag(MeshDev m, StateDev s, Ctrl *ctrl, Prim64 *prim)
{
    const int nc = m.nc;
    FOR_ACTIVE_CELLS(m.act, c) {
        const Ctrl &ct = ctrl[m.cell_sid[c]];
        if (!ct.active || ct.done) continue;
        const double *q = ct.cur ? s.q[1] : s.q[0];
        double h = q[c], hu = q[nc + c], hv = q[2 * nc + c];
        drag_cell(ct, .5 * ct.trial, h, hu, hv);
        s.work[c] = h; s.work[nc + c] = hu; s.work[2 * nc + c] = hv;
        if (prim) put_prim64(prim, c, h, hu, hv, s.z[c], ct.dry);
    }
}

// ---------------------------------------------------------------------------
// Boundary: one CTA per scenario evaluates its open segments (stage sums,
// conveyance weights, exterior traces/fluxes) and caps outlet outflow by the
// owners' stage-start stock. Sums use the reference's fixed tree: 64-face
// tiles from each segment start, then the tiles in order.
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ F exterior_chezy(int mode, F h, F parameter, F floor_, F gravity, int waqua)
{
    const F d = fmax(h, floor_);
    if (mode == 1) return parameter;
    if (mode == 2) return pow(d, F(1.) / F(6.)) / parameter;
    return waqua ? F(18.) * log10(F(12.) * fmax(F(.5), d / parameter))
                 : sqrt(gravity) / F(.41) * log1p(F(30.) * d / (exp(F(1.)) * parameter));
}

// Conveyance weight per unit width of an inlet face: section^1.5 times
// Chezy's coefficient at depth h (at least the dry depth). In FP64 the powers
// are section sqrt(section) and cbrt(sqrt(h)): 36 FP64 instructions instead of
// 176, each good to about one ulp.
template <class F>
__device__ __forceinline__ double conveyance(int mode, int waqua, F section, F h, const Ctrl &ct)
{
    if constexpr (sizeof(F) == 8) {
        const double chezy = mode == 2 ? quotient(cbrt(sqrt(h)), ct.roughness_value, ct.rrough)
                                       : exterior_chezy<F>(mode, h, ct.roughness_value, ct.dry, ct.grav, waqua);
        return section * sqrt(section) * chezy;
    } else
        return double(pow(section, F(1.5)) *
                      exterior_chezy<F>(mode, h, F(ct.roughness_value), F(ct.dry), F(ct.grav), waqua));
}

// c = sqrt(gravity h)
__device__ __forceinline__ void stage_wave(double h, double un, double target, double gravity, double c, double &depth,
                                           double &velocity)
{
    depth = h; velocity = un;
    if (target > h) {
        const double k = sqrt(.5 * gravity * (quotient(1., target, reciprocal(target)) + quotient(1., h, reciprocal(h))));
        const double shock = un - target * k;
        if (shock >= 0.) return;
        depth = target; velocity = un - (target - h) * k;
        return;
    }
    if (un - c >= 0.) return;
    const double cb = sqrt(gravity * target), ub = un + 2. * (c - cb);
    if (ub - cb > 0. || target == 0.) {
        velocity = (un + 2. * c) / 3.; depth = velocity * velocity / gravity;
        return;
    }
    depth = target; velocity = ub;
}

__device__ __forceinline__ bool is_outlet(int mode)
{
    return mode == 2 || mode == 3 || mode == 4 || mode == 5 || mode == 10 || mode == 11;
}

// The scenario's slots in tiles of 64 from each segment start.
__device__ __forceinline__ int tile_count(const BoundaryDev &b, int sg)
{
    return max(1, (b.seg_off[sg + 1] - b.seg_off[sg] + 63) / 64);
}

struct SlotTile { int sg, first, end; };

__device__ __forceinline__ SlotTile slot_tile(const BoundaryDev &b, int s0, int t)
{
    int sg = s0;
    for (int n = tile_count(b, sg); t >= n; n = tile_count(b, sg)) { t -= n; ++sg; }
    const int first = b.seg_off[sg] + 64 * t;
    return {sg, first, min(b.seg_off[sg + 1], first + 64)};
}

constexpr int BOUNDARY_THREADS = 128;      // one warp per sub-partition: FP64 work does not overlap within one
// openings beyond a cluster, which keep one block: its loads and FP32 powers want
// more warps. Openings of 1,030 / 2,000 / 4,000 faces, 128 -> 512 threads, us a
// stage: FP64 193 / 359 / 711 -> 147 / 264 / 522, mixed 176 / 329 / 652 -> 129 / 231 / 464
// (256: 155 / 283 / 555 and 138 / 252 / 498)
constexpr int BOUNDARY_WIDE = 512;

// The sum of a tile's terms in slot order, formed by one warp: lane l's terms
// are those of slots first + l and first + 32 + l; rows are summed by as many
// lanes at once. Result of row r in lane r.
template <int ROWS>
__device__ __forceinline__ double tile_sum(double (*buf)[64], int n, const double (&lo)[ROWS], const double (&hi)[ROWS])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) { buf[r][lane] = lo[r]; buf[r][lane + 32] = hi[r]; }
    __syncwarp();
    double sum = 0.;
    if (lane < ROWS)
        for (int i = 0; i < n; ++i) sum += buf[lane][i];
    __syncwarp();
    return sum;
}

// ---------------------------------------------------------------------------
// Q-H rating outlet (mode 11): the common water elevation at which the
// outgoing characteristic discharge of the opening equals the rating curve,
// then each face's trace (river_rating_outlet.h:15-102). One thread per
// segment, faces in boundary order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rating_velocity(double h, double hi, double u, double g)
{
    return h > hi ? u - (h - hi) * sqrt(.5 * g * (1. / h + 1. / hi)) : u + 2. * (sqrt(g * hi) - sqrt(g * h));
}

__device__ double rating_q(const BoundaryDev &b, int sg, double eta)
{
    const int a = b.rt_off[sg], end = b.rt_off[sg + 1];
    if (eta <= b.rt_eta[a]) return b.rt_q[a];
    if (eta >= b.rt_eta[end - 1]) return b.rt_q[end - 1];
    int lo = a, hi = end - 1;
    while (hi - lo > 1) { const int mid = (lo + hi) / 2; if (b.rt_eta[mid] <= eta) lo = mid; else hi = mid; }
    const double w = (eta - b.rt_eta[lo]) / (b.rt_eta[hi] - b.rt_eta[lo]);
    return (1. - w) * b.rt_q[lo] + w * b.rt_q[hi];
}

__device__ double rating_residual(const MeshDev &m, const BoundaryDev &b, int sg, double eta, double g, double dry,
                                  const double *q, const double *z, double &actual)
{
    const int nc = m.nc, nf = m.nf;
    double Q = 0.;
    for (int k = b.seg_off[sg]; k < b.seg_off[sg + 1]; ++k) {
        const int f = b.slot_face[k], c = m.owner[f];
        const double bed = b.ext_bed[k], hc = q[c], hi = fmax(hc + z[c] - bed, 0.);
        if (hc <= dry || hi <= dry) continue;
        const double u = (q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[nf + f]) / hc;
        if (u >= sqrt(g * hi)) { Q += hi * u * m.length[f]; continue; }
        const double h = fmax(eta - bed, 0.);
        if (h > dry) Q += h * fmax(rating_velocity(h, hi, u, g), 0.) * m.length[f];
    }
    actual = Q;
    return Q - rating_q(b, sg, eta);
}

// 0, or the section failure: 1 no bracket, 2 residual, 3 a fictitious zero-flow root.
__device__ __noinline__ int rating_section(const MeshDev &m, const BoundaryDev &b, int sg, double g, double dry, double speed,
                              const double *q, const double *z, bool &bad)
{
    const int nc = m.nc, nf = m.nf;
    double lo = b.rt_eta[b.rt_off[sg]], hi = b.rt_eta[b.rt_off[sg + 1] - 1];
    int wet = 0;
    for (int k = b.seg_off[sg]; k < b.seg_off[sg + 1]; ++k) {
        const int f = b.slot_face[k], c = m.owner[f];
        const double h0 = q[c], h = fmax(h0 + z[c] - b.ext_bed[k], 0.);
        if (h0 <= dry || h <= dry) continue;
        const double u = (q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[nf + f]) / h0;
        if (u >= sqrt(g * h)) continue;
        double left = dry, right = fmax(h, 1.);
        for (int it = 0; it < 60 && rating_velocity(right, h, u, g) > sqrt(g * right); ++it) right *= 2.;
        for (int it = 0; it < 60; ++it) {
            const double mid = .5 * (left + right);
            if (rating_velocity(mid, h, u, g) > sqrt(g * mid)) left = mid; else right = mid;
        }
        lo = fmax(lo, b.ext_bed[k] + right);
        ++wet;
    }
    double level = 0., actual = 0.;
    if (wet) {
        if (!(lo <= hi)) return 1;
        const double rlo = rating_residual(m, b, sg, lo, g, dry, q, z, actual);
        const double rhi = rating_residual(m, b, sg, hi, g, dry, q, z, actual);
        if (!isfinite(rlo) || !isfinite(rhi) || rlo < 0. || rhi > 0.) return 1;
        for (int it = 0; it < 90; ++it) {
            const double mid = .5 * (lo + hi);
            if (mid == lo || mid == hi) break;
            if (rating_residual(m, b, sg, mid, g, dry, q, z, actual) > 0.) lo = mid; else hi = mid;
        }
        level = .5 * (lo + hi);
        const double r = rating_residual(m, b, sg, level, g, dry, q, z, actual);
        if (!isfinite(r) || fabs(r) > 1e-10 * fmax(1., fabs(actual))) return 2;
        if (actual <= 1e-14)
            for (int k = b.seg_off[sg]; k < b.seg_off[sg + 1]; ++k) {
                const int f = b.slot_face[k], c = m.owner[f];
                const double hc = q[c], hh = fmax(hc + z[c] - b.ext_bed[k], 0.);
                if (hc <= dry || hh <= dry) continue;
                const double ui = (q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[nf + f]) / hc;
                const double h = fmax(level - b.ext_bed[k], 0.);
                if (h > dry && ui < sqrt(g * hh) && rating_velocity(h, hh, ui, g) < -1e-12) return 3;
            }
    }
    const size_t ns = b.nslot;
    for (int k = b.seg_off[sg]; k < b.seg_off[sg + 1]; ++k) {
        const int f = b.slot_face[k], c = m.owner[f];
        const double bed = b.ext_bed[k], h0 = q[c], geom = fmax(h0 + z[c] - bed, 0.);
        const double nx = m.normal[f], ny = m.normal[nf + f];
        double ux = 0., uy = 0.;
        if (h0 > dry) { ux = q[nc + c] / h0; uy = q[2 * nc + c] / h0; }
        double un = ux * nx + uy * ny, h = geom;
        const double tx = ux - un * nx, ty = uy - un * ny;
        if (h0 <= dry || geom <= dry) { h = 0.; un = 0.; }
        else if (!(un >= sqrt(g * geom))) {     // subcritical: the common level; supercritical keeps its own
            const double incoming = un;
            h = fmax(level - bed, 0.);
            un = h > dry ? rating_velocity(h, geom, incoming, g) : 0.;
            if (un <= 0.) {                      // reflected: the stagnation depth of the incoming stream
                double left = dry, right = fmax(geom, 1.);
                for (int it = 0; it < 60 && rating_velocity(right, geom, incoming, g) > 0.; ++it) right *= 2.;
                for (int it = 0; it < 80; ++it) {
                    const double mid = .5 * (left + right);
                    if (rating_velocity(mid, geom, incoming, g) > 0.) left = mid; else right = mid;
                }
                h = .5 * (left + right);
                un = 0.;
            }
        }
        if (!isfinite(h) || !isfinite(un) || sqrt(un * un + tx * tx + ty * ty) > speed) { bad = true; continue; }
        double water = 0., fx = 0., fy = 0., t0 = 0., t1 = 0., t2 = 0.;
        if (h > dry) {
            t0 = h; t1 = h * (un * nx + tx); t2 = h * (un * ny + ty);
            water = h * un;
            fx = water * (un * nx + tx) + .5 * g * h * h * nx;
            fy = water * (un * ny + ty) + .5 * g * h * h * ny;
        }
        const double pressure = h0 > dry ? .5 * g * (h0 * h0 - geom * geom) : 0.;
        b.trace[k] = t0; b.trace[ns + k] = t1; b.trace[2 * ns + k] = t2;
        b.flux[k] = water; b.flux[ns + k] = fx + pressure * nx; b.flux[2 * ns + k] = fy + pressure * ny;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Normal-depth outlet (mode 10): per connected face chain, the level at which
// the outgoing characteristic discharge equals the uniform-flow conveyance
// at the chain's bed slope (river_normal_outlet.h:17-134). One thread per
// chain; dry faces close with their owner's pressure.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double nout_chezy(int law, double r, double value, double g)
{
    if (law == 1) return value;
    if (law == 2) return pow(r, 1. / 6.) / value;
    if (law == 3) return sqrt(g) / .41 * log1p(30. * r / (exp(1.) * value));
    return 18. * log10(12. * fmax(.5, r / value));
}

__device__ double nout_residual(const MeshDev &m, const BoundaryDev &b, const int *slots, int start, int end,
                                double eta, double slope, double g, double dry, int law, double rough,
                                const double *q, const double *z, double &area_out, double &q_out)
{
    const int nc = m.nc, nf = m.nf;
    double area = 0., perimeter = 0., rate = 0., drag = 0., prev = 0.;
    for (int k = start; k < end; ++k) {
        const int sl = slots[k], f = b.slot_face[sl];
        const double h = fmax(eta - b.ext_bed[sl], 0.);
        area += h * m.length[f];
        perimeter += h > dry ? m.length[f] : 0.;
        if (k == start) perimeter += h; else perimeter += fabs(h - prev);
        prev = h;
    }
    perimeter += prev;
    if (area <= 0. || perimeter <= 0.) { area_out = 0.; q_out = 0.; return 0.; }
    const double radius = area / perimeter;
    const double manning_radius = law == 2 ? pow(radius, 1. / 6.) : 0.;
    for (int k = start; k < end; ++k) {
        const int sl = slots[k], f = b.slot_face[sl], c = m.owner[f];
        const double bed = b.ext_bed[sl], h0 = q[c], hi = fmax(h0 + z[c] - bed, 0.), h = fmax(eta - bed, 0.);
        double face_rate = 0.;
        if (h0 > dry && hi > dry) {
            const double ui = (q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[nf + f]) / h0;
            if (ui >= sqrt(g * hi)) face_rate = ui * hi;
            else {
                const double invariant = fmax(ui + 2. * sqrt(g * hi), 0.), sonic = invariant * invariant / (9. * g);
                if (h < sonic) face_rate = sonic * sqrt(g * sonic);
                else if (h > dry) face_rate = h * fmax(rating_velocity(h, hi, ui, g), 0.);
            }
        }
        rate += face_rate * m.length[f];
        if (h <= dry) continue;
        const double left = k == start ? 0. : fmax(eta - b.ext_bed[slots[k - 1]], 0.);
        const double right = k + 1 == end ? 0. : fmax(eta - b.ext_bed[slots[k + 1]], 0.);
        const double p = m.length[f] + fmax(h - left, 0.) + fmax(h - right, 0.);
        const double C = law == 2 ? manning_radius / rough : nout_chezy(law, radius, rough, g);
        drag += p / (C * C);
    }
    area_out = area; q_out = rate;
    return rate - (drag > 0. ? area * sqrt(area * slope / drag) : 0.);
}

// 0, or the chain's failure (a trial rejection in the reference).
__device__ __noinline__ int normal_chain(const MeshDev &m, const BoundaryDev &b, int ch, double g, double dry, double speed,
                            int law, double rough, const double *q, const double *z, bool &bad)
{
    const int nc = m.nc, nf = m.nf;
    const size_t ns = b.nslot;
    const int *slots = b.chain_slot;
    const double slope = b.chain_slope[ch];
    int cursor = b.chain_off[ch];
    const int stop = b.chain_off[ch + 1];
    while (cursor < stop) {
        const int fsl = slots[cursor], ff = b.slot_face[fsl], fc = m.owner[ff];
        const double fh = q[fc], fgeom = fmax(fh + z[fc] - b.ext_bed[fsl], 0.);
        if (fh <= dry || fgeom <= dry) {
            const double pressure = fh > dry ? .5 * g * fh * fh : 0.;
            b.trace[fsl] = 0.; b.trace[ns + fsl] = 0.; b.trace[2 * ns + fsl] = 0.;
            b.flux[fsl] = 0.; b.flux[ns + fsl] = pressure * m.normal[ff]; b.flux[2 * ns + fsl] = pressure * m.normal[nf + ff];
            ++cursor;
            continue;
        }
        const int start = cursor;
        while (cursor < stop) {
            const int sl = slots[cursor], f = b.slot_face[sl], c = m.owner[f];
            const double hh = q[c];
            if (hh <= dry || hh + z[c] - b.ext_bed[sl] <= dry) break;
            ++cursor;
        }
        const int end = cursor;
        int wet = 0;
        double lo = 1e300, hi = -1e300, area = 0., rate = 0.;
        for (int k = start; k < end; ++k) {
            const int sl = slots[k], f = b.slot_face[sl], c = m.owner[f];
            const double h0 = q[c], hf = fmax(h0 + z[c] - b.ext_bed[sl], 0.);
            if (h0 <= dry || hf <= dry) continue;
            const double u = (q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[nf + f]) / h0;
            if (u >= sqrt(g * hf)) continue;
            lo = fmin(lo, b.ext_bed[sl] + 2. * dry);
            hi = fmax(hi, z[c] + h0);
            ++wet;
        }
        double level = 0.;
        bool fallback = false;
        if (wet) {
            hi = fmax(hi, lo + 1.);
            double r = nout_residual(m, b, slots, start, end, lo, slope, g, dry, law, rough, q, z, area, rate);
            if (!isfinite(r)) return 1;
            if (r < 0.) fallback = true;           // supercritical normal flow: keep the outgoing trace
            else {
                double rh = nout_residual(m, b, slots, start, end, hi, slope, g, dry, law, rough, q, z, area, rate);
                for (int it = 0; it < 60 && rh > 0.; ++it) {
                    hi = lo + 2. * (hi - lo);
                    rh = nout_residual(m, b, slots, start, end, hi, slope, g, dry, law, rough, q, z, area, rate);
                }
                if (!isfinite(rh) || rh > 0.) return 2;
                for (int it = 0; it < 90; ++it) {
                    const double mid = .5 * (lo + hi);
                    if (mid == lo || mid == hi) break;
                    r = nout_residual(m, b, slots, start, end, mid, slope, g, dry, law, rough, q, z, area, rate);
                    if (r > 0.) lo = mid; else hi = mid;
                }
                level = .5 * (lo + hi);
                r = nout_residual(m, b, slots, start, end, level, slope, g, dry, law, rough, q, z, area, rate);
                if (!isfinite(r) || fabs(r) > 1e-10 * fmax(1., fabs(rate))) return 3;
            }
        }
        for (int k = start; k < end; ++k) {
            const int sl = slots[k], f = b.slot_face[sl], c = m.owner[f];
            const double bed = b.ext_bed[sl], h0 = q[c], geom = fmax(h0 + z[c] - bed, 0.);
            const double nx = m.normal[f], ny = m.normal[nf + f];
            double ux = 0., uy = 0.;
            if (h0 > dry) { ux = q[nc + c] / h0; uy = q[2 * nc + c] / h0; }
            double un = ux * nx + uy * ny, h = geom;
            const double tx = ux - un * nx, ty = uy - un * ny;
            if (h0 <= dry || geom <= dry) { h = 0.; un = 0.; }
            else if (fallback) { }
            else if (un >= sqrt(g * geom)) { }
            else {
                const double incoming = un;
                h = fmax(level - bed, 0.);
                const double invariant = fmax(incoming + 2. * sqrt(g * geom), 0.), sonic = invariant * invariant / (9. * g);
                if (h < sonic) { h = sonic; un = sqrt(g * sonic); }
                else un = h > dry ? rating_velocity(h, geom, incoming, g) : 0.;
                if (un <= 0.) {
                    double left = dry, right = fmax(geom, 1.);
                    for (int it = 0; it < 60 && rating_velocity(right, geom, incoming, g) > 0.; ++it) right *= 2.;
                    for (int it = 0; it < 80; ++it) {
                        const double mid = .5 * (left + right);
                        if (rating_velocity(mid, geom, incoming, g) > 0.) left = mid; else right = mid;
                    }
                    h = .5 * (left + right);
                    un = 0.;
                }
            }
            if (!isfinite(h) || !isfinite(un) || sqrt(un * un + tx * tx + ty * ty) > speed) { bad = true; continue; }
            double water = 0., fx = 0., fy = 0., t0 = 0., t1 = 0., t2 = 0.;
            if (h > dry) {
                t0 = h; t1 = h * (un * nx + tx); t2 = h * (un * ny + ty);
                water = h * un;
                fx = water * (un * nx + tx) + .5 * g * h * h * nx;
                fy = water * (un * ny + ty) + .5 * g * h * h * ny;
            }
            const double pressure = h0 > dry ? .5 * g * (h0 * h0 - geom * geom) : 0.;
            b.trace[sl] = t0; b.trace[ns + sl] = t1; b.trace[2 * ns + sl] = t2;
            b.flux[sl] = water; b.flux[ns + sl] = fx + pressure * nx; b.flux[2 * ns + sl] = fy + pressure * ny;
        }
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Section solves with 128 logical lanes (river_exterior_outlet.h): the whole
// boundary CTA works on one section; lane l (threads 0..127) sums entries
// l, l+128, ... of the section and thread 0 adds the lane sums in lane order,
// the order of the reference's OpenMP and CUDA forms. Every thread of the
// CTA calls these functions (they synchronise the block).
// ---------------------------------------------------------------------------
constexpr int SECTION_LANES = 128;

struct SectionWork {
    double part[4][SECTION_LANES];
    double sum[4];
    int error;
};

// Sums of the first ROWS rows of w.part over lanes 0 .. n-1 in lane order, one
// thread per row in a warp of its own (their FP64 chains then run side by
// side); every thread gets them. Lanes from n on hold nothing: the section has
// n < SECTION_LANES faces. Block-cooperative.
template <int ROWS>
__device__ __forceinline__ void lane_sums(SectionWork &w, int n, double (&sum)[ROWS])
{
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        for (int r = threadIdx.x >> 5; r < ROWS; r += blockDim.x >> 5) {
            double t = 0.;
            for (int lane = 0; lane < n; ++lane) t += w.part[r][lane];
            w.sum[r] = t;
        }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROWS; ++r) sum[r] = w.sum[r];
}

// Bisect [lo, hi], f(lo) >= 0 >= f(hi), to neighbouring numbers. Where f has
// several roots the one found depends on the points tried: these are the
// reference's. Critical outlets of 8 / 128 / 1,030 faces: 191 / 521 / 1,851 us a stage
// (by the steps below, which may end on another root, 106 / 286 / 1,318; with the
// lanes summed by one thread 1,039 / 1,085 / 2,144).
template <class Fn>
__device__ __forceinline__ void bisect_bracket(double &lo, double &hi, const Fn &f)
{
    for (int j = 0; j < 90; ++j) {
        const double mid = lo + .5 * (hi - lo);
        if (mid == lo || mid == hi) return;
        if (f(mid) > 0.) lo = mid; else hi = mid;
    }
}

// The same end for an f that decreases throughout, and so has one root. Each
// round evaluates the secant point and then twice the distance it is still
// off, which as a rule is just across the root: the width falls with the
// square, some twelve evaluations instead of bisection's fifty-odd. A round
// that does not halve the interval bisects.
template <class Fn>
__device__ __forceinline__ void shrink_bracket(double &lo, double &hi, double flo, double fhi, const Fn &f)
{
    for (int round = 0; round < 90; ++round) {
        const double mid = lo + .5 * (hi - lo);
        if (mid == lo || mid == hi) return;
        const double width = hi - lo, fall = flo - fhi;
        double x = fall > 0. ? lo + width * (flo / fall) : mid;
        if (!(x > lo && x < hi)) x = mid;
        const double fx = f(x);
        const bool left = fx > 0.;
        if (left) { lo = x; flo = fx; } else { hi = x; fhi = fx; }
        const double off = fall > 0. ? fmax(2. * fabs(fx) * (width / fall), 4. * EPS * fabs(x)) : width;
        const double y = left ? x + off : x - off;
        if (y > lo && y < hi) {
            const double fy = f(y);
            if (fy > 0.) { lo = y; flo = fy; } else { hi = y; fhi = fy; }
        }
        if (hi - lo > .5 * width) {
            const double v = lo + .5 * (hi - lo);
            if (v == lo || v == hi) return;
            const double fv = f(v);
            if (fv > 0.) { lo = v; flo = fv; } else { hi = v; fhi = fv; }
        }
    }
}

__device__ __forceinline__ double weir_velocity(double h, double hi, double ui, double g)
{
    return h > hi ? ui - (h - hi) * sqrt(.5 * g * (1. / h + 1. / hi)) : ui + 2. * (sqrt(g * hi) - sqrt(g * h));
}

// river_exterior_outlet.h:207-227: discharge minus the weir's at stage eta,
// the same in every thread.
__device__ __noinline__ double weir_residual(SectionWork &w, const MeshDev &m, const BoundaryDev &b, int k0, int k1, double eta,
                                double g, double dry, double crest, double factor, const double *q, const double *z)
{
    const int n = min(k1 - k0, SECTION_LANES);
    for (int lane = threadIdx.x; lane < n; lane += blockDim.x) {
        double rate = 0.;
        for (int k = k0 + lane; k < k1; k += SECTION_LANES) {
            if (!b.branch[k]) continue;
            const int f = b.slot_face[k], c = m.owner[f];
            const double bed = b.ext_bed[k], h = fmax(eta - bed, 0.), hi = fmax(q[c] + z[c] - bed, 0.);
            if (h <= dry) continue;
            const double u = fmax(weir_velocity(h, hi, b.invariant[k], g), 0.);
            if (u > 0.) rate += h * u * m.length[f];
        }
        w.part[0][lane] = rate;
    }
    double sum[1];
    lane_sums<1>(w, n, sum);
    const double head = fmax(eta - crest, 0.);
    return sum[0] - factor * head * sqrt(head);
}

// Free weir on segment sg (river_exterior_outlet.h:229-360): the common
// subcritical stage at which the outgoing Lax-curve discharge equals
// coefficient x width x head^1.5. Returns 0 or the section failure (a trial
// rejection in the reference); `bad` gets the speed-limit face status.
__device__ __noinline__ int weir_section(SectionWork &w, const MeshDev &m, const BoundaryDev &b, int sg, double g, double dry,
                            double speed, const double *q, const double *z, bool &bad)
{
    const int nc = m.nc, nf = m.nf, nseg = b.nseg, k0 = b.seg_off[sg], k1 = b.seg_off[sg + 1];
    const size_t ns = b.nslot;
    const double tol = 128. * EPS, crest = b.weir[sg], factor = b.weir[nseg + sg] * b.weir[2 * nseg + sg];
    if (threadIdx.x == 0) w.error = 0;
    // wet faces, each with its incoming normal speed; the bracket of the stage
    // from their sonic depths and their own levels (maxima: in any order)
    double lo = -INFINITY, hi = -INFINITY;
    double highest = -INFINITY;              // bed of the wet faces
    bool some = false;
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int f = b.slot_face[k], c = m.owner[f];
        b.branch[k] = 0; b.invariant[k] = 0.;
        const double hc = q[c], h0 = fmax(hc + z[c] - b.ext_bed[k], 0.);
        if (hc <= dry || h0 <= dry) continue;
        const double u = (q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[nf + f]) / hc;
        b.branch[k] = 1; b.invariant[k] = u;
        some = true;
        double left = 0., right = fmax(h0, 1.);
        for (int it = 0; it < 60 && weir_velocity(right, h0, u, g) > sqrt(g * right); ++it) right *= 2.;
        const auto f_sonic = [&](double h) { return weir_velocity(h, h0, u, g) - sqrt(g * h); };
        shrink_bracket(left, right, f_sonic(left), f_sonic(right), f_sonic);
        lo = fmax(lo, b.ext_bed[k] + right);
        hi = fmax(hi, hc + z[c]);
        highest = fmax(highest, b.ext_bed[k]);
    }
    double eta = 0.;
    if (__syncthreads_or(some)) {
        const int n = min(k1 - k0, (int)blockDim.x);
        if ((int)threadIdx.x < n) { w.part[0][threadIdx.x] = lo; w.part[1][threadIdx.x] = hi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 0; i < n; ++i) { lo = fmax(lo, w.part[0][i]); hi = fmax(hi, w.part[1][i]); }
            w.sum[0] = lo; w.sum[1] = hi;
        }
        __syncthreads();
        lo = fmax(w.sum[0], crest);
        hi = fmax(w.sum[1], lo + 1.);
        __syncthreads();
        const auto residual = [&](double at) { return weir_residual(w, m, b, k0, k1, at, g, dry, crest, factor, q, z); };
        int error = 0;
        const double rlo = residual(lo);
        double rhi = 0.;
        if (rlo < 0. || !isfinite(rlo)) error = 1;
        else {
            rhi = residual(hi);
            for (int j = 0; j < 60 && rhi > 0.; ++j) { hi = lo + 2. * (hi - lo); rhi = residual(hi); }
            if (rhi > 0. || !isfinite(rhi)) error = 1;
        }
        if (!error) {
            // Above every face's sonic stage its discharge falls with the stage,
            // unless the face is not deeper than the dry depth there: its
            // discharge then sets in at a jump within the bracket, and there may
            // be a root on either side.
            if (__syncthreads_or(some && highest + dry * (1. + 1.e-9) + 4. * EPS * fabs(highest) >= lo))
                bisect_bracket(lo, hi, residual);
            else shrink_bracket(lo, hi, rlo, rhi, residual);
            eta = lo + .5 * (hi - lo);
            const double r = residual(eta), head = fmax(eta - crest, 0.), requested = factor * head * sqrt(head);
            if (!isfinite(r) || fabs(r) > 1e-10 * fmax(requested, 1.)) error = 2;
            bool inward = false;
            for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
                if (b.branch[k] != 1) continue;
                const int c = m.owner[b.slot_face[k]];
                const double bed = b.ext_bed[k], h0 = fmax(q[c] + z[c] - bed, 0.), h = fmax(eta - bed, 0.);
                const double u = weir_velocity(h, h0, b.invariant[k], g);
                if (h <= dry || u <= 0.) { b.branch[k] = 0; continue; }
                // a downstream-only shock may not enter the domain
                if (h > h0 && b.invariant[k] - h * sqrt(.5 * g * (1. / h + 1. / h0)) > tol) inward = true;
            }
            if (__syncthreads_or(inward)) error = 5;
        }
        if (error) return error;             // the same in every thread
    } else {
        for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) b.branch[k] = 0;
    }
    __syncthreads();
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int f = b.slot_face[k], c = m.owner[f];
        const double bed = b.ext_bed[k], h0 = q[c], geom = fmax(h0 + z[c] - bed, 0.);
        const double nx = m.normal[f], ny = m.normal[nf + f];
        double h = geom, ux = 0., uy = 0.;
        if (h0 > dry) { ux = q[nc + c] / h0; uy = q[2 * nc + c] / h0; } else h = 0.;
        double un = ux * nx + uy * ny;
        const double tx = ux - un * nx, ty = uy - un * ny;
        if (b.branch[k] == 0) {
            // a blocked stream reflects with its stagnation / shock depth
            if (geom > dry && h0 > dry && un != 0.) {
                double lo = 0., hi = fmax(geom, 1.);
                for (int it = 0; it < 60 && weir_velocity(hi, geom, un, g) > 0.; ++it) hi *= 2.;
                for (int it = 0; it < 80; ++it) {
                    const double mid = .5 * (lo + hi);
                    if (weir_velocity(mid, geom, un, g) > 0.) lo = mid; else hi = mid;
                }
                h = .5 * (lo + hi);
            }
            un = 0.;
        } else {
            h = fmax(eta - bed, 0.);
            un = weir_velocity(h, geom, b.invariant[k], g);
        }
        if (!isfinite(h) || !isfinite(un) || sqrt(un * un + tx * tx + ty * ty) > speed) { bad = true; continue; }
        double water = 0., fx = 0., fy = 0., t0 = 0., t1 = 0., t2 = 0.;
        if (h > dry) {
            t0 = h; t1 = h * (un * nx + tx); t2 = h * (un * ny + ty);
            water = t1 * nx + t2 * ny;
            fx = water * t1 / h + .5 * g * h * h * nx;
            fy = water * t2 / h + .5 * g * h * h * ny;
        }
        const double pressure = h0 > dry ? .5 * g * (h0 * h0 - geom * geom) : 0.;
        b.trace[k] = t0; b.trace[ns + k] = t1; b.trace[2 * ns + k] = t2;
        b.flux[k] = water; b.flux[ns + k] = fx + pressure * nx; b.flux[2 * ns + k] = fy + pressure * ny;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Critical outlet (mode 4): on the controlled faces of an opening the
// outgoing characteristic discharge equals sqrt(g A^3 / B); faces turning
// inward or dry leave the control and the root is recomputed
// (river_exterior_outlet.h:29-175). Slot lists: `slots` null means the
// segment's own slots k0, k0+1, ...
// ---------------------------------------------------------------------------
__device__ __forceinline__ double resolved_bed(const MeshDev &m, const BoundaryDev &b, int k, const double *q,
                                               const double *z)
{
    const int c = m.owner[b.slot_face[k]];
    const double h = fmax(q[c], 0.), bed = b.ext_bed[k];
    if (h >= 1.e-3) return bed;
    const double bounded = fmax(bed, z[c] - h);
    double blend = fmin(1., fmax(0., (h - 1.e-4) / 9.e-4));
    blend = blend * blend * (3. - 2. * blend);
    return bed + (bounded - bed) * (1. - blend);
}

// Controlled discharge minus sqrt(g A^3 / B) at stage eta, the same in every
// thread; area, width out.
__device__ __noinline__ double crit_residual(SectionWork &w, const MeshDev &m, const BoundaryDev &b, const int *slots, int k0,
                                int n, double eta, double g, double dry, const double *q, const double *z, double &area,
                                double &width_)
{
    const int lanes = min(n, SECTION_LANES);
    for (int lane = threadIdx.x; lane < lanes; lane += blockDim.x) {
        double a = 0., width = 0., rate = 0.;
        for (int i = lane; i < n; i += SECTION_LANES) {
            const int k = slots ? slots[i] : k0 + i;
            if (b.branch[k] != 1) continue;
            const double h = fmax(eta - resolved_bed(m, b, k, q, z), 0.);
            if (h <= dry) continue;
            const double len = m.length[b.slot_face[k]];
            a += h * len; width += len; rate += h * (b.invariant[k] - 2. * sqrt(g * h)) * len;
        }
        w.part[0][lane] = a; w.part[1][lane] = width; w.part[2][lane] = rate;
    }
    double sum[3];
    lane_sums<3>(w, lanes, sum);
    area = sum[0]; width_ = sum[1];
    return sum[2] - (sum[1] > 0. ? sqrt(g * sum[0] * sum[0] * sum[0] / sum[1]) : 0.);
}

__device__ int crit_group(SectionWork &w, const MeshDev &m, const BoundaryDev &b, const int *slots, int k0, int n,
                          double g, double dry, double speed, const double *q, const double *z, bool &bad)
{
    const int nc = m.nc, nf = m.nf;
    const size_t ns = b.nslot;
    const double tol = 128. * EPS;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int k = slots ? slots[i] : k0 + i, f = b.slot_face[k], c = m.owner[f];
        b.branch[k] = 0; b.invariant[k] = 0.;
        const double h0 = q[c], h = fmax(h0 + z[c] - resolved_bed(m, b, k, q, z), 0.);
        if (h0 <= dry || h <= dry) continue;
        const double un = (q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[nf + f]) / h0, wave = sqrt(g * h);
        if (un < -tol * fmax(1., fabs(un))) continue;
        if (un > wave * (1. + 1e-10)) { b.branch[k] = 2; continue; }
        b.branch[k] = 1; b.invariant[k] = un + 2. * wave;
    }
    __syncthreads();
    int error = 0;
    bool done = false;
    double eta = 0., area = 0., width = 0.;
    const auto residual = [&](double at) { return crit_residual(w, m, b, slots, k0, n, at, g, dry, q, z, area, width); };
    for (int active = 0; active <= n && !done && !error; ++active) {
        double lo = INFINITY, hi = -INFINITY;
        bool some = false;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int k = slots ? slots[i] : k0 + i;
            if (b.branch[k] != 1) continue;
            const int c = m.owner[b.slot_face[k]];
            lo = fmin(lo, resolved_bed(m, b, k, q, z)); hi = fmax(hi, q[c] + z[c]);
            some = true;
        }
        if (!__syncthreads_or(some)) { done = true; break; }
        const int used = min(n, (int)blockDim.x);
        if ((int)threadIdx.x < used) { w.part[0][threadIdx.x] = lo; w.part[1][threadIdx.x] = hi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 0; i < used; ++i) { lo = fmin(lo, w.part[0][i]); hi = fmax(hi, w.part[1][i]); }
            w.sum[0] = lo; w.sum[1] = hi;
        }
        __syncthreads();
        lo = w.sum[0]; hi = w.sum[1];
        __syncthreads();
        lo += fmax(2. * dry, tol * fmax(1., fabs(lo)));
        const double rlo = residual(lo);
        if (rlo < 0.) {                            // unresolved controlled depth: the opening closes
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const int k = slots ? slots[i] : k0 + i;
                if (b.branch[k] == 1) b.branch[k] = 0;
            }
            eta = lo;
            done = true;
            break;
        }
        double rhi = residual(hi);
        for (int j = 0; j < 60 && rhi > 0.; ++j) { hi = lo + 2. * (hi - lo); rhi = residual(hi); }
        if (rhi > 0. || !isfinite(rhi)) { error = 1; break; }
        // several roots on an uneven bed: a face's discharge rises with the stage
        // before it falls, and the critical discharge drops where a face wets
        bisect_bracket(lo, hi, residual);
        eta = lo + .5 * (hi - lo);
        bool changed = false;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int k = slots ? slots[i] : k0 + i;
            if (b.branch[k] != 1) continue;
            const double h = fmax(eta - resolved_bed(m, b, k, q, z), 0.), un = b.invariant[k] - 2. * sqrt(g * h);
            if (h <= dry || un < -tol) { b.branch[k] = 0; changed = true; }
        }
        if (__syncthreads_or(changed)) continue;
        const double r = residual(eta), qc = width > 0. ? sqrt(g * area * area * area / width) : 0.;
        if (area <= 0. || width <= 0. || !isfinite(r) || fabs(r) > 1e-10 * fmax(qc, 1.)) error = 2;
        done = true;
    }
    if (!done && !error) error = 3;
    __syncthreads();
    if (error) return error;                 // the same in every thread
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int k = slots ? slots[i] : k0 + i, f = b.slot_face[k], c = m.owner[f];
        const double rbed = resolved_bed(m, b, k, q, z), h0 = q[c], geom = fmax(h0 + z[c] - rbed, 0.);
        const double nx = m.normal[f], ny = m.normal[nf + f];
        double h = geom, ux = 0., uy = 0.;
        if (h0 > dry) { ux = q[nc + c] / h0; uy = q[2 * nc + c] / h0; } else h = 0.;
        double un = ux * nx + uy * ny;
        const double tx = ux - un * nx, ty = uy - un * ny;
        if (b.branch[k] == 0) un = 0.;
        else if (b.branch[k] == 1) { h = fmax(eta - rbed, 0.); un = b.invariant[k] - 2. * sqrt(g * h); }
        if (!isfinite(h) || !isfinite(un) || sqrt(un * un + tx * tx + ty * ty) > speed) { bad = true; continue; }
        double water = 0., fx = 0., fy = 0., t0 = 0., t1 = 0., t2 = 0.;
        if (h > dry) {
            t0 = h; t1 = h * (un * nx + tx); t2 = h * (un * ny + ty);
            water = t1 * nx + t2 * ny;
            fx = water * t1 / h + .5 * g * h * h * nx;
            fy = water * t2 / h + .5 * g * h * h * ny;
        }
        const double pressure = h0 > dry ? .5 * g * (h0 * h0 - geom * geom) : 0.;
        b.trace[k] = t0; b.trace[ns + k] = t1; b.trace[2 * ns + k] = t2;
        b.flux[k] = water; b.flux[ns + k] = fx + pressure * nx; b.flux[2 * ns + k] = fy + pressure * ny;
    }
    return 0;
}

// The critical owner of segment sg: the whole opening, then, when dry faces
// split its chains into several wet groups, each group alone with the dry
// faces closed at their owners' pressure (river_exterior_outlet.py:37-72).
__device__ __noinline__ int crit_section(SectionWork &w, const MeshDev &m, const BoundaryDev &b, int sg, double g, double dry,
                            double speed, const double *q, const double *z, bool &bad)
{
    const int nf = m.nf, k0 = b.seg_off[sg], n = b.seg_off[sg + 1] - k0;
    const size_t ns = b.nslot;
    bool bad_whole = false;
    const int err = crit_group(w, m, b, nullptr, k0, n, g, dry, speed, q, z, bad_whole);
    if (!b.crit_seg_chain) { bad = bad || bad_whole; return err; }
    __shared__ int ngroup;
    if (threadIdx.x == 0) {          // wet runs along each chain, as slot lists in the segment's scratch
        int groups = 0, flat = 0;
        for (int ch = b.crit_seg_chain[sg]; ch < b.crit_seg_chain[sg + 1]; ++ch) {
            bool open = false;
            for (int e = b.crit_chain_off[ch]; e < b.crit_chain_off[ch + 1]; ++e) {
                const int k = b.crit_chain_slot[e], c = m.owner[b.slot_face[k]];
                const double h = q[c], geom = h + z[c] - b.ext_bed[k];
                if ((h > dry) && (geom > dry)) { b.gslot[k0 + flat++] = k; open = true; }
                else if (open) { b.gend[k0 + groups++] = flat; open = false; }
            }
            if (open) b.gend[k0 + groups++] = flat;
        }
        ngroup = groups;
    }
    __syncthreads();
    const int groups = ngroup;
    __syncthreads();
    if (groups <= 1) { bad = bad || bad_whole; return err; }
    int worst = 0, start = 0;
    bool bad_groups = bad_whole;      // a face the groups do not rewrite keeps its earlier status
    for (int gi = 0; gi < groups; ++gi) {
        const int end = b.gend[k0 + gi];
        bool gb = false;
        const int e = crit_group(w, m, b, b.gslot + k0 + start, 0, end - start, g, dry, speed, q, z, gb);
        worst = max(worst, e);
        bad_groups = bad_groups || gb;
        start = end;
    }
    // dry chain faces close at their owners' pressure; their status clears
    bool any_dry_bad = false;
    for (int ch = b.crit_seg_chain[sg]; ch < b.crit_seg_chain[sg + 1]; ++ch)
        for (int e = b.crit_chain_off[ch] + threadIdx.x; e < b.crit_chain_off[ch + 1]; e += blockDim.x) {
            const int k = b.crit_chain_slot[e], f = b.slot_face[k], c = m.owner[f];
            const double h = q[c], geom = h + z[c] - b.ext_bed[k];
            if ((h > dry) && (geom > dry)) continue;
            const double height = fmax(q[c], 0.), pressure = .5 * g * height * height;
            b.trace[k] = 0.; b.trace[ns + k] = 0.; b.trace[2 * ns + k] = 0.;
            b.flux[k] = 0.; b.flux[ns + k] = pressure * m.normal[f]; b.flux[2 * ns + k] = pressure * m.normal[nf + f];
        }
    (void)any_dry_bad;
    __syncthreads();
    bad = bad || bad_groups;
    return worst;
}

// ---------------------------------------------------------------------------
// Exact-discharge inlet (mode 9, river_exterior_inlet.h): the exact 1-D SWE
// Riemann solution between a virtual reservoir at the requested water line
// and each face's interior state; the reservoir's common normal velocity is
// solved (bracket, then safeguarded Newton with the analytical derivative)
// so that the net section discharge equals the request.
// ---------------------------------------------------------------------------
struct InletRiemann {
    double h, u, derivative;
    int iterations, error;
};

// Jump across the wave between h and the state of depth hk, and its
// derivative; ck = sqrt(g hk), rk = 1 / hk, rh = 1 / h.
__device__ __forceinline__ void inlet_wave(double h, double rh, double hk, double ck, double rk, double g, double &f,
                                           double &df)
{
    if (greater(h, hk)) {
        const double a = sqrt(.5 * g * (rh + rk)), den = a * h * h;
        f = (h - hk) * a;
        df = a - quotient(.25 * g * (h - hk), den, reciprocal(den));
    } else {
        f = 2. * (sqrt(g * h) - ck);
        df = sqrt(quotient(g, h, rh));
    }
}

// river_exterior_inlet.h:32-69: left = reservoir, right = interior (normal into the domain)
__device__ __noinline__ InletRiemann inlet_exact(double hl, double ul, double hr, double ur, double g)
{
    InletRiemann r = {0., 0., 0., 0, 0};
    const double cl = sqrt(g * hl), cr = sqrt(g * hr);
    if (hl == 0. && hr == 0.) return r;
    if (hr == 0. || hl == 0. || ur - ul >= 2. * (cl + cr)) {
        if (hl > 0. && ul - cl >= 0.) { r.h = hl; r.u = ul; r.derivative = hl; }
        else if (hl > 0. && ul + 2. * cl > 0.) { r.u = (ul + 2. * cl) / 3.; r.h = r.u * r.u / g; r.derivative = r.h; }
        else if (hr > 0. && ur + cr <= 0.) { r.h = hr; r.u = ur; }
        else if (hr > 0. && ur - 2. * cr < 0.) { r.u = (ur - 2. * cr) / 3.; r.h = r.u * r.u / g; }
        return r;
    }
    double guess = .5 * (cl + cr) - .25 * (ur - ul);
    guess = guess * guess / g;
    const double rl = quotient(1., hl, reciprocal(hl)), rr = quotient(1., hr, reciprocal(hr));
    double lo = 0., hi = fmax(fmax(hl, hr), guess), fl, fr, dl, dr;
    const auto waves = [&](double h) {
        const double rh = quotient(1., h, reciprocal(h));
        inlet_wave(h, rh, hl, cl, rl, g, fl, dl);
        inlet_wave(h, rh, hr, cr, rr, g, fr, dr);
    };
    waves(hi);
    for (int j = 0; j < 60 && fl + fr + ur - ul < 0.; ++j) { hi *= 2.; waves(hi); }
    if (!isfinite(hi) || fl + fr + ur - ul < 0.) { r.error = 1; return r; }
    const double scale = fmax(1., cl + cr + fabs(ul) + fabs(ur));
    double h = fmax(fmin(guess, hi), 1e-30), residual = 0.;
    for (int j = 0; j < 70; ++j) {
        waves(h);
        residual = fl + fr + ur - ul;
        r.iterations = j + 1;
        if (fabs(residual) <= 4e-14 * scale) break;
        if (residual < 0.) lo = h; else hi = h;
        const double slope = dl + dr;
        double next = h - quotient(residual, slope, reciprocal(slope));
        if (!(next > lo && next < hi)) next = lo + .5 * (hi - lo);
        h = next;
    }
    if (fabs(residual) > 4e-14 * scale) waves(h);
    residual = fl + fr + ur - ul;
    if (!isfinite(h) || fabs(residual) > 2e-11 * scale) { r.error = 2; return r; }
    const double u = .5 * (ul + ur + fr - fl), c = sqrt(g * h);
    r.h = h; r.u = u; r.derivative = fmax(0., (u + h * dr) / (dl + dr));
    if (u >= 0.) {
        if (h > hl) {
            if (ul - sqrt(.5 * g * h * (h + hl) / hl) >= 0.) { r.h = hl; r.u = ul; r.derivative = hl; }
        } else if (ul - cl >= 0.) { r.h = hl; r.u = ul; r.derivative = hl; }
        else if (u - c > 0.) { r.u = (ul + 2. * cl) / 3.; r.h = r.u * r.u / g; r.derivative = r.h; }
    } else {
        if (h > hr) {
            if (ur + sqrt(.5 * g * h * (h + hr) / hr) <= 0.) { r.h = hr; r.u = ur; r.derivative = 0.; }
        } else if (ur + cr <= 0.) { r.h = hr; r.u = ur; r.derivative = 0.; }
        else if (u + c < 0.) { r.u = (ur - 2. * cr) / 3.; r.h = r.u * r.u / g; r.derivative = 0.; }
    }
    return r;
}

// Interior depth above the face's exterior bed and inward normal speed of slot k.
__device__ __forceinline__ void inlet_interior(const MeshDev &m, const BoundaryDev &b, int k, double dry,
                                               const double *q, const double *z, double &hi, double &ui)
{
    const int nc = m.nc, f = b.slot_face[k], c = m.owner[f];
    const double h0 = q[c];
    hi = h0 > dry ? fmax(h0 + z[c] - b.ext_bed[k], 0.) : 0.;
    if (hi <= dry) hi = 0.;
    ui = h0 > dry ? -(q[nc + c] * m.normal[f] + q[2 * nc + c] * m.normal[m.nf + f]) / h0 : 0.;
}

// river_exterior_inlet.h:71-95: section discharge, its derivative and the
// gross throughflow at the common velocity (lane sums, lane order), the same
// in every thread; returns whether a face's Riemann solution failed.
__device__ __noinline__ bool inlet_rate(SectionWork &w, const MeshDev &m, const BoundaryDev &b, int k0, int k1, double requested,
                           double velocity, double g, double dry, const double *q, const double *z, double &rate,
                           double &derivative, double &gross)
{
    const int n = min(k1 - k0, SECTION_LANES);
    bool failed = false;
    for (int lane = threadIdx.x; lane < n; lane += blockDim.x) {
        double sum = 0., slope = 0., through = 0.;
        for (int k = k0 + lane; k < k1; k += SECTION_LANES) {
            double hi, ui;
            inlet_interior(m, b, k, dry, q, z, hi, ui);
            double hr = fmax(requested - b.ext_bed[k], 0.);
            if (hr <= dry) hr = 0.;
            const InletRiemann r = inlet_exact(hr, velocity, hi, ui, g);
            const double len = m.length[b.slot_face[k]];
            sum += r.h * r.u * len; slope += r.derivative * len;
            through += fabs(r.h * r.u * len);
            failed = failed || r.error;
        }
        w.part[0][lane] = sum; w.part[1][lane] = slope; w.part[2][lane] = through;
    }
    double sums[3];
    lane_sums<3>(w, n, sums);
    rate = sums[0]; derivative = sums[1]; gross = sums[2];
    return __syncthreads_or(failed);
}

// river_exterior_inlet.h:97-186: the inlet of segment sg. Returns 0 or the
// section failure (a trial rejection in the reference); `bad` gets the faces
// whose Riemann solution failed or exceeds the speed limit (face status 3).
__device__ __noinline__ int inlet_section(SectionWork &w, const MeshDev &m, const BoundaryDev &b, int sg, double g, double dry,
                             double speed, const double *q, const double *z, bool &bad)
{
    const int nc = m.nc, nf = m.nf, nseg = b.nseg, k0 = b.seg_off[sg], k1 = b.seg_off[sg + 1];
    const size_t ns = b.nslot;
    const double Q = b.forcing[sg], requested = b.forcing[nseg + sg];
    const int n = min(k1 - k0, SECTION_LANES);
    for (int lane = threadIdx.x; lane < n; lane += blockDim.x) {
        double area = 0., scale = 1.;
        for (int k = k0 + lane; k < k1; k += SECTION_LANES) {
            double hi, ui;
            inlet_interior(m, b, k, dry, q, z, hi, ui);
            const double hr = fmax(requested - b.ext_bed[k], 0.);
            if (hr > dry) area += hr * m.length[b.slot_face[k]];
            scale = fmax(scale, fabs(ui) + 2. * sqrt(g * hi) + 2. * sqrt(g * hr));
        }
        w.part[0][lane] = area; w.part[1][lane] = scale;
    }
    double sums[1];
    lane_sums<1>(w, n, sums);
    double scale = 1.;
    for (int lane = 0; lane < n; ++lane) scale = fmax(scale, w.part[1][lane]);
    __syncthreads();
    const double area = sums[0];
    int error = 0;
    if (!isfinite(Q) || Q < 0. || !isfinite(requested) || (Q > 0. && area <= 0.)) error = 1;
    double velocity = area > 0. ? Q / area : 0.;
    scale = fmax(scale, 1. + fabs(velocity));
    if (Q > 0. && !error) {
        double lo = velocity - scale, hi = velocity + scale, rate, derivative, gross;
        const auto eval = [&](double at) {
            velocity = at;
            if (inlet_rate(w, m, b, k0, k1, requested, at, g, dry, q, z, rate, derivative, gross)) error = 5;
        };
        eval(lo);
        for (int j = 0; j < 60 && rate > Q && !error; ++j) { lo -= scale; scale *= 2.; eval(lo); }
        if (rate > Q) error = 2;
        eval(hi);
        for (int j = 0; j < 60 && rate < Q && !error; ++j) { hi += scale; scale *= 2.; eval(hi); }
        if (rate < Q) error = 2;
        double at = fmin(hi, fmax(lo, Q / area));
        for (int j = 0; j < 80 && !error; ++j) {
            eval(at);
            // net Q may be far below the signed face throughflow: relative
            // tolerance plus a double-precision budget on the gross flow
            if (fabs(rate - Q) <= 3e-13 * Q + 256. * EPS * gross) break;
            if (rate < Q) lo = at; else hi = at;
            double next = derivative > 0. ? at + (Q - rate) / derivative : lo + .5 * (hi - lo);
            if (!(next > lo && next < hi)) next = lo + .5 * (hi - lo);
            at = next;
        }
        if (velocity != at) eval(at);                // the loop ran out: its last point
        velocity = at;
        if (!isfinite(rate) || fabs(rate - Q) > 1e-10 * Q + 1024. * EPS * gross) error = 3;
    }
    if (error) return error;                         // the same in every thread
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int f = b.slot_face[k], c = m.owner[f];
        const double nx = m.normal[f], ny = m.normal[nf + f], h0 = q[c];
        double hi, ui;
        inlet_interior(m, b, k, dry, q, z, hi, ui);
        const double vt = h0 > dry ? (-q[nc + c] * ny + q[2 * nc + c] * nx) / h0 : 0.;
        double hr = fmax(requested - b.ext_bed[k], 0.);
        if (hr <= dry) hr = 0.;
        InletRiemann r = Q == 0. ? inlet_exact(h0, -ui, h0, ui, g) : inlet_exact(hr, velocity, hi, ui, g);
        if (Q == 0.) r.u = 0.;
        if (r.error || !isfinite(r.h) || !isfinite(r.u) || fabs(r.u) > speed) { bad = true; continue; }
        const double water = -r.h * r.u, tangent = r.u < 0. ? vt : 0.;
        b.trace[k] = r.h; b.trace[ns + k] = water * nx - r.h * tangent * ny; b.trace[2 * ns + k] = water * ny + r.h * tangent * nx;
        const double pressure = Q == 0. ? 0. : .5 * g * (h0 * h0 - hi * hi);
        const double momentum = r.h * r.u * r.u + .5 * g * r.h * r.h + pressure;
        b.flux[k] = water;
        b.flux[ns + k] = momentum * nx - water * tangent * ny;
        b.flux[2 * ns + k] = momentum * ny + water * tangent * nx;
    }
    __syncthreads();
    return 0;
}

// ---------------------------------------------------------------------------
// Reference water lines of the exact-discharge inlets, written into the
// forcing stage before the exterior flux: 1 critical depth
// (river_exterior_section.h:17-74), 2 normal depth
// (river_exterior_normal.h:18-104). Every distinct bed level of the section
// starts one constant-wet-width branch (a candidate); 128 lanes take the
// candidates and thread 0 reduces the lanes to the lexicographic minimum of
// (rank, stage), which does not depend on the order. A solved line is kept
// per segment with its discharge and reused while the discharge is equal
// (the inputs besides it are fixed; the host clears the cache when it
// changes them), as the reference's SectionCache.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void line_pick(double rank, double cand, double &best, double &stage)
{
    if (rank < best || (rank == best && cand < stage)) { best = rank; stage = cand; }
}

__device__ void line_critical_candidate(const MeshDev &m, const BoundaryDev &b, int i, int k0, int k1, double Q,
                                        double g, double dry, double &rank, double &cand)
{
    const double level = b.ext_bed[i];
    double minimum = level, next = INFINITY, width = 0., excess = 0.;
    for (int k = k0; k < k1; ++k) {
        const double zb = b.ext_bed[k], len = m.length[b.slot_face[k]];
        minimum = fmin(minimum, zb);
        if (zb > level) next = fmin(next, zb);
        else { width += len; excess += (level - zb) * len; }
    }
    rank = INFINITY; cand = 0.;
    if (Q == 0.) { cand = minimum; rank = 0.; return; }
    const double area = cbrt(Q * Q * width / g), eta = level + (area - excess) / width;
    if (!(isfinite(area) && area > 0. && isfinite(eta) && eta > level + dry) || eta > next + dry) return;
    double actual = 0., wet_width = 0.;
    for (int k = k0; k < k1; ++k) {
        const double h = eta - b.ext_bed[k], len = m.length[b.slot_face[k]];
        if (h > dry) { actual += h * len; wet_width += len; }
    }
    if (wet_width != width || !(actual > 0.)) return;
    const double residual = fabs(Q * Q * wet_width / (g * actual * actual * actual) - 1.);
    const double tolerance = 1e-10 + 64. * EPS * fmax(1., fabs(eta)) * width / actual;
    if (residual > tolerance) return;
    cand = eta;
    rank = eta - minimum + Q * Q / (2. * g * actual * actual);
}

// wetted perimeter of slot k: its length plus the wetted steps to its neighbours
__device__ __forceinline__ double line_perimeter(const MeshDev &m, const BoundaryDev &b, int k, double eta, double dry)
{
    const double h = eta - b.ext_bed[k];
    if (h <= dry) return 0.;
    const int l = b.line_left[k], r = b.line_right[k];
    double hl = l < 0 ? 0. : fmax(eta - b.ext_bed[l], 0.), hr = r < 0 ? 0. : fmax(eta - b.ext_bed[r], 0.);
    if (hl <= dry) hl = 0.;
    if (hr <= dry) hr = 0.;
    return m.length[b.slot_face[k]] + fmax(h - hl, 0.) + fmax(h - hr, 0.);
}

__device__ double line_rate(const MeshDev &m, const BoundaryDev &b, int k0, int k1, double eta, double slope,
                            double g, double dry, int law, double rough)
{
    double area = 0., perimeter = 0., drag = 0.;
    for (int k = k0; k < k1; ++k) {
        const double h = eta - b.ext_bed[k];
        if (h > dry) { area += h * m.length[b.slot_face[k]]; perimeter += line_perimeter(m, b, k, eta, dry); }
    }
    if (!(area > 0. && perimeter > 0.)) return 0.;
    const double c = nout_chezy(law, fmax(area / perimeter, dry), rough, g);
    for (int k = k0; k < k1; ++k)
        if (eta - b.ext_bed[k] > dry) drag += line_perimeter(m, b, k, eta, dry) / (c * c);
    return drag > 0. ? area * sqrt(area * slope / drag) : 0.;
}

__device__ void line_normal_candidate(const MeshDev &m, const BoundaryDev &b, int i, int k0, int k1, double Q,
                                      double slope, double g, double dry, int law, double rough, double &rank,
                                      double &cand)
{
    rank = INFINITY; cand = 0.;
    const double level = b.ext_bed[i];
    const int fi = b.slot_face[i];
    double minimum = level, next = INFINITY;
    for (int k = k0; k < k1; ++k) {
        const double zb = b.ext_bed[k];
        minimum = fmin(minimum, zb);
        if (zb > level) next = fmin(next, zb);
        if (zb == level && b.slot_face[k] < fi) return;          // one candidate per distinct level
    }
    if (Q == 0.) { cand = rank = minimum; return; }
    const double epsilon = 8. * EPS * fmax(1., fabs(level));
    double lo = level + dry + epsilon, hi = isfinite(next) ? next + dry : level + fmax(1., 64. * dry);
    if (!(hi > lo)) return;
    double rlo = line_rate(m, b, k0, k1, lo, slope, g, dry, law, rough) - Q;
    double rhi = line_rate(m, b, k0, k1, hi, slope, g, dry, law, rough) - Q;
    if (!isfinite(next))
        for (int k = 0; k < 60 && rhi < 0.; ++k) {
            hi = level + 2. * (hi - level);
            rhi = line_rate(m, b, k0, k1, hi, slope, g, dry, law, rough) - Q;
        }
    if (!isfinite(rlo) || !isfinite(rhi)) return;
    const double start = lo, end = hi;
    double previous = rlo;
    bool found = false;
    for (int j = 1; j <= 32; ++j) {          // sub-brackets: the lowest sign change of the branch
        const double at = start + (end - start) * (double(j) / 32.);
        const double value = j == 32 ? rhi : line_rate(m, b, k0, k1, at, slope, g, dry, law, rough) - Q;
        if (isfinite(value) && ((previous <= 0. && value >= 0.) || (previous >= 0. && value <= 0.))) {
            hi = at; rhi = value; rlo = previous; found = true;
            break;
        }
        lo = at; previous = value;
    }
    if (!found) return;
    for (int j = 0; j < 80; ++j) {
        const double mid = lo + .5 * (hi - lo);
        if (mid == lo || mid == hi) break;
        const double value = line_rate(m, b, k0, k1, mid, slope, g, dry, law, rough) - Q;
        if ((rlo <= 0. && value >= 0.) || (rlo >= 0. && value <= 0.)) { hi = mid; rhi = value; }
        else { lo = mid; rlo = value; }
    }
    const double eta = fabs(rlo) < fabs(rhi) ? lo : hi;
    const double rate = line_rate(m, b, k0, k1, eta, slope, g, dry, law, rough);
    const double tolerance = 1e-10 + 128. * EPS * fmax(1., fabs(eta)) / fmax(eta - minimum, dry);
    if (isfinite(rate) && fabs(rate / Q - 1.) <= tolerance) { cand = eta; rank = eta; }
}

// The line of segment sg (block-cooperative); false when the section has no
// resolved root (the reference rejects the trial).
__device__ __noinline__ bool line_section(SectionWork &w, const MeshDev &m, const BoundaryDev &b, int sg, double g, double dry,
                             int law, double rough)
{
    const int k0 = b.seg_off[sg], k1 = b.seg_off[sg + 1], kind = b.line_kind[sg];
    const double Q = b.forcing[sg];
    const bool cached = b.line_q[sg] == Q;
    __syncthreads();
    if (cached) {
        if (threadIdx.x == 0) b.forcing[b.nseg + sg] = b.line_stage[sg];
        __syncthreads();
        return true;
    }
    for (int lane = threadIdx.x; lane < SECTION_LANES; lane += blockDim.x) {
        double best = INFINITY, stage = 0.;
        for (int i = k0 + lane; i < k1; i += SECTION_LANES) {
            double rank, cand;
            if (kind == 1) line_critical_candidate(m, b, i, k0, k1, Q, g, dry, rank, cand);
            else line_normal_candidate(m, b, i, k0, k1, Q, b.line_slope[sg], g, dry, law, rough, rank, cand);
            line_pick(rank, cand, best, stage);
        }
        w.part[0][lane] = best; w.part[1][lane] = stage;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double best = INFINITY, stage = 0.;
        for (int lane = 0; lane < SECTION_LANES; ++lane) line_pick(w.part[0][lane], w.part[1][lane], best, stage);
        w.error = !isfinite(best);
        if (!w.error) {
            b.forcing[b.nseg + sg] = stage;
            b.line_q[sg] = Q;
            b.line_stage[sg] = stage;
        }
    }
    __syncthreads();
    const bool ok = !w.error;
    __syncthreads();
    return ok;
}

// Exact-discharge inlet allocation of one scenario (boundary CTA, after the outlet cap).
__device__ void inlet_allocation(const MeshDev &m, const BoundaryDev &b, const Ctrl &ct, const double *base, int s0,
                                 int s1, int u0, int u1)
{
    // exact-discharge inlet allocation (inlet_feasibility.py:34-57): each
    // owner's outward inlet debit capped by its stock after its other
    // boundary debits (owner factor kept per slot in terms), then per inlet
    // segment the removed outflow taken from its incoming faces; sums in
    // boundary order, as the reference's bincounts
    __syncthreads();
    const size_t ns = b.nslot;
    for (int u = u0 + threadIdx.x; u < u1; u += blockDim.x) {
        const int c = b.own_cell[u];
        double total = 0., reserved = 0.;
        for (int j = b.own_off[u]; j < b.own_off[u + 1]; ++j) {
            const int k = b.own_slot[j], f = b.slot_face[k];
            const double rate = fmax(b.flux[k], 0.) * m.length[f];
            if (b.seg_mode[m.bid[f]] == 9) total += rate; else reserved += rate;
        }
        const double available = fmax(0., base[c] * m.area[c] / ct.trial - reserved);
        const double ratio = fmin(1., available / fmax(total, 1e-300)) * (1. - 32. * EPS);
        const double factor = total > available ? ratio : 1.;
        for (int j = b.own_off[u]; j < b.own_off[u + 1]; ++j) b.terms[b.own_slot[j]] = factor;
    }
    __syncthreads();
    for (int sg = s0 + threadIdx.x; sg < s1; sg += blockDim.x) {
        if (b.seg_mode[sg] != 9) continue;
        double removed = 0., incoming = 0.;
        for (int k = b.seg_off[sg]; k < b.seg_off[sg + 1]; ++k) {
            const double water = b.flux[k], len = m.length[b.slot_face[k]];
            removed += water > 0. ? fmax(water, 0.) * len * (1. - b.terms[k]) : 0.;
            incoming += fmax(-water, 0.) * len;
        }
        const bool feasible = removed <= incoming;
        const double in_scale = incoming > 0. ? 1. - removed / fmax(incoming, 1e-300) : 1.;
        for (int k = b.seg_off[sg]; k < b.seg_off[sg + 1]; ++k) {
            const double water = b.flux[k];
            const double scale = (feasible && water > 0.) ? b.terms[k] : ((feasible && water < 0.) ? in_scale : 1.);
            const double depth = b.trace[k], denom = fmax(depth, 1e-300);
            const double ux = depth > 0. ? b.trace[ns + k] / denom : 0.;
            const double uy = depth > 0. ? b.trace[2 * ns + k] / denom : 0.;
            b.flux[ns + k] += (scale * scale - 1.) * water * ux;
            b.flux[2 * ns + k] += (scale * scale - 1.) * water * uy;
            b.flux[k] = water * scale;
            b.trace[ns + k] *= scale;
            b.trace[2 * ns + k] *= scale;
        }
    }
}

// stage 1 / 2: the SSPRK stages (state work / q1, its own stock, clock t or
// t + dt); STAGE_HANCOCK: the HLLC predicted state q1 at t + dt/2, outlet
// stock of the substep's start state work (hllc.py:91-97), status of stage 1.
constexpr int STAGE_HANCOCK = 3;

// One open face: its ids, geometry and its owner's state.
struct OpenFace {
    int f, c, sg, mode;
    double h, hu, hv, z, bed, nx, ny, len;
};

__device__ __forceinline__ OpenFace open_face(const MeshDev &m, const BoundaryDev &b, int k, int sg, const double *q,
                                              const double *z)
{
    OpenFace o;
    o.f = b.slot_face[k]; o.c = m.owner[o.f]; o.sg = sg; o.mode = b.seg_mode[sg];
    o.h = q[o.c]; o.hu = q[m.nc + o.c]; o.hv = q[2 * m.nc + o.c]; o.z = z[o.c];
    o.bed = b.ext_bed[k]; o.nx = m.normal[o.f]; o.ny = m.normal[m.nf + o.f]; o.len = m.length[o.f];
    return o;
}

// Forcing table row (0 discharge, 1 stage) of segment sg at time t:
// piecewise linear, the end values outside.
__device__ __forceinline__ double table_forcing(const BoundaryDev &b, int row, int sg, double t)
{
    const int L = b.table_len;
    const double *y = b.table_value + ((size_t)row * b.nseg + sg) * L;
    if (t <= b.table_time[0]) return y[0];
    if (t >= b.table_time[L - 1]) return y[L - 1];
    // last knot at or before t, capped at L - 2; (1 - w) y_i + w y_{i+1}
    // (RiverHydraulicSchedule.sample, river_hydraulic_schedule.py:57-65)
    int i = 0;
    while (i < L - 2 && b.table_time[i + 1] <= t) ++i;
    const double w = (t - b.table_time[i]) / (b.table_time[i + 1] - b.table_time[i]);
    return (1. - w) * y[i] + w * y[i + 1];
}

// Conveyance weight of an inlet face under its segment's mean wetted stage.
template <class F>
__device__ __forceinline__ double face_weight(const Ctrl &ct, const OpenFace &o, double stage_sum, double width)
{
    if (!(width > 0.)) return 0.;
    const double h = o.h + o.z - o.bed, depth = stage_sum / width - o.bed;
    if (!greater(h, ct.dry) || !greater(depth, 0.)) return 0.;
    const int rmode = ct.roughness_mode < 3 ? ct.roughness_mode : 3;
    return conveyance<F>(rmode, ct.roughness_mode == 4, F(depth), F(h), ct) * o.len;
}

// Exterior trace and flux of a face on a segment of mode 2, 3 or 6 with
// discharge Q or stage level (river_exterior_bed.h:94-174); returns the face
// status. total: the segment's conveyance, w: the face's.
__device__ __forceinline__ int plain_face(const OpenFace &o, double Q, double level, int policy, double dry, double grav,
                                          double speed_limit, double total, double w, double tr[3], double fl[3])
{
    const double nx = o.nx, ny = o.ny, bed = o.bed;
    double h = o.h + o.z - bed, ux = 0., uy = 0.;
    if (!greater(h, 0.)) h = 0.;
    const double geometric = h;
    const bool wet0 = greater(o.h, dry);
    if (wet0) {
        const double r = reciprocal(o.h);
        ux = quotient(o.hu, o.h, r); uy = quotient(o.hv, o.h, r);
    }
    const double un = ux * nx + uy * ny;
    double tx = ux - un * nx, ty = uy - un * ny, speed = 0.;
    if (o.mode == 6) {
        if (Q > 0. && total <= 0.) return 1;
        if (greater(h, dry) && Q > 0.) {
            const double den = total * h * o.len;
            speed = quotient(-Q * w, den, reciprocal(den));
        }
    } else if (o.mode == 3) {
        if (!wet0) h = 0.;
        else if (greater(h, dry)) {
            if (un < sqrt(grav * h)) return 6;
            speed = un;
        }
    } else if (o.mode == 2) {
        const double target = greater(level - bed, 0.) ? level - bed : 0.;
        if (policy && (!wet0 || !greater(h, dry)) && greater(target, dry)) return 4;
        if (!wet0) h = 0.;
        if (greater(h, dry)) {
            const double wave = sqrt(grav * h);
            if (un <= -wave) {
                if (policy) return 5;
                tx = ty = 0.;
            } else {
                double hb, ub;
                stage_wave(h, un, target, grav, wave, hb, ub);
                if (ub < 0. && policy) {
                    if (ub <= -sqrt(grav * hb)) return 5;
                    h = hb; speed = ub; tx = ty = 0.;
                } else if (ub < 0.) tx = ty = 0.;
                else { h = hb; speed = ub; }
            }
        }
    } else return 2;
    if (!finite_bits(h) || !finite_bits(speed) || greater(0., h)) return 3;
    // sqrt(s2) > limit, with the square root only where the squares are near
    const double s2 = speed * speed + tx * tx + ty * ty;
    if (!greater(speed_limit * speed_limit * .999999, s2) && sqrt(s2) > speed_limit) return 3;
    double water = 0., fx = 0., fy = 0.;
    if (greater(h, dry)) {
        const double r = reciprocal(h);
        tr[0] = h;
        tr[1] = h * (speed * nx + tx);
        tr[2] = h * (speed * ny + ty);
        water = tr[1] * nx + tr[2] * ny;
        fx = quotient(water * tr[1], h, r) + .5 * grav * h * h * nx;
        fy = quotient(water * tr[2], h, r) + .5 * grav * h * h * ny;
    }
    const double pressure = wet0 ? .5 * grav * (o.h * o.h - geometric * geometric) : 0.;
    fl[0] = water; fl[1] = fx + pressure * nx; fl[2] = fy + pressure * ny;
    return 0;
}

// Outlet faces' share of an owner's stock: total and reserved outward rates
// against base area / trial; returns 1 where nothing is to be capped.
__device__ __forceinline__ double cap_factor(double base, double area, double trial, double rtrial, double total,
                                             double reserved)
{
    const double left = quotient(base * area, trial, rtrial) - reserved;
    const double available = greater(left, 0.) ? left : 0.;
    if (!greater(total, available)) return 1.;
    return fmin(1., available / fmax(total, 1e-300)) * (1. - 32. * EPS);
}

// Trace and flux of an outlet face capped by the owner's factor.
__device__ __forceinline__ void cap_face(double factor, double tr[3], double fl[3])
{
    const double water = fl[0], depth = tr[0], denom = fmax(depth, 1e-300);
    const double ux = depth > 0. ? tr[1] / denom : 0., uy = depth > 0. ? tr[2] / denom : 0.;
    fl[1] += (factor * factor - 1.) * water * ux;
    fl[2] += (factor * factor - 1.) * water * uy;
    fl[0] = water * factor;
    tr[1] *= factor;
    tr[2] *= factor;
}

// The cap of every owner from u0 + first on, in steps (an owner's faces in boundary order).
__device__ __forceinline__ void cap_owners(const MeshDev &m, const BoundaryDev &b, const double *base, double trial,
                                           int first, int u1, int step, bool several)
{
    const size_t ns = b.nslot;
    const double rtrial = reciprocal(trial);
    for (int u = first; u < u1; u += step) {
        const int j0 = b.own_off[u], j1 = b.own_off[u + 1], c = b.own_cell[u];
        if (several && j1 - j0 < 2) continue;
        double total = 0., reserved = 0.;
        for (int j = j0; j < j1; ++j) {
            const int k = b.own_slot[j], f = b.slot_face[k];
            const double flux = b.flux[k], debit = greater(flux, 0.) ? flux * m.length[f] : 0.;
            if (is_outlet(b.seg_mode[m.bid[f]])) total += debit; else reserved += debit;
        }
        const double factor = cap_factor(base[c], m.area[c], trial, rtrial, total, reserved);
        if (factor == 1.) continue;
        for (int j = j0; j < j1; ++j) {
            const int k = b.own_slot[j];
            double tr[3] = {b.trace[k], b.trace[ns + k], b.trace[2 * ns + k]};
            double fl[3] = {b.flux[k], b.flux[ns + k], b.flux[2 * ns + k]};
            if (!is_outlet(b.seg_mode[m.bid[b.slot_face[k]]]) || !(fl[0] > 0.)) continue;
            cap_face(factor, tr, fl);
#pragma unroll
            for (int r = 0; r < 3; ++r) { b.trace[r * ns + k] = tr[r]; b.flux[r * ns + k] = fl[r]; }
        }
    }
}

// Water and gross water of 32 faces by a butterfly; the result in every lane.
__device__ __forceinline__ double2 warp_water(double v)
{
    double2 a = make_double2(v, fabs(v));
    for (int o = 16; o > 0; o >>= 1) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    }
    return a;
}

// The scenario's sum over its open faces of (outward water flux x length),
// with each face's water as the update consumes it (the mixed form carries it
// in FP32), and of its magnitude, from the sums of 32 faces in slot order. The
// controller turns the stage sums into the boundary ledger. Threads 0 and 1.
__device__ __forceinline__ void scenario_water(const BoundaryDev &b, Ctrl &ct, int stage, int s0, int ntile)
{
    if (threadIdx.x >= 2) return;
    double total = 0.;
    for (int i = 0; i < ntile; ++i) {
        const SlotTile tile = slot_tile(b, s0, i);
        for (int k = tile.first; k < tile.end; k += 32) total += threadIdx.x ? b.water_sum[k].y : b.water_sum[k].x;
    }
    if (threadIdx.x) ct.bgross[stage - 1] = total; else ct.bflux[stage - 1] = total;
}

// The open boundary of one scenario whose segments have modes 2, 3 and 6 and
// at most 64 faces x 2 x cluster size: a thread per face, a thread-block
// cluster per scenario. What bounds it: short FP64 phases (a warp's FP64
// instruction takes 65 clocks, so a block has one warp per sub-partition and
// wide openings more blocks) between dependent loads; each face's data is
// loaded once, at the start. The sums keep the reference's fixed tree (64-face
// tiles, then the tiles in order), so no result depends on the cluster's size.
template <class F>
__global__ void __launch_bounds__(BOUNDARY_THREADS) k_boundary_plain(MeshDev m, StateDev s, BoundaryDev b, Ctrl *ctrl,
                                                                     int stage_in)
{
    __shared__ double buf[2][2][64];
    const auto cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank(), size = (int)cluster.num_blocks();
    const int sid = blockIdx.x / size, pair = threadIdx.x >> 6, at = threadIdx.x & 63;
    Ctrl &ct = ctrl[sid];
    const bool hancock = stage_in == STAGE_HANCOCK;
    const int stage = hancock ? 1 : stage_in;
    const int s0 = b.scen_seg[sid], s1 = b.scen_seg[sid + 1];
    if (s0 == s1 || skip_stage(ct, stage)) return;            // the same for every block of the cluster
    const int nseg = b.nseg;
    const size_t ns = b.nslot;
    const double *q = stage == 1 && !hancock ? s.work : s.q1;
    const double *base = hancock ? s.work : q;    // stock of the stage start (the substep start for Hancock)
    int ntile = 0;
    for (int sg = s0; sg < s1; ++sg) ntile += tile_count(b, sg);
    const int i = 2 * rank + pair;
    const SlotTile tile = i < ntile ? slot_tile(b, s0, i) : SlotTile{s0, 0, 0};
    const int k = tile.first + at, n = tile.end - tile.first;
    const bool on = at < n;
    OpenFace o{};
    double stock = 0., area = 0.;
    bool several = false;
    if (on) {
        o = open_face(m, b, k, tile.sg, q, s.z);
        stock = hancock ? base[o.c] : o.h;
        area = m.area[o.c];
        several = b.several[k];
    }
    const int mode = n > 0 ? b.seg_mode[tile.sg] : 0, policy = n > 0 ? b.stage_policy[tile.sg] : 0;
    const double dry = ct.dry, trial = ct.trial;
    double Q = 0., level = 0.;
    if (b.table_len > 0) {
        const double t = ct.time0 + ct.elapsed + (stage == 2 ? trial : hancock ? .5 * trial : 0.0);
        // writes the sampled rows, those of a segment without faces too
        const bool first = i < ntile && tile.first == b.seg_off[tile.sg] && at == 0;
        if (mode == 6 || first) Q = table_forcing(b, 0, tile.sg, t);
        if (mode == 2 || first) level = table_forcing(b, 1, tile.sg, t);
        if (first) { b.forcing[tile.sg] = Q; b.forcing[nseg + tile.sg] = level; }
    } else if (n > 0) { Q = b.forcing[tile.sg]; level = b.forcing[nseg + tile.sg]; }
    // wetted stage sum and wetted width of the conveyance inlets' tiles: a row
    // per warp, its first lane in slot order
    const bool inlet = mode == 6;
    if (inlet && on) {
        const double w = greater(o.h, dry) ? o.len : 0.;
        buf[pair][0][at] = (o.z + o.h) * w;
        buf[pair][1][at] = w;
    }
    __syncthreads();
    if (inlet && (threadIdx.x & 31) == 0) {
        const int row = (threadIdx.x >> 5) & 1;
        double sum = 0.;
#pragma unroll 8
        for (int j = 0; j < n; ++j) sum += buf[pair][row][j];
        b.terms[row * ns + tile.first] = sum;
    }
    cluster.sync();
    double w = 0., total = 0.;
    if (inlet) {
        double stage_sum = 0., width = 0.;
        for (int j = b.seg_off[tile.sg]; j < b.seg_off[tile.sg + 1]; j += 64) { stage_sum += b.terms[j]; width += b.terms[ns + j]; }
        if (on) { w = face_weight<F>(ct, o, stage_sum, width); buf[pair][0][at] = w; }
    }
    __syncthreads();
    if (inlet && at == 0) {
        double sum = 0.;
#pragma unroll 8
        for (int j = 0; j < n; ++j) sum += buf[pair][0][j];
        b.terms[2 * ns + tile.first] = sum;
    }
    cluster.sync();
    double tr[3] = {0., 0., 0.}, fl[3] = {0., 0., 0.};
    bool bad = false;
    if (inlet)
        for (int j = b.seg_off[tile.sg]; j < b.seg_off[tile.sg + 1]; j += 64) total += b.terms[2 * ns + j];
    if (on) {
        bad = plain_face(o, Q, level, policy, dry, ct.grav, ct.speed_limit, total, w, tr, fl) != 0;
        // outlet stock cap of an owner with one open face; the others below
        if (!several && is_outlet(mode) && greater(fl[0], 0.)) {
            const double factor = cap_factor(stock, area, trial, reciprocal(trial), fl[0] * o.len, 0.);
            if (factor != 1.) cap_face(factor, tr, fl);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) { b.trace[r * ns + k] = tr[r]; b.flux[r * ns + k] = fl[r]; }
    }
    if (bad) raise_status(ct, stage, ST_SPATIAL);
    if (b.scen_several[sid]) {
        cluster.sync();
        if (rank == 0)
            cap_owners(m, b, base, trial, b.scen_own[sid] + (int)threadIdx.x, b.scen_own[sid + 1], BOUNDARY_THREADS, true);
        cluster.sync();
        if (on && several) fl[0] = b.flux[k];
    }
    const double2 sum = warp_water(on ? double(F(fl[0])) * o.len : 0.);
    if (on && (threadIdx.x & 31) == 0) b.water_sum[k] = sum;
    cluster.sync();
    if (rank == 0) scenario_water(b, ct, stage, s0, ntile);
}

// The open boundary of one scenario in one block: any width, and any modes with
// BOUNDARY_THREADS (a section solve's lanes); with more, no section solves.
template <class F, int THREADS>
__global__ void __launch_bounds__(THREADS) k_boundary(MeshDev m, StateDev s, BoundaryDev b, Ctrl *ctrl, int stage_in)
{
    const bool sections = THREADS == BOUNDARY_THREADS && b.sections;
    __shared__ double tile_buf[2][BOUNDARY_TILES], warp_buf[THREADS / 32][2][64];
    const int sid = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Ctrl &ct = ctrl[sid];
    const bool hancock = stage_in == STAGE_HANCOCK;
    const int stage = hancock ? 1 : stage_in;
    if (skip_stage(ct, stage)) return;
    const int s0 = b.scen_seg[sid], s1 = b.scen_seg[sid + 1];
    if (s0 == s1) return;
    const int nseg = b.nseg;
    const size_t ns = b.nslot;
    const double *q = stage == 1 && !hancock ? s.work : s.q1;
    const double *base = hancock ? s.work : q;    // stock of the stage start (the substep start for Hancock)
    const double *z = s.z;
    const double dry = ct.dry, grav = ct.grav;
    // forcing at the stage clock (piecewise linear tables, else constant)
    if (b.table_len > 0) {
        const double t = ct.time0 + ct.elapsed + (stage == 2 ? ct.trial : hancock ? .5 * ct.trial : 0.0);
        for (int sg = s0 + threadIdx.x; sg < s1; sg += blockDim.x)
            for (int row = 0; row < 2; ++row) b.forcing[(size_t)row * nseg + sg] = table_forcing(b, row, sg, t);
        __syncthreads();
    }
    // critical, then normal reference lines of the exact-discharge inlets
    // (river_exterior_bed.py:199-200); a section without a root rejects the trial
    __shared__ SectionWork section;
    bool line_failed = false;
    if (sections && b.line_kind) {
        for (int pass = 1; pass <= 2; ++pass)
            for (int sg = s0; sg < s1; ++sg)          // block-uniform
                if (b.seg_mode[sg] == 9 && b.line_kind[sg] == pass &&
                    !line_section(section, m, b, sg, grav, dry, ct.roughness_mode, ct.roughness_value))
                    line_failed = true;
        __syncthreads();
    }
    int ntile = 0;
    for (int sg = s0; sg < s1; ++sg) ntile += tile_count(b, sg);
    // wetted stage sum and wetted width of the conveyance inlets' segments
    for (int i = warp; i < ntile; i += THREADS / 32) {
        const SlotTile tile = slot_tile(b, s0, i);
        if (b.seg_mode[tile.sg] != 6) continue;
        double lo[2] = {0., 0.}, hi[2] = {0., 0.};
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int k = tile.first + lane + 32 * half;
            if (k >= tile.end) continue;
            const int f = b.slot_face[k], c = m.owner[f];
            const double hc = q[c], w = greater(hc, dry) ? m.length[f] : 0.;
            (half ? hi : lo)[0] = (z[c] + hc) * w;
            (half ? hi : lo)[1] = w;
        }
        const double sum = tile_sum<2>(warp_buf[warp], tile.end - tile.first, lo, hi);
        if (lane < 2) tile_buf[lane][i] = sum;
    }
    __syncthreads();
    for (int sg = s0 + threadIdx.x; sg < s1; sg += blockDim.x) {
        if (b.seg_mode[sg] != 6) continue;
        int first = 0;
        for (int u = s0; u < sg; ++u) first += tile_count(b, u);
        double stage_sum = 0., width = 0.;
        for (int i = 0; i < tile_count(b, sg); ++i) { stage_sum += tile_buf[0][first + i]; width += tile_buf[1][first + i]; }
        b.seg_sums[sg] = stage_sum; b.seg_sums[nseg + sg] = width;
    }
    __syncthreads();
    // conveyance weights
    for (int i = warp; i < ntile; i += THREADS / 32) {
        const SlotTile tile = slot_tile(b, s0, i);
        if (b.seg_mode[tile.sg] != 6) continue;
        double lo[1] = {0.}, hi[1] = {0.};
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int k = tile.first + lane + 32 * half;
            if (k >= tile.end) continue;
            const double w = face_weight<F>(ct, open_face(m, b, k, tile.sg, q, z), b.seg_sums[tile.sg], b.seg_sums[nseg + tile.sg]);
            b.terms[2 * ns + k] = w;
            (half ? hi : lo)[0] = w;
        }
        const double sum = tile_sum<1>(warp_buf[warp], tile.end - tile.first, lo, hi);
        if (lane == 0) tile_buf[0][i] = sum;
    }
    __syncthreads();
    for (int sg = s0 + threadIdx.x; sg < s1; sg += blockDim.x) {
        if (b.seg_mode[sg] != 6) continue;
        int first = 0;
        for (int u = s0; u < sg; ++u) first += tile_count(b, u);
        double total = 0.;
        for (int i = 0; i < tile_count(b, sg); ++i) total += tile_buf[0][first + i];
        b.seg_sums[2 * (size_t)nseg + sg] = total;
    }
    __syncthreads();
    unsigned bad = 0;
    for (int i = threadIdx.x >> 6; i < ntile; i += THREADS / 64) {
        const SlotTile tile = slot_tile(b, s0, i);
        const int k = tile.first + (threadIdx.x & 63), mode = b.seg_mode[tile.sg];
        if (k >= tile.end) continue;
        double tr[3] = {0., 0., 0.}, fl[3] = {0., 0., 0.};
        if (!(mode == 4 || mode == 5 || mode == 9 || mode == 10 || mode == 11) &&
            plain_face(open_face(m, b, k, tile.sg, q, z), b.forcing[tile.sg], b.forcing[nseg + tile.sg],
                       b.stage_policy[tile.sg], dry, grav, ct.speed_limit,
                       mode == 6 ? b.seg_sums[2 * (size_t)nseg + tile.sg] : 0., mode == 6 ? b.terms[2 * ns + k] : 0., tr, fl))
            bad = 1;
#pragma unroll
        for (int r = 0; r < 3; ++r) { b.trace[r * ns + k] = tr[r]; b.flux[r * ns + k] = fl[r]; }
    }
    __syncthreads();
    if (sections) {
        // section owners of the remaining outlet modes, after the face loop, in
        // the reference's order (river_exterior_bed.py:213-217): a normal-depth
        // chain without a root rejects the trial before the rating owner runs; a
        // rating section without a solution fails the scenario
        __shared__ int section_reject;
        if (threadIdx.x == 0) section_reject = line_failed;
        __syncthreads();
        if (b.inlet && !section_reject) {
            bool inlet_failed = false;
            for (int sg = s0; sg < s1; ++sg)              // block-uniform: the CTA solves one section at a time
                if (b.seg_mode[sg] == 9) {
                    bool sbad = false;
                    if (inlet_section(section, m, b, sg, grav, dry, ct.speed_limit, q, z, sbad)) inlet_failed = true;
                    if (sbad) bad = 1;
                }
            if (threadIdx.x == 0 && inlet_failed) section_reject = 1;
            __syncthreads();
        }
        if (b.branch && !section_reject) {
            bool crit_failed = false;
            for (int sg = s0; sg < s1; ++sg)              // block-uniform: the CTA solves one section at a time
                if (b.seg_mode[sg] == 4) {
                    bool sbad = false;
                    if (crit_section(section, m, b, sg, grav, dry, ct.speed_limit, q, z, sbad)) crit_failed = true;
                    if (sbad) bad = 1;
                }
            if (threadIdx.x == 0 && crit_failed) section_reject = 1;
            __syncthreads();
        }
        if (b.weir && !section_reject) {
            for (int sg = s0; sg < s1; ++sg)              // block-uniform: the CTA solves one section at a time
                if (b.seg_mode[sg] == 5) {
                    bool sbad = false;
                    const int e = weir_section(section, m, b, sg, grav, dry, ct.speed_limit, q, z, sbad);
                    if (threadIdx.x == 0 && e) section_reject = 1;
                    if (sbad) bad = 1;
                }
            __syncthreads();
        }
        if (b.scen_chain && !section_reject) {
            const int law = ct.roughness_mode;
            for (int ch = b.scen_chain[sid] + threadIdx.x; ch < b.scen_chain[sid + 1]; ch += blockDim.x) {
                bool sbad = false;
                if (normal_chain(m, b, ch, grav, dry, ct.speed_limit, law, ct.roughness_value, q, z, sbad))
                    atomicOr(&section_reject, 1);
                if (sbad) bad = 1;
            }
        }
        __syncthreads();
        if (!section_reject)
            for (int sg = s0 + threadIdx.x; sg < s1; sg += blockDim.x)
                if (b.seg_mode[sg] == 11) {
                    bool sbad = false;
                    if (rating_section(m, b, sg, grav, dry, ct.speed_limit, q, z, sbad)) raise_status(ct, stage, ST_FATAL);
                    if (sbad) bad = 1;
                }
        if (section_reject) bad = 1;
        __syncthreads();
    }
    if (bad) raise_status(ct, stage, ST_SPATIAL);
    // outlet stock cap, one thread per unique owner, its faces in boundary order
    const int u0 = b.scen_own[sid], u1 = b.scen_own[sid + 1];
    cap_owners(m, b, base, ct.trial, u0 + (int)threadIdx.x, u1, THREADS, false);
    if (b.inlet) inlet_allocation(m, b, ct, base, s0, s1, u0, u1);
    __syncthreads();
    for (int i = warp; i < 2 * ntile; i += THREADS / 32) {
        const SlotTile tile = slot_tile(b, s0, i >> 1);
        const int first = tile.first + 32 * (i & 1), k = first + lane;
        const double2 sum = warp_water(k < tile.end ? double(F(b.flux[k])) * m.length[b.slot_face[k]] : 0.);
        if (lane == 0 && first < tile.end) b.water_sum[first] = sum;
    }
    __syncthreads();
    scenario_water(b, ct, stage, s0, ntile);
}

// Launch over nscen scenarios: b.cluster blocks each where every scenario fits
// a thread per face, else (b.cluster = 0) one block.
template <class F>
inline void launch_boundary(const MeshDev &m, const StateDev &s, const BoundaryDev &b, Ctrl *ctrl, int nscen, int stage,
                            cudaStream_t st)
{
    if (b.cluster == 0) {
        if (b.sections) k_boundary<F, BOUNDARY_THREADS><<<nscen, BOUNDARY_THREADS, 0, st>>>(m, s, b, ctrl, stage);
        else k_boundary<F, BOUNDARY_WIDE><<<nscen, BOUNDARY_WIDE, 0, st>>>(m, s, b, ctrl, stage);
        return;
    }
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = b.cluster; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nscen * b.cluster); cfg.blockDim = dim3(BOUNDARY_THREADS); cfg.stream = st;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_boundary_plain<F>, m, s, b, ctrl, stage);
}

// ---------------------------------------------------------------------------
// Cells: primitive values, limited least-squares gradients, flattening flag.
// The general FP64 sweep: cells of more than four faces, and the
// allocation-free residual.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool feasible(double x, double y, int count, const double *ax, const double *ay, const double *bb)
{
    for (int i = 0; i < count; ++i)
        if (ax[i] * x + ay[i] * y > bb[i] + 2.e-14) return false;
    return true;
}

static __device__ __noinline__ void project_pair(double &x, double &y, int count, const double *ax, const double *ay, const double *bb)
{
    const double rx = x, ry = y;
    if (feasible(rx, ry, count, ax, ay, bb)) return;
    double bx = 0., by = 0., best = rx * rx + ry * ry;
    for (int i = 0; i < count; ++i) {
        const double dot = ax[i] * rx + ay[i] * ry - bb[i];
        double cx = rx - dot * ax[i], cy = ry - dot * ay[i];
        double d = (cx - rx) * (cx - rx) + (cy - ry) * (cy - ry);
        if (d < best && feasible(cx, cy, count, ax, ay, bb)) { bx = cx; by = cy; best = d; }
        for (int j = 0; j < i; ++j) {
            const double det = ax[i] * ay[j] - ay[i] * ax[j];
            if (fabs(det) < 1.e-12) continue;
            cx = (bb[i] * ay[j] - ay[i] * bb[j]) / det;
            cy = (ax[i] * bb[j] - bb[i] * ax[j]) / det;
            d = (cx - rx) * (cx - rx) + (cy - ry) * (cy - ry);
            if (d < best && feasible(cx, cy, count, ax, ay, bb)) { bx = cx; by = cy; best = d; }
        }
    }
    x = bx; y = by;
}

// MAXF bounds the faces of one cell.
template <int MAXF>
__global__ void __launch_bounds__(128) k_cells(MeshDev m, StateDev s, Ctrl *ctrl, Work w, int stage)
{
    const int nc = m.nc, nf = m.nf, nadj = m.nadj;
    FOR_ACTIVE_CELLS(m.act, c) {
        Ctrl &ct = ctrl[m.cell_sid[c]];
        if (skip_stage(ct, stage)) continue;
        const double *q = stage == 1 ? s.work : s.q1;
        const double *z = s.z;
        const double dry = ct.dry, grav = ct.grav;
        const double h = q[c], hu = q[nc + c], hv = q[2 * nc + c], zc = z[c];
        if (h < 0.0 || !isfinite(h) || !isfinite(zc) || !isfinite(hu) || !isfinite(hv))
            raise_status(ct, stage, ST_SPATIAL);
        double centre[4] = {h + zc, 0., 0., zc};
        if (h > dry) { centre[1] = hu / h; centre[2] = hv / h; }
        double lo[4], hi[4];
        double gx[4] = {0., 0., 0., 0.}, gy[4] = {0., 0., 0., 0.};
#pragma unroll
        for (int p = 0; p < 4; ++p) { lo[p] = centre[p]; hi[p] = centre[p]; }
        const int k0 = m.offset[c], k1 = m.offset[c + 1];
        // active: wet, or touching an open face or a wet neighbour
        bool active = h > dry;
        double bx[4] = {0., 0., 0., 0.}, by[4] = {0., 0., 0., 0.};
        for (int k = k0; k < k1; ++k) {
            const int f = m.faces[k];
            const int n = m.signs[k] < 0 ? m.owner[f] : m.neighbour[f];
            if (n < 0) { if (m.bid[f] >= 0) active = true; continue; }
            const double hn = q[n], zn = z[n];
            if (hn > dry) active = true;
            double vn[4] = {hn + zn, 0., 0., zn};
            if (hn > dry) { vn[1] = q[nc + n] / hn; vn[2] = q[2 * nc + n] / hn; }
            const double rx = m.ls_delta[k], ry = m.ls_delta[nadj + k], wt = m.ls_weight[k];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                double adj = vn[p];
                if (p == 0 && centre[0] - centre[3] > dry && vn[0] - vn[3] <= dry && vn[3] >= centre[0]) adj = centre[0];
                const double d = adj - centre[p];
                bx[p] += wt * rx * d;
                by[p] += wt * ry * d;
                lo[p] = fmin(lo[p], adj); hi[p] = fmax(hi[p], adj);
            }
        }
        if (active) {
            const double a11 = m.ls_matrix[c], a12 = m.ls_matrix[nc + c], a22 = m.ls_matrix[2 * nc + c],
                    det = m.ls_matrix[3 * nc + c];
            if (a11 + a22 > 0.0) {
                if (h > dry)
                    for (int k = k0; k < k1; ++k) {
                        const int f = m.faces[k];
                        if (m.neighbour[f] >= 0 || m.bid[f] >= 0) continue;
                        const double nx = m.normal[f], ny = m.normal[nf + f];
                        const double un = centre[1] * nx + centre[2] * ny;
                        const double mx = centre[1] - 2. * un * nx, my = centre[2] - 2. * un * ny;
                        lo[1] = fmin(lo[1], mx); hi[1] = fmax(hi[1], mx);
                        lo[2] = fmin(lo[2], my); hi[2] = fmax(hi[2], my);
                    }
                const bool full = det > 1.e-12 * ((a11 + a22) * (a11 + a22));
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    if (full) {
                        gx[p] = (a22 * bx[p] - a12 * by[p]) / det;
                        gy[p] = (a11 * by[p] - a12 * bx[p]) / det;
                    } else {
                        gx[p] = (a11 * bx[p] + a12 * by[p]) / ((a11 + a22) * (a11 + a22));
                        gy[p] = (a12 * bx[p] + a22 * by[p]) / ((a11 + a22) * (a11 + a22));
                    }
                }
                const double hh = centre[0] - centre[3];
                const double sq = hh > dry ? sqrt(grav * hh) : 0.;
                const double bedtol = 64.0 * EPS * fmax(1.0, fabs(centre[3]));
                double theta1 = 1., theta2 = 1.;
                double ax0[2 * MAXF], ay0[2 * MAXF], b0[2 * MAXF];
                double ax3[2 * MAXF], ay3[2 * MAXF], b3[2 * MAXF];
                int n0 = 0, n3 = 0;
                for (int k = k0; k < k1; ++k) {
                    const int f = m.faces[k];
                    const int side = m.signs[k] < 0;
                    const double rx = m.disp[side * nf + f], ry = m.disp[(2 + side) * nf + f];
                    // an open stage outlet with a subcritical wet owner keeps its bed slope
                    if (m.bmode[f] == 2 && m.neighbour[f] < 0 && hh > dry &&
                        fabs(centre[1] * m.normal[f] + centre[2] * m.normal[nf + f]) < sq &&
                        fabs(gx[3] * rx + gy[3] * ry) > bedtol) continue;
#pragma unroll
                    for (int p = 1; p < 3; ++p) {
                        const double d = gx[p] * rx + gy[p] * ry;
                        if (fabs(d) <= 64.0 * EPS * fmax(1.0, fmax(fabs(centre[p]), fmax(fabs(lo[p]), fabs(hi[p])))))
                            continue;
                        double &th = p == 1 ? theta1 : theta2;
                        if (d > 0.) th = fmin(th, (hi[p] - centre[p]) / d);
                        if (d < 0.) th = fmin(th, (lo[p] - centre[p]) / d);
                    }
                    const double len = m.disp_len[side * nf + f];
                    if (len <= 0.) continue;
                    const double ux = m.disp_unit[side * nf + f], uy = m.disp_unit[(2 + side) * nf + f];
                    ax0[n0] = ux; ay0[n0] = uy; b0[n0++] = fmax(0., hi[0] - centre[0]) / len;
                    ax0[n0] = -ux; ay0[n0] = -uy; b0[n0++] = fmax(0., centre[0] - lo[0]) / len;
                    if (m.neighbour[f] < 0 && m.bid[f] < 0) continue;   // walls do not bound the bed
                    ax3[n3] = ux; ay3[n3] = uy; b3[n3++] = fmax(0., hi[3] - centre[3]) / len;
                    ax3[n3] = -ux; ay3[n3] = -uy; b3[n3++] = fmax(0., centre[3] - lo[3]) / len;
                }
                double px0 = gx[0], py0 = gy[0], px3 = gx[3], py3 = gy[3];
                project_pair(px0, py0, n0, ax0, ay0, b0);
                project_pair(px3, py3, n3, ax3, ay3, b3);
                gx[1] *= fmax(0., theta1); gy[1] *= fmax(0., theta1);
                gx[2] *= fmax(0., theta2); gy[2] *= fmax(0., theta2);
                gx[0] = px0; gy[0] = py0; gx[3] = px3; gy[3] = py3;
            }
        }
        bool flatten = h <= dry;
        if (!flatten)
            for (int k = k0; k < k1; ++k) {
                const int f = m.faces[k];
                const int side = (c == m.owner[f]) ? 0 : 1;
                const double rx = m.disp[side * nf + f], ry = m.disp[(2 + side) * nf + f];
                const double eta = (centre[0] + gx[0] * rx) + gy[0] * ry;
                const double zb = (centre[3] + gx[3] * rx) + gy[3] * ry;
                if (eta - zb <= dry || fabs(zb - centre[3]) >= h) { flatten = true; break; }
            }
        CellRec r;
        r.h = h; r.eta = centre[0]; r.u = centre[1]; r.v = centre[2]; r.b = centre[3];
#pragma unroll
        for (int p = 0; p < 4; ++p) { r.gx[p] = gx[p]; r.gy[p] = gy[p]; }
        r.flags = (flatten ? 1 : 0) | (active ? 2 : 0);
        r.pad = 0; r.pad2 = 0.;
        w.rec[c] = r;
    }
}

// midpoint_faces: limit donor outflow, carry the removed advective momentum.
__global__ void __launch_bounds__(256) k_limit(MeshDev m, StateDev s, Ctrl *ctrl, Work w, int stage)
{
    const int nf = m.nf, nc = m.nc;
    FOR_ACTIVE_FACES(m.act, f) {
        const Ctrl &ct = ctrl[m.face_sid[f]];
        if (skip_stage(ct, stage)) continue;
        const double *q = stage == 1 ? s.work : s.q1;
        double water = w.ws[f].x, cx = 0., cy = 0.;
        if (water != 0. && m.bslot[f] < 0) {
            const int donor = water < 0. ? m.neighbour[f] : m.owner[f];
            if (donor >= 0) {
                const double th = w.theta[donor];
                if (th != 1.) {
                    const double delta = (th - 1.) * water;
                    water *= th;
                    const double hd = q[donor];
                    if (hd > ct.dry) { cx = delta * q[nc + donor] / hd; cy = delta * q[2 * nc + donor] / hd; }
                }
            }
        }
        w.lim[f] = make_double4_32a(water, cx, cy, 0.);
    }
}

// ---------------------------------------------------------------------------
// Conservative wet-bank viscosity (shoreline_viscosity.py:57-72): velocity
// gradients of the safe state by the flow engines' least squares
// (bend_methods_v1_kernels.h:23-39, rows u and v; dry columns read as depth
// 0.001001 without momentum, secondary_vector_ops.py:39-48), then the
// shared-face stress of wet columns (shoreline_viscosity.h:14-33); the
// updates gather it as sum(s len stress) / area after the rotor terms.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_visc_grad(MeshDev m, Work w, const double *q, Ctrl *ctrl, int stage)
{
    const int n = m.nc, na = m.nadj;
    const ViscDev v = w.visc;
    FOR_ACTIVE_CELLS(m.act, i) {
        const int sid = m.cell_sid[i];
        if (!(v.nu[sid] > 0.) || skip_stage(ctrl[sid], stage)) continue;
        const double dry = ctrl[sid].dry;
        const bool wi = q[i] > dry;
        const double hi = wi ? q[i] : .001001;
        const double x0 = (wi ? q[n + i] : 0.) / hi, x1 = (wi ? q[2 * n + i] : 0.) / hi;
        double bx0 = 0., bx1 = 0., by0 = 0., by1 = 0.;
        for (int k = m.offset[i]; k < m.offset[i + 1]; ++k) {
            const int f = m.faces[k], j = m.owner[f] == i ? m.neighbour[f] : m.owner[f];
            if (j < 0) continue;
            const double dx = v.dxdy[k], dy = v.dxdy[na + k], wt = 1. / (dx * dx + dy * dy);
            const bool wj = q[j] > dry;
            const double hj = wj ? q[j] : .001001;
            const double y0 = (wj ? q[n + j] : 0.) / hj, y1 = (wj ? q[2 * n + j] : 0.) / hj;
            bx0 += wt * dx * (y0 - x0); by0 += wt * dy * (y0 - x0);
            bx1 += wt * dx * (y1 - x1); by1 += wt * dy * (y1 - x1);
        }
        v.grad[i] = v.inverse[i] * bx0 + v.inverse[n + i] * by0;
        v.grad[n + i] = v.inverse[n + i] * bx0 + v.inverse[2 * n + i] * by0;
        v.grad[2 * n + i] = v.inverse[i] * bx1 + v.inverse[n + i] * by1;
        v.grad[3 * n + i] = v.inverse[n + i] * bx1 + v.inverse[2 * n + i] * by1;
    }
}

__global__ void __launch_bounds__(256) k_visc_faces(MeshDev m, Work w, const double *q, const double *z, Ctrl *ctrl,
                                                    int stage)
{
    const int n = m.nc, nf = m.nf;
    const ViscDev v = w.visc;
    FOR_ACTIVE_FACES(m.act, i) {
        const int sid = m.face_sid[i];
        const double nu = v.nu[sid];
        if (!(nu > 0.) || skip_stage(ctrl[sid], stage)) continue;
        const double dry = ctrl[sid].dry;
        double sx = 0., sy = 0.;
        const int o = m.owner[i], j = m.neighbour[i];
        if (j >= 0 && q[o] > dry && q[j] > dry) {
            double h = fmin(q[o], q[j]);
            h = fmin(h, fmax(0., .5 * (q[o] + z[o] + q[j] + z[j]) - fmax(z[o], z[j])));
            const double d = m.distance[i] + m.distance[nf + i], wo = m.distance[nf + i] / d, wj = m.distance[i] / d;
            const double nx = m.normal[i], ny = m.normal[nf + i], dx = v.xy[j] - v.xy[o], dy = v.xy[n + j] - v.xy[n + o];
            const double dn = dx * nx + dy * ny;
            const double tx = dx - dn * nx, ty = dy - dn * ny;
            const double du = q[n + j] / q[j] - q[n + o] / q[o], dv = q[2 * n + j] / q[j] - q[2 * n + o] / q[o];
            const double ux = wo * v.grad[o] + wj * v.grad[j], uy = wo * v.grad[n + o] + wj * v.grad[n + j];
            const double vx = wo * v.grad[2 * n + o] + wj * v.grad[2 * n + j];
            const double vy = wo * v.grad[3 * n + o] + wj * v.grad[3 * n + j];
            sx = nu * h * (du - ux * tx - uy * ty) / dn;
            sy = nu * h * (dv - vx * tx - vy * ty) / dn;
        }
        v.face[i] = sx;
        v.face[nf + i] = sy;
    }
}

// The wet-bank viscosity's momentum rate of one cell: sum(s len stress) / area
// with unit weights (flow2dh_fixed_bed_kernels.h:54-60).
__device__ __forceinline__ void add_viscosity(const MeshDev &m, const ViscDev &v, int c, double area, double &r1,
                                              double &r2)
{
    const int nf = m.nf;
    double x = 0., y = 0.;
    for (int k = m.offset[c]; k < m.offset[c + 1]; ++k) {
        const int f = m.faces[k];
        x += m.signs[k] * m.length[f] * v.face[f];
        y += m.signs[k] * m.length[f] * v.face[nf + f];
    }
    r1 += 1. * x / area;
    r2 += 1. * y / area;
}

// ---------------------------------------------------------------------------
// Control: accept/reject the trial and set the next one (RiverExplicit.advance).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void set_trial(Ctrl &c)
{
    c.trial = fmin(c.hint, c.dt_outer - c.elapsed);
    c.truncated = c.trial < c.hint * (1 - 1e-12);
    c.status1 = 0; c.status2 = 0; c.peak1 = 0ull; c.peak2 = 0ull;
    c.gravf = float(c.grav); c.dryf = float(c.dry); c.trialf = float(c.trial);
    c.roughf = float(c.roughness_value); c.cfl1 = 0;
}

// The active set of the next trial from the control blocks, as runs of
// consecutive active scenarios: warp 0 scans the scenarios 32 at a time
// (ballots for run starts, shuffle scans for the cell and face prefixes).
__device__ void active_rebuild(const Ctrl *ctrl, int nscen, const ActiveDev &a)
{
    if (threadIdx.x >= 32) return;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x;
    int nrun = 0, ncell = 0, nface = 0;
    bool carry = false;                       // the previous chunk's last scenario was active
    for (int base = 0; base < nscen; base += 32) {
        const int i = base + lane;
        const bool on = i < nscen && ctrl[i].active && !ctrl[i].done;
        bool prev = __shfl_up_sync(full, on, 1);
        if (lane == 0) prev = carry;
        const bool first = on && !prev;
        const int cells = on ? a.cell_off[i + 1] - a.cell_off[i] : 0;
        const int faces = on ? a.face_off[i + 1] - a.face_off[i] : 0;
        const unsigned starts = __ballot_sync(full, first);
        int cs = cells, fs = faces;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int x = __shfl_up_sync(full, cs, d), y = __shfl_up_sync(full, fs, d);
            if (lane >= d) { cs += x; fs += y; }
        }
        if (first) {
            const int r = nrun + __popc(starts & ((1u << lane) - 1u));
            const int c0 = ncell + cs - cells, f0 = nface + fs - faces;
            a.cstart[r] = c0; a.cdelta[r] = a.cell_off[i] - c0;
            a.fstart[r] = f0; a.fdelta[r] = a.face_off[i] - f0;
        }
        nrun += __popc(starts);
        ncell += __shfl_sync(full, cs, 31);
        nface += __shfl_sync(full, fs, 31);
        carry = __shfl_sync(full, on, 31);
    }
    if (lane == 0) {
        a.cstart[nrun] = ncell; a.fstart[nrun] = nface;
        a.count[0] = nrun; a.count[1] = ncell; a.count[2] = nface;
        a.count[3] = a.count[4] = 0;
    }
}

// Active set of the first trial of an interval (after the host's control upload).
__global__ void k_active_init(const Ctrl *ctrl, int nscen, ActiveDev a) { active_rebuild(ctrl, nscen, a); }

__device__ void control_one(Ctrl &c);

// Substep control of every scenario (one block), then the next trial's active set.
__global__ void k_control(Ctrl *ctrl, int nscen, ActiveDev a)
{
    for (int i = threadIdx.x; i < nscen; i += blockDim.x) control_one(ctrl[i]);
    __syncthreads();
    active_rebuild(ctrl, nscen, a);
}

// A chained scenario has completed an interval: record it and begin the
// next one as the host begins an interval (begin_interval_each), with the
// start time advanced by one interval and the controller's hint carried
// over, so the chain reproduces consecutive intervals bit for bit. The
// accepted state stays in the buffer it is in (the kernels read q[cur]).
__device__ __forceinline__ void chain_next(Ctrl &c)
{
    IvStat &r = c.hist[c.chain_pos];
    r.substeps = c.substeps; r.rejections = c.rejections; r.failed = 0; r.pad = 0;
    r.min_dt = c.min_dt; r.max_dt = c.max_dt; r.cfl_max = c.cfl_max; r.hint = c.hint;
    r.ledger = c.ledger; r.gross = c.gross;
    c.time0 += c.dt_outer;
    c.elapsed = 0.0;
    c.substeps = c.rejections = 0;
    c.min_dt = c.max_dt = c.cfl_max = 0.0;
    c.bflux[0] = c.bflux[1] = c.ledger = 0.0;
    c.bgross[0] = c.bgross[1] = c.gross = 0.0;
    --c.chain_left;
    ++c.chain_pos;
}

__device__ void control_one(Ctrl &c)
{
    if (!c.active || c.done) return;
    // a rotor outside its model's domain ends the scenario (the reference raises)
    if ((c.status1 | c.status2) & ST_TURBINE) { c.failed = 4; c.done = 1; return; }
    if ((c.status1 | c.status2) & ST_FATAL) { c.failed = 5; c.done = 1; return; }
    const double f1 = bits_to_double(c.peak1), f2 = bits_to_double(c.peak2);
    // the reference's frequency peak only sees stages that reached the CFL evaluation
    double peak = 0.;
    bool reject = false;
    if (c.status1 & ST_PRE) reject = true;
    else {
        peak = f1;
        if (c.trial * f1 > c.cfl * (1 + 1e-12) || (c.status1 & ST_ENDPOINT)) reject = true;
        else if (c.status2 & ST_PRE) reject = true;
        else {
            peak = fmax(peak, f2);
            if (c.trial * f2 > c.cfl * (1 + 1e-12) || (c.status2 & ST_ENDPOINT)) reject = true;
        }
    }
    if (reject) {
        c.rejections++;
        c.hint = peak > 0 ? fmin(.5 * c.trial, .98 * c.cfl / peak) : .5 * c.trial;
        if (c.hint < c.floor_ || c.rejections > 100) { c.failed = 1; c.done = 1; return; }
    } else {
        c.cur ^= 1;
        c.elapsed += c.trial;
        c.ledger -= c.trial * (c.one_stage ? c.bflux[0] : .5 * (c.bflux[0] + c.bflux[1]));
        c.gross += c.trial * (c.one_stage ? c.bgross[0] : .5 * (c.bgross[0] + c.bgross[1]));
        c.substeps++;
        if (c.substeps == 1 || c.trial < c.min_dt) c.min_dt = c.trial;
        if (c.trial > c.max_dt) c.max_dt = c.trial;
        if (c.trial * peak > c.cfl_max) c.cfl_max = c.trial * peak;
        const double growth = c.truncated ? c.hint : 2 * c.trial;
        c.hint = peak > 0 ? fmin(growth, .98 * c.cfl / peak) : growth;
        if (c.substeps > c.max_substeps) { c.failed = 2; c.done = 1; return; }
        if (!(c.elapsed < c.dt_outer - 1e-13 * fmax(1., c.dt_outer))) {
            if (c.chain_left <= 0) { c.done = 1; return; }
            chain_next(c);
        }
    }
    set_trial(c);
}

// Limited water flux of the last stage into a caller buffer.
__global__ void k_water_out(MeshDev m, Work w, double *water)
{
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < m.nf; f += gridDim.x * blockDim.x) water[f] = w.lim[f].x;
}

// Compensated per-scenario sums of a state, Neumaier summation in a fixed order
// (the same on every run): each thread a strided slice of its block's chunk,
// pairs merged by a halving tree, then the blocks' partial pairs by one warp of
// the block that finishes last. Bound by the chain of FP64 additions in a
// thread, not by memory: a scenario gets a block per 2,048 cells (8 cells a
// thread), so that a large one is not left to one SM. A call with its copies,
// one block per scenario before: 360 cells 176 -> 45 us, 50k cells 683 -> 63 us,
// 190k cells 1,780 -> 63 us.
struct Pair { double sum, comp; };

__device__ __forceinline__ void neumaier_add(Pair &p, double v)
{
    const double t = p.sum + v;
    if (magnitude(p.sum) >= magnitude(v)) p.comp += (p.sum - t) + v;
    else p.comp += (v - t) + p.sum;
    p.sum = t;
}

__device__ __forceinline__ void merge_warp(Pair &p)
{
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const double s = __shfl_down_sync(0xffffffffu, p.sum, w), c = __shfl_down_sync(0xffffffffu, p.comp, w);
        neumaier_add(p, s);
        p.comp += c;
    }
}

constexpr int TOTALS_CHUNK = 2048;
__host__ __device__ __forceinline__ int totals_blocks(int cells) { return (cells + TOTALS_CHUNK - 1) / TOTALS_CHUNK; }

// BUDGET false: water volume sum(A h) and mechanical energy per unit density
// sum(A (|hu|^2 / (2h) + g h^2 / 2 + g h z)) (kinetic only where h > dry; gd: the
// scenarios' gravity and dry depth). BUDGET true: volume of the start state q0,
// volume of q, and the inventory sum(A max(h0, h)). One grid dimension over the
// blocks of all scenarios (a grid's second holds 65,535): block i works for
// scenario block_sid[i], whose blocks begin at first[]. part: (blocks, 3)
// scratch; tickets (nscen) zero, left zero.
template <bool BUDGET>
__global__ void __launch_bounds__(256) k_totals(MeshDev m, const double *q, const double *q0, const double *z,
                                                const double *gd, const int *first, const int *block_sid, Pair *part,
                                                unsigned *tickets, double *out)
{
    constexpr int N = BUDGET ? 3 : 2;
    __shared__ Pair warps[N][8];
    __shared__ bool last;
    const int sid = block_sid[blockIdx.x], nc = m.nc, c0 = m.act.cell_off[sid], c1 = m.act.cell_off[sid + 1];
    const int blocks = totals_blocks(c1 - c0), block = blockIdx.x - first[sid];
    const int from = c0 + block * TOTALS_CHUNK, to = min(c1, from + TOTALS_CHUNK);
    const double g = BUDGET ? 0. : gd[2 * sid], dry = BUDGET ? 0. : gd[2 * sid + 1];
    Pair p[N] = {};
    for (int c = from + threadIdx.x; c < to; c += blockDim.x) {
        const double h = q[c], a = m.area[c];
        if constexpr (BUDGET) {
            const double h0 = q0[c];
            neumaier_add(p[0], a * h0);
            neumaier_add(p[1], a * h);
            neumaier_add(p[2], a * (greater(h0, h) ? h0 : h));
        } else {
            neumaier_add(p[0], a * h);
            double e = .5 * g * h * h + g * h * z[c];
            if (greater(h, dry)) {
                const double hu = q[nc + c], hv = q[2 * nc + c];
                e += quotient(.5 * (hu * hu + hv * hv), h, reciprocal(h));
            }
            neumaier_add(p[1], a * e);
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < N; ++k) { merge_warp(p[k]); if (lane == 0) warps[k][warp] = p[k]; }
    __syncthreads();
    if (warp < N) {
        Pair v = lane < 8 ? warps[warp][lane] : Pair{0., 0.};
        merge_warp(v);
        if (lane == 0) { part[3 * (size_t)blockIdx.x + warp] = v; __threadfence(); }
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(&tickets[sid], blocks - 1) == (unsigned)(blocks - 1);
    __syncthreads();
    if (!last || warp >= N) return;
    __threadfence();
    Pair v{0., 0.};
    for (int b = lane; b < blocks; b += 32) {
        const volatile Pair &o = part[3 * (size_t)(first[sid] + b) + warp];
        const double os = o.sum, oc = o.comp;
        neumaier_add(v, os);
        v.comp += oc;
    }
    merge_warp(v);
    if (lane == 0) out[N * sid + warp] = v.sum + v.comp;
}

// Make the caller-bound buffer q[0] hold every scenario's accepted state.
__global__ void k_commit(MeshDev m, StateDev s, Ctrl *ctrl)
{
    const int nc = m.nc;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        if (!ctrl[m.cell_sid[c]].cur) continue;
        s.q[0][c] = s.q[1][c];
        s.q[0][nc + c] = s.q[1][nc + c];
        s.q[0][2 * nc + c] = s.q[1][2 * nc + c];
    }
}

}  // namespace BRX_NS
