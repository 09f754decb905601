// Exner bed update with Meyer-Peter-Mueller transport, one grain size, once per
// outer interval (FP64 in both arithmetic forms; compiled in the FP64 unit):
//
//   finish / bed_faces    src/braids_core/sediment/shoreline_solver.py:209-240,
//                         flow2dh_mobile_bed.py:101-109
//   MPM capacity          river_mpm.h:32-46 (hI = 0: no secondary-flow spiral)
//   bed gradient          bend_methods_v1_kernels.h:23-39 (z row)
//   face inputs, flux     flow2dh_mobile_kernels.h:13-53
//   slope correction      src/braids_gpu/flow_bed_slope_runtime.cu:13-144 (ISlope 3)
//   donor limit, div      bend_methods_v1_kernels.h:389-405
//
// Cells, faces and donor factors are grid-stride sweeps over every scenario with
// a bed model. The trial sweep limits each flux as it reads it and reduces the
// budget residual, donor minimum and relative change in a fixed order, a block
// per 1,024 cells; the block that finishes last adds the boundary volume and
// decides, and a last sweep commits the trial bed where the checks pass.
//
// Bound by FP64 instructions (brx_num64.cuh), and at one block per scenario for
// the reduction it was bound by that block, 1.3 of 2.2 ms. With no secondary-flow
// spiral the effective transport direction is the velocity's (the spiral's angle
// is a zero, its factors are ones), so its hypotenuses, square roots and unit
// powers are left out, theta^.5 is a square root, x^1.5 is x sqrt(x). One update
// of 192k cells, call to return: 2,230 -> 215 us.
#pragma once
#include "brx_num64.cuh"

namespace brx {

enum { EP_D = 0, EP_POROSITY, EP_CHEZY, EP_MORFAC, EP_SEDDEPTH, EP_D90, EP_HIDING, EP_N = 8 };
enum { ES_OK = 0, ES_RESIDUAL, ES_BOUNDARY, ES_DONOR, ES_CHANGE, ES_BAD, ES_N = 8 };

struct ExnerDev {
    const int *enabled;          // (nscen)
    const double *param;         // (nscen, 8)
    const int *bedbc;            // (nf) 0 wall, 1 feed, 2 outflow, 3 capacity
    const double *feed, *rock;   // (nf) (nc)
    const double *wdxdy;         // (2, nadj) centre offsets over their squared length
    const double *inverse, *xy;
    double *cell;                // (3, nc) transport x, y and Shields stress
    double *gz;                  // (2, nc) bed gradient
    double *flux;                // (nf) solid volume flux per length
    double *fac;                 // (nc) donor factors
    double *ztrial;              // (nc)
    double *stats;               // (nscen, 8)
    double *part;                // (blocks, 3) residual sum, donor minimum, change maximum of a chunk of cells
    const int *first, *chunk_sid;   // (nscen+1) first chunk of each scenario; (chunks) scenario of each
    unsigned *tickets;           // (nscen) zero between calls
    int *wet;                    // (nc)
    int *bad;                    // (nscen) slope operator status
    int *out_of_range;           // (nscen) a trial bed below the non-erodible layer or nonfinite
    const double *dt;            // (nscen) interval of each scenario (seconds of hydraulics)
};

__global__ void __launch_bounds__(256) k_ex_cells(MeshDev m, ExnerDev e, const double *q, const double *z)
{
    const int n = m.nc, na = m.nadj;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int sid = m.cell_sid[i];
        if (!e.enabled[sid]) continue;
        const double *p = e.param + (size_t)sid * EP_N;
        const double d = p[EP_D], c = p[EP_CHEZY], d90 = p[EP_D90], hide = p[EP_HIDING];
        // division-safe state at the sediment working depth (secondary_vector_ops.safe)
        const bool wet = q[i] > p[EP_SEDDEPTH];          // false for a NaN
        e.wet[i] = wet;
        const double h = wet ? q[i] : .001001, hu = wet ? q[n + i] : 0., hv = wet ? q[2 * n + i] : 0.;
        double bx = 0., by = 0.;
        for (int s = m.offset[i]; s < m.offset[i + 1]; ++s) {
            const int f = m.faces[s];
            const int j = m.signs[s] < 0 ? m.owner[f] : m.neighbour[f];
            if (j < 0) continue;
            const double dz = z[j] - z[i];
            bx += e.wdxdy[s] * dz; by += e.wdxdy[na + s] * dz;
        }
        e.gz[i] = e.inverse[i] * bx + e.inverse[n + i] * by;
        e.gz[n + i] = e.inverse[n + i] * bx + e.inverse[2 * n + i] * by;
        const double r = reciprocal(h), u = any_quotient(hu, h, r), v = any_quotient(hv, h, r), speed = hypot(u, v);
        const double unit = c * c * 1.65 * d, theta = any_quotient(speed * speed, unit, reciprocal(unit));
        double x = 0., y = 0.;
        if (speed > 0.) {                                // false for a NaN, which the slope operator reports
            const double depth = greater(h, .01) ? h : .01, rough = quotient(depth, d90, reciprocal(d90));
            const double grain = 18. * log10(12. * (greater(rough, 1.) ? rough : 1.)), part = quotient(c, grain, reciprocal(grain));
            const double power = part * sqrt(part), mu = greater(power, 1.) ? 1. : power;
            const double excess = mu * theta - .047 * hide;
            if (greater(excess, 0.)) {
                const double mag = 2650. * 8. * sqrt(9.81 * 1.65 * d * excess) * d * excess, rs = reciprocal(speed);
                x = any_quotient(mag * u, speed, rs); y = any_quotient(mag * v, speed, rs);
            }
        }
        e.cell[i] = x; e.cell[n + i] = y; e.cell[2 * n + i] = theta;
    }
}

// Koch--Flokstra slope correction, FLOW ISlope 3 with alfabs = alfabn = 0 (no
// change of magnitude), ashld .85, bshld .5, cshld = dshld = 0. Returns 0 or
// the operator's status.
__device__ __forceinline__ int slope_ks3(double qx, double qy, double down_x, double down_y, double stress,
                                         double &cx, double &cy)
{
    cx = qx; cy = qy;
    if (!finite_bits(qx) || !finite_bits(qy) || !finite_bits(down_x) || !finite_bits(down_y) || !finite_bits(stress) ||
        stress < 0.) return 2;
    const double magnitude = sqrt(qx * qx + qy * qy);
    if (!finite_bits(magnitude)) return 2;
    if (!greater(magnitude, 1.0e-6)) return 0;
    const double rm = reciprocal(magnitude);
    double dirx, diry;
    if (down_x != 0.0 || down_y != 0.0) {
        const double ftheta = .85 * sqrt(stress);
        dirx = quotient(ftheta * qx, magnitude, rm) + down_x; diry = quotient(ftheta * qy, magnitude, rm) + down_y;
    } else { dirx = quotient(qx, magnitude, rm); diry = quotient(qy, magnitude, rm); }
    const double norm = sqrt(dirx * dirx + diry * diry);
    if (!finite_bits(norm) || !greater(norm, 2.2250738585072014e-308)) return 3;
    cx = magnitude * dirx / norm; cy = magnitude * diry / norm;
    if (!finite_bits(cx) || !finite_bits(cy)) { cx = qx; cy = qy; return 4; }
    return 0;
}

__global__ void __launch_bounds__(128) k_ex_faces(MeshDev m, ExnerDev e, const double *z)
{
    const int n = m.nc, nf = m.nf;
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
        const int sid = m.face_sid[f];
        if (!e.enabled[sid]) continue;
        const int o = m.owner[f], j = m.neighbour[f];
        const double nx = m.normal[f], ny = m.normal[nf + f];
        double x = e.cell[o], y = e.cell[n + o], gx = e.gz[o], gy = e.gz[n + o], stress = e.cell[2 * n + o];
        if (j >= 0) {
            const double dd = m.distance[f] + m.distance[nf + f], rd = reciprocal(dd);
            const double wo = quotient(m.distance[nf + f], dd, rd), wj = quotient(m.distance[f], dd, rd);
            const double xj = e.cell[j], yj = e.cell[n + j];
            const double a = x * nx + y * ny, b = xj * nx + yj * ny;
            // upwind sign rule in the face-normal basis, tangential part interpolated
            const double un = (a > 0. && b > 0.) ? a : ((a < 0. && b < 0.) ? b : .5 * (a + b));
            const double ut = wo * (-x * ny + y * nx) + wj * (-xj * ny + yj * nx);
            x = un * nx - ut * ny; y = un * ny + ut * nx;
            gx = wo * gx + wj * e.gz[j]; gy = wo * gy + wj * e.gz[n + j];
            const double dx = e.xy[j] - e.xy[o], dy = e.xy[n + j] - e.xy[n + o], dn = dx * nx + dy * ny;
            const double correction = quotient(z[j] - z[o] - gx * dx - gy * dy, dn, reciprocal(dn));
            gx += correction * nx; gy += correction * ny;
            stress = wo * stress + wj * e.cell[2 * n + j];
        } else {
            const double normal_slope = gx * nx + gy * ny;
            gx -= normal_slope * nx; gy -= normal_slope * ny;
        }
        double cx, cy;
        if (slope_ks3(x, y, -gx, -gy, stress, cx, cy)) atomicOr(&e.bad[sid], 1);
        double fl = (cx * nx + cy * ny) / 2650.;
        if (j < 0) {
            const int bc = e.bedbc[f];
            if (bc == 1) fl = -e.feed[f];
            else if (bc == 2) fl = fmax(0., fl);
            else if (bc != 3) fl = 0.;
        }
        // no bed flux across a face with a dry side
        const bool active = e.wet[o] && (j >= 0 ? e.wet[j] : true);
        e.flux[f] = fl * (active ? 1. : 0.);
    }
}

__global__ void __launch_bounds__(256) k_ex_donor(MeshDev m, ExnerDev e, const double *z)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m.nc; i += gridDim.x * blockDim.x) {
        const int sid = m.cell_sid[i];
        if (!e.enabled[sid]) continue;
        const double *p = e.param + (size_t)sid * EP_N;
        const double dtm = e.dt[sid] * p[EP_MORFAC], phi = 1.0 - p[EP_POROSITY];
        double outgoing = 0.;
        for (int k = m.offset[i]; k < m.offset[i + 1]; ++k) {
            const int f = m.faces[k];
            outgoing += fmax(0., m.signs[k] * e.flux[f]) * m.length[f];
        }
        const double available = phi * (z[i] - e.rock[i]);
        e.fac[i] = outgoing > 0. ? fmin(1., fmax(0., available) * m.area[i] / (dtm * outgoing)) : 1.;
    }
}

// A face's flux limited by its donor's factor.
__device__ __forceinline__ double limited_flux(const MeshDev &m, const ExnerDev &e, int f)
{
    const double flux = e.flux[f];
    const int j = flux >= 0. ? m.owner[f] : m.neighbour[f];
    return j >= 0 ? flux * e.fac[j] : flux;
}

// Trial bed of a chunk of one scenario's cells, and the scenario's checks:
// budget residual, boundary volume, donor minimum, relative change, positivity
// and finiteness, in a fixed order (threads by a halving tree, then the chunks
// in order).
constexpr int EX_CHUNK = 1024;
__host__ __device__ __forceinline__ int exner_blocks(int cells) { return (cells + EX_CHUNK - 1) / EX_CHUNK; }

__global__ void __launch_bounds__(256) k_ex_trial(MeshDev m, ExnerDev e, BoundaryDev b, const double *q, const double *z)
{
    __shared__ double red[3][256];
    __shared__ bool last;
    const int sid = e.chunk_sid[blockIdx.x], tid = threadIdx.x;
    if (!e.enabled[sid]) return;
    const int c0 = m.act.cell_off[sid], c1 = m.act.cell_off[sid + 1], blocks = exner_blocks(c1 - c0);
    const double *p = e.param + (size_t)sid * EP_N;
    const double dtm = e.dt[sid] * p[EP_MORFAC], phi = 1.0 - p[EP_POROSITY], sd = p[EP_SEDDEPTH], scale = dtm / phi;
    double res = 0., donor = 1., change = 0.;
    bool wrong = false;
    const int from = c0 + ((int)blockIdx.x - e.first[sid]) * EX_CHUNK, to = min(c1, from + EX_CHUNK);
    for (int i = from + tid; i < to; i += blockDim.x) {
        double r = 0.;
        for (int k = m.offset[i]; k < m.offset[i + 1]; ++k) {
            const int f = m.faces[k];
            r -= m.signs[k] * m.length[f] * limited_flux(m, e, f);
        }
        const double area = m.area[i];
        r = r / area;
        const double zi = z[i], zt = zi + scale * r, moved = fabs(zt - zi), deep = q[i] > sd ? q[i] : sd;
        e.ztrial[i] = zt;
        if (!finite_bits(zt) || zt < e.rock[i] - 1e-13) wrong = true;
        res += phi * (zt - zi) * area;
        donor = fmin(donor, e.fac[i]);
        if (greater(moved, change * deep * (1. - 8. * EPS))) change = fmax(change, moved / deep);
    }
    red[0][tid] = res; red[1][tid] = donor; red[2][tid] = change;
    const bool any_wrong = __syncthreads_or(wrong);
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (tid < w) {
            red[0][tid] += red[0][tid + w];
            red[1][tid] = fmin(red[1][tid], red[1][tid + w]); red[2][tid] = fmax(red[2][tid], red[2][tid + w]);
        }
        __syncthreads();
    }
    if (tid == 0) {
        double *o = e.part + 3 * (size_t)blockIdx.x;
        o[0] = red[0][0]; o[1] = red[1][0]; o[2] = red[2][0];
        if (any_wrong) atomicOr(&e.out_of_range[sid], 1);
        __threadfence();
        last = atomicInc(&e.tickets[sid], blocks - 1) == (unsigned)(blocks - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the boundary volume over the open faces, then the chunks
    double bnd = 0.;
    const int s0 = b.scen_seg[sid], s1 = b.scen_seg[sid + 1];
    if (s1 > s0)
        for (int k = b.seg_off[s0] + tid; k < b.seg_off[s1]; k += blockDim.x) {
            const int f = b.slot_face[k];
            bnd -= dtm * limited_flux(m, e, f) * m.length[f];
        }
    res = 0.; donor = 1.; change = 0.;
    const volatile double *part = e.part + 3 * (size_t)e.first[sid];
    for (int k = tid; k < blocks; k += blockDim.x) {
        res += part[3 * k];
        donor = fmin(donor, part[3 * k + 1]); change = fmax(change, part[3 * k + 2]);
    }
    __shared__ double sum[256];
    red[0][tid] = res; red[1][tid] = donor; red[2][tid] = change; sum[tid] = bnd;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (tid < w) {
            red[0][tid] += red[0][tid + w]; sum[tid] += sum[tid + w];
            red[1][tid] = fmin(red[1][tid], red[1][tid + w]); red[2][tid] = fmax(red[2][tid], red[2][tid + w]);
        }
        __syncthreads();
    }
    if (tid == 0) {
        double *s = e.stats + (size_t)sid * ES_N;
        const double residual = red[0][0] - sum[0];
        const bool slope_bad = e.bad[sid] != 0, range_bad = *(volatile int *)&e.out_of_range[sid] != 0;
        s[ES_OK] = (!range_bad && !slope_bad && fabs(residual) <= 1e-10 && red[2][0] <= .05) ? 1. : 0.;
        s[ES_RESIDUAL] = residual; s[ES_BOUNDARY] = sum[0]; s[ES_DONOR] = red[1][0]; s[ES_CHANGE] = red[2][0];
        s[ES_BAD] = slope_bad ? 1. : 0.;
    }
}

__global__ void __launch_bounds__(256) k_ex_commit(MeshDev m, ExnerDev e, double *z)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m.nc; i += gridDim.x * blockDim.x) {
        const int sid = m.cell_sid[i];
        if (e.enabled[sid] && e.stats[(size_t)sid * ES_N + ES_OK] != 0.) z[i] = e.ztrial[i];
    }
}

}  // namespace brx
