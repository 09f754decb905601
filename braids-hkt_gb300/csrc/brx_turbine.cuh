// Rotor arrays: Thetis actuator-disk sink, coverage gate, diagnostics and the
// balanced-pressure / ambient-stress face terms. FP64 in both arithmetic
// forms (turbine power is integrated in FP64); compiled in the FP64 unit
// without FMA contraction so the operation order follows the reference:
//
//   wet gradients       src/braids_core/sediment/river_turbine_flow.h:13-37
//   rotor sample        river_turbine_thetis.py:263-297 (ThetisRotor.sample)
//   coverage gate       river_turbine_flow.py:82-120 (CoveredRotor._operating_state)
//   cut-in              river_turbine_thetis.py:219-241 (stop_below_cut_in)
//   cell terms          river_turbine_thetis.py:175-216 (cell_terms, lookup)
//   sink                river_turbine_thetis.py:356-362 (ThetisArray.apply)
//   balanced pressure   river_turbine_flow.h:54-82
//   ambient stress      river_hydrokinetic_stress.h:13-35
//
// One CTA per rotor reduces its support and rotor-plane samples (a handful of
// cells), decides the operating state and writes the per-cell sink
// coefficients; the sink itself is formed per support cell, summing the
// rotors that cover the cell in rotor order.
#pragma once
#include "brx_num64.cuh"

namespace brx {

enum { TD_ACTIVE = 0, TD_REASON, TD_MARGIN, TD_CLEARANCE, TD_U1, TD_U0, TD_DEPTH, TD_CT, TD_CP, TD_FORCE,
       TD_POWER, TD_REMOVED, TD_LOW, TD_HIGH, TD_ERROR, TD_N = 16 };
enum { TP_D = 0, TP_HUB, TP_BEDCLEAR, TP_SURFCLEAR, TP_TOL, TP_MODE, TP_CT, TP_CP, TP_N };
enum { TM_CONSTANT = 0, TM_SPEED_TABLE = 1, TM_INCIDENT_TABLE = 2, TM_INCIDENT_CURVES = 3 };
enum { TR_COVERED = 0, TR_DEPTH, TR_BED, TR_SURFCLEAR, TR_BEDCLEAR, TR_DRY, TR_REVERSE, TR_NOFLOW, TR_CUTIN };
constexpr double PI_D = 3.14159265358979323846;
constexpr int TURB_THREADS = 128;

// Weighted centre offsets of the flow metric: (1 / |d|^2) d per CSR entry.
__global__ void __launch_bounds__(256) k_flow_weights(int na, const double *dxdy, double *out)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < na; k += gridDim.x * blockDim.x) {
        const double dx = dxdy[k], dy = dxdy[na + k], w = 1. / (dx * dx + dy * dy);
        out[k] = w * dx; out[na + k] = w * dy;
    }
}

// Wet-only least-squares gradients of u, v and eta (fully wet pairs) of every
// cell of scenarios with rotors: rows u_x u_y v_x v_y eta_x eta_y. prim: the
// stage input's primitives, or null (formed per use).
__global__ void __launch_bounds__(256) k_hkt_gradients(MeshDev m, TurbDev t, const double *q, const double *z,
                                                       Ctrl *ctrl, int stage, const Prim64 *prim)
{
    const int n = m.nc, na = m.nadj;
    FOR_ACTIVE_CELLS(m.act, i) {
        const int sid = m.cell_sid[i];
        if (!t.hkt[sid]) continue;
        const Ctrl &ct = ctrl[sid];
        if (stage && skip_stage(ct, stage)) continue;
        const double dry = ct.dry;
        const auto cell = [&](int j) {
            if (prim) return prim[j];
            Prim64 p;
            p.h = q[j]; p.eta = q[j] + z[j]; p.u = p.v = 0.;
            if (greater(p.h, dry)) { p.u = q[n + j] / p.h; p.v = q[2 * n + j] / p.h; }
            return p;
        };
        const Prim64 own = cell(i);
        double xx = 0., xy = 0., yy = 0., bx[3] = {0., 0., 0.}, by[3] = {0., 0., 0.}, g[6] = {0., 0., 0., 0., 0., 0.};
        if (greater(own.h, dry)) {
            for (int s = m.offset[i]; s < m.offset[i + 1]; ++s) {
                const int f = m.faces[s];
                const int j = m.signs[s] < 0 ? m.owner[f] : m.neighbour[f];
                if (j < 0) continue;
                const Prim64 o = cell(j);
                if (!greater(o.h, dry)) continue;
                // weight 1 / |d|^2 of the flow metric's centre offset
                const double dx = t.dxdy[s], dy = t.dxdy[na + s], wx = t.wdxdy[s], wy = t.wdxdy[na + s];
                xx += wx * dx; xy += wx * dy; yy += wy * dy;
                const double d[3] = {o.u - own.u, o.v - own.v, o.eta - own.eta};
#pragma unroll
                for (int k = 0; k < 3; ++k) { bx[k] += wx * d[k]; by[k] += wy * d[k]; }
            }
            const double det = xx * yy - xy * xy, size = xx * yy;
            if (greater(det, 1e-12 * (greater(size, 1.) ? size : 1.))) {
                const double r = reciprocal(det);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    g[2 * k] = quotient(yy * bx[k] - xy * by[k], det, r);
                    g[2 * k + 1] = quotient(xx * by[k] - xy * bx[k], det, r);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) t.grad[k * n + i] = g[k];
    }
}

// numpy.interp on one table, zero outside [x0, xlast); the knot slopes
// (y[k+1]-y[k])/(x[k+1]-x[k]) are precomputed with the same division
__device__ __forceinline__ double table_lookup(const double *x, const double *y, const double *slope, int count,
                                               double v)
{
    if (!(v >= x[0]) || v >= x[count - 1]) return 0.;
    int lo = 0, hi = count - 1;           // x[lo] <= v < x[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (greater(x[mid], v)) hi = mid; else lo = mid;
    }
    if (v == x[lo]) return y[lo];
    return slope[lo] * (v - x[lo]) + y[lo];
}

// Thetis terms of one cell of speed |u|: K, P, incident speed U, Ct, Cp.
// Returns 0 or an error code.
__device__ int rotor_cell_terms(const TurbDev &t, int r, double depth, double speed, double out[5])
{
    const double *p = t.param + (size_t)r * TP_N;
    const double D = p[TP_D];
    const int mode = (int)p[TP_MODE];
    const int *cv = t.curve + 4 * r;
    const double *tx = t.curve_x + cv[0], *ty = t.curve_y + cv[0], *ts = t.curve_slope + cv[0];
    const double *px = t.curve_x + cv[2], *py = t.curve_y + cv[2], *ps = t.curve_slope + cv[2];
    const double area = PI_D * (D * D) / 4;
    double ct, cp, alpha, incident;
    if (mode == TM_INCIDENT_TABLE || mode == TM_INCIDENT_CURVES) {
        if (depth < D * (1 - 1e-10)) return 2;
        const double d4 = 4 * depth, c = quotient(PI_D * D, d4, reciprocal(d4));
        const double first = tx[0], last = tx[cv[1] - 1];
        double low = first, high = last;
        const double in_table = .5 * (1 + sqrt(1 - c * ty[0]));
        const double smin = low * in_table;
        const double smax = high * (t.flat_thrust[r] ? in_table : .5 * (1 + sqrt(1 - c * ty[cv[1] - 1])));
        const bool active = speed >= smin && speed < smax;
        // induction-corrected operating point: bisection on the incident speed
        if (!active) incident = speed;
        else {
            if (t.flat_thrust[r]) {
                // constant Ct: inside the table the local speed is mid x in_table,
                // beyond it mid. Products by a constant are monotone, so the test
                // is mid < edge, the least number whose product reaches the speed:
                // one addition a step is left on the FP64 pipe
                double edge = quotient(speed, in_table, reciprocal(in_table));
                while (edge * in_table < speed) edge = unordered(ordered(edge) + 1);
                while (unordered(ordered(edge) - 1) * in_table >= speed) edge = unordered(ordered(edge) - 1);
                for (int it = 0; it < 44; ++it) {
                    const double sum = low + high;
                    const double mid = __hiloint2double(__double2hiint(sum) - 0x00100000, __double2loint(sum));   // / 2
                    if (greater(greater(last, mid) ? edge : speed, mid)) low = mid; else high = mid;
                }
            } else {
                for (int it = 0; it < 44; ++it) {
                    const double mid = .5 * (low + high);
                    const double local = mid * .5 * (1 + sqrt(1 - c * table_lookup(tx, ty, ts, cv[1], mid)));
                    if (greater(speed, local)) low = mid; else high = mid;
                }
            }
            incident = .5 * (low + high);
        }
        ct = active ? table_lookup(tx, ty, ts, cv[1], incident) : 0.;
        cp = active ? table_lookup(px, py, ps, cv[3], incident) : 0.;
        alpha = ct == ty[0] ? in_table : .5 * (1 + sqrt(1 - c * ct));
    } else {
        ct = mode == TM_CONSTANT ? p[TP_CT] : table_lookup(tx, ty, ts, cv[1], speed);
        const double disk = D * depth, radicand = 1 - quotient(area * ct, disk, reciprocal(disk));
        if (radicand < 0) return 1;
        alpha = .5 * (1 + sqrt(radicand));
        incident = quotient(speed, alpha, reciprocal(alpha));
        cp = mode == TM_CONSTANT ? p[TP_CP] : table_lookup(px, py, ps, cv[3], incident);
    }
    const double a2 = 2 * (alpha * alpha);
    out[0] = quotient(area * ct, a2, reciprocal(a2));
    out[1] = .5 * area * cp * (incident * incident * incident);
    out[2] = incident; out[3] = ct; out[4] = cp;
    return 0;
}

// Sums of N values over the block in the order of a halving tree (thread t with
// t + 64, then t + 32, 16, ... 1), a warp per row; every thread gets them.
template <int N>
__device__ __forceinline__ void block_sum(double (*s)[TURB_THREADS], double *out, double (&v)[N])
{
    const int tid = threadIdx.x, lane = tid & 31;
#pragma unroll
    for (int k = 0; k < N; ++k) s[k][tid] = v[k];
    __syncthreads();
    for (int k = tid >> 5; k < N; k += TURB_THREADS / 32) {
        double a = (s[k][lane] + s[k][lane + 64]) + (s[k][lane + 32] + s[k][lane + 96]);
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) a += __shfl_down_sync(0xffffffffu, a, w);
        if (lane == 0) out[k] = a;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = out[k];
}

// Surface and bed slopes of a rotor-plane cell: the wet least-squares gradient
// of the surface and the unweighted-metric gradient of the bed
// (river_turbine_flow.h:13-37).
__device__ __forceinline__ void plane_gradient(const MeshDev &m, const TurbDev &t, const double *q, const double *z,
                                               double dry, int i, double &ex, double &ey, double &zx, double &zy)
{
    const int n = m.nc, na = m.nadj;
    const double hi = q[i], zi = z[i], etai = hi + zi;
    const bool wet = greater(hi, dry);
    double xx = 0., xy = 0., yy = 0., bx = 0., by = 0., cx = 0., cy = 0.;
    for (int s = m.offset[i]; s < m.offset[i + 1]; ++s) {
        const int f = m.faces[s];
        const int j = m.signs[s] < 0 ? m.owner[f] : m.neighbour[f];
        if (j < 0) continue;
        const double dx = t.dxdy[s], dy = t.dxdy[na + s], d2 = dx * dx + dy * dy, w = quotient(1., d2, reciprocal(d2));
        const double wx = w * dx, wy = w * dy, hj = q[j], zj = z[j], dz = zj - zi;
        cx += wx * dz; cy += wy * dz;
        if (!wet || !greater(hj, dry)) continue;
        xx += wx * dx; xy += wx * dy; yy += wy * dy;
        const double d = (hj + zj) - etai;
        bx += wx * d; by += wy * d;
    }
    zx = t.inverse[i] * cx + t.inverse[n + i] * cy;
    zy = t.inverse[n + i] * cx + t.inverse[2 * n + i] * cy;
    ex = ey = 0.;
    const double det = xx * yy - xy * xy;
    if (det > 1e-12 * fmax(1., xx * yy)) {
        const double r = reciprocal(det);
        ex = quotient(yy * bx - xy * by, det, r);
        ey = quotient(xx * by - xy * bx, det, r);
    }
}

// One rotor per CTA: plane and support samples, the operating state, the sink
// coefficients and the rotor's diagnostics. stage 0 samples a state outside a
// trial (no skip, no status). A serial chain of FP64 phases on one SM bounds
// it: a support cell's state and speed are formed once and kept, the trees run
// a row per warp, extremes on integer images.
// Per launch, before -> after (events): two rotors of constant Ct 26 -> 19 us,
// the batch's rotors with incident-speed curves 53 -> 32 us.
__global__ void __launch_bounds__(TURB_THREADS) k_turbine_sample(MeshDev m, TurbDev t, const double *q,
                                                                 const double *z, Ctrl *ctrl, int stage, double *diag)
{
    __shared__ double red[6][TURB_THREADS], total[6];
    __shared__ long long extreme[2][TURB_THREADS / 32];
    const int r = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int sid = t.rotor_sid[r];
    Ctrl &ct = ctrl[sid];
    if (stage && skip_stage(ct, stage)) return;      // uniform over the CTA
    const int n = m.nc, np_ = t.np;
    const double dry = ct.dry;
    const int e0 = t.support_offset[r] + tid, e1 = t.support_offset[r + 1];
    struct Support { int c; double h, u, v, speed; };
    const auto support = [&](int e) {
        Support o;
        o.c = t.support_cell[e];
        o.h = q[o.c];
        const double d = greater(o.h, dry) ? o.h : dry, rd = reciprocal(d);
        o.u = quotient(q[n + o.c], d, rd); o.v = quotient(q[2 * n + o.c], d, rd);
        o.speed = hypot(o.u, o.v);
        return o;
    };
    Support own{};                                   // this thread's first support cell
    if (e0 < e1) own = support(e0);
    const double *p = t.param + (size_t)r * TP_N;
    const double D = p[TP_D], tol = p[TP_TOL];
    const double top = p[TP_HUB] + D / 2, bottom = p[TP_HUB] - D / 2;
    const int mode = (int)p[TP_MODE];
    const int *cv = t.curve + 4 * r;
    // rotor plane: lowest surface, highest bed
    long long low_key = ordered(INFINITY), high_key = ordered(-INFINITY);
    for (int j = t.plane_offset[r] + tid; j < t.plane_offset[r + 1]; j += TURB_THREADS) {
        const int c = t.plane_cell[j];
        double ex, ey, zx, zy;
        plane_gradient(m, t, q, z, dry, c, ex, ey, zx, zy);   // the plane cell's own gradients, FP64
        const double zc = z[c], eta = q[c] + zc, px = t.plane_delta[j], py = t.plane_delta[np_ + j];
        low_key = min(low_key, min(ordered(eta + ex * px + ey * py), ordered(eta)));
        high_key = max(high_key, max(ordered(zc + zx * px + zy * py), ordered(zc)));
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        low_key = min(low_key, __shfl_xor_sync(0xffffffffu, low_key, w));
        high_key = max(high_key, __shfl_xor_sync(0xffffffffu, high_key, w));
    }
    if (lane == 0) { extreme[0][warp] = low_key; extreme[1][warp] = high_key; }
    // support: dry cells, weighted speed and depth, cut-in
    double sums[2] = {0., 0.};
    bool support_dry = false, below = false;
    for (int e = e0; e < e1; e += TURB_THREADS) {
        const Support o = e == e0 ? own : support(e);
        const double w = t.support_weight[e];
        if (!greater(o.h, dry)) support_dry = true;
        sums[0] += w * o.speed; sums[1] += w * o.h;
        t.kcell[e] = 0.;
        if (mode != TM_CONSTANT) {
            double minimum = t.curve_x[cv[0]];
            if (mode != TM_SPEED_TABLE) {
                const double h4 = 4 * o.h;
                minimum = minimum * .5 * (1 + sqrt(1 - quotient(PI_D * D * t.curve_y[cv[0]], h4, reciprocal(h4))));
            }
            if (o.speed < minimum) below = true;
        }
    }
    support_dry = __syncthreads_or(support_dry);
    below = __syncthreads_or(below);
    block_sum<2>(red, total, sums);
    double low = unordered(extreme[0][0]), high = unordered(extreme[1][0]);
#pragma unroll
    for (int w = 1; w < TURB_THREADS / 32; ++w) {
        low = unordered(min(ordered(low), extreme[0][w]));
        high = unordered(max(ordered(high), extreme[1][w]));
    }
    const double u1 = sums[0], depth = sums[1];
    const double margin = low - top, clearance = bottom - high;
    int reason = TR_COVERED;
    if (margin < tol) reason = TR_DEPTH;
    else if (clearance < tol) reason = TR_BED;
    else if (margin + tol < p[TP_SURFCLEAR]) reason = TR_SURFCLEAR;
    else if (clearance + tol < p[TP_BEDCLEAR]) reason = TR_BEDCLEAR;
    else if (support_dry) reason = TR_DRY;
    bool active = reason == TR_COVERED;
    if (active && u1 <= 1e-10) { active = false; reason = u1 < 0 ? TR_REVERSE : TR_NOFLOW; }
    if (active && mode != TM_CONSTANT && below) { active = false; reason = TR_CUTIN; }
    double out[6] = {0., 0., 0., 0., 0., 0.};   // F, removed, P, incoming, Ct, Cp
    int error = 0;
    double kown = 0.;                           // this thread's first coefficient
    if (active) {
        for (int e = e0; e < e1; e += TURB_THREADS) {
            const Support o = e == e0 ? own : support(e);
            const double w = t.support_weight[e], density = t.support_density[e];
            double k[5];
            const int failed = rotor_cell_terms(t, r, o.h, o.speed, k);
            if (failed) { error = max(error, failed); continue; }
            const double area = m.area[o.c], kc = quotient(k[0] * density, area, reciprocal(area));
            t.kcell[e] = kc;
            if (e == e0) kown = kc;
            out[0] += k[0] * density * (o.speed * o.speed);
            out[1] += k[0] * density * (o.speed * o.speed * o.speed);
            out[2] += k[1] * density;
            out[3] += w * k[2]; out[4] += w * k[3]; out[5] += w * k[4];
        }
    }
    // actuator sink of the support cells no other rotor's support holds:
    // 0 - k |u| u from this rotor alone (k_turbine_raw's sum with one term)
    if (stage)
        for (int e = e0; e < e1; e += TURB_THREADS) {
            if (!t.single[e]) continue;
            const Support o = e == e0 ? own : support(e);
            const double kc = e == e0 ? kown : t.kcell[e];
            double rx = 0., ry = 0.;
            rx -= kc * o.speed * o.u;
            ry -= kc * o.speed * o.v;
            t.raw[o.c] = rx; t.raw[n + o.c] = ry;
        }
    if (active) {
        if (__syncthreads_or(error))
            for (int level = 2; level >= 1; --level)
                if (__syncthreads_or(error == level)) { error = level; break; }
        block_sum<6>(red, total, out);
    }
    if (tid == 0) {
        double *d = diag + (size_t)r * TD_N;
        for (int k = 0; k < TD_N; ++k) d[k] = 0.;
        d[TD_ACTIVE] = active; d[TD_REASON] = reason; d[TD_MARGIN] = margin; d[TD_CLEARANCE] = clearance;
        d[TD_U1] = u1; d[TD_U0] = active ? out[3] : u1; d[TD_DEPTH] = depth; d[TD_LOW] = low; d[TD_HIGH] = high;
        if (active) {
            d[TD_FORCE] = out[0]; d[TD_REMOVED] = out[1]; d[TD_POWER] = out[2];
            d[TD_CT] = out[4]; d[TD_CP] = out[5];
        }
        d[TD_ERROR] = error;
        if (error && stage) raise_status(ct, stage, ST_TURBINE);
    }
}

// Actuator sink per support cell: 0 - sum over its rotors of k |u| u.
__global__ void __launch_bounds__(256) k_turbine_raw(MeshDev m, TurbDev t, const double *q, Ctrl *ctrl, int stage)
{
    const int n = m.nc;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < t.nucell; i += gridDim.x * blockDim.x) {
        const int c = t.ucell[i];
        const Ctrl &ct = ctrl[m.cell_sid[c]];
        if (stage && skip_stage(ct, stage)) continue;
        const double h = q[c], u = q[n + c] / fmax(h, ct.dry), v = q[2 * n + c] / fmax(h, ct.dry);
        const double speed = hypot(u, v);
        double rx = 0., ry = 0.;
        for (int k = t.uoff[i]; k < t.uoff[i + 1]; ++k) {
            const double kc = t.kcell[t.uent[k]];
            rx -= kc * speed * u;
            ry -= kc * speed * v;
        }
        t.raw[c] = rx; t.raw[n + c] = ry;
    }
}

// Symmetric-strain ambient stress of an interior face between two wet cells.
__device__ __forceinline__ void rotor_stress(const MeshDev &m, const TurbDev &t, const double *q, const double *z, int i,
                                             int a, int b, double nx, double ny, double &ox, double &oy)
{
    const int nf = m.nf, n = m.nc;
    double h = fmin(q[a], q[b]);
    h = fmin(h, fmax(0., .5 * (q[a] + z[a] + q[b] + z[b]) - fmax(z[a], z[b])));
    const double da = m.distance[i], db = m.distance[nf + i], d = da + db, wo = db / d, wj = da / d;
    const double visc = wo * t.nu[a] + wj * t.nu[b];
    const double dx = t.xy[b] - t.xy[a], dy = t.xy[n + b] - t.xy[n + a];
    const double dn = dx * nx + dy * ny;
    const double du = q[n + b] / q[b] - q[n + a] / q[a], dv = q[2 * n + b] / q[b] - q[2 * n + a] / q[a];
    double ux = wo * t.grad[a] + wj * t.grad[b], uy = wo * t.grad[n + a] + wj * t.grad[n + b];
    double vx = wo * t.grad[2 * n + a] + wj * t.grad[2 * n + b], vy = wo * t.grad[3 * n + a] + wj * t.grad[3 * n + b];
    const double cu = (du - ux * dx - uy * dy) / dn, cvv = (dv - vx * dx - vy * dy) / dn;
    ux += cu * nx; uy += cu * ny; vx += cvv * nx; vy += cvv * ny;
    ox = visc * h * (2. * ux * nx + (uy + vx) * ny);
    oy = visc * h * ((uy + vx) * nx + 2. * vy * ny);
}

// Ambient stress of the HLLC owner's scenarios (the f-wave owner's is formed
// in its face sweep).
__global__ void __launch_bounds__(128) k_hkt_stress(MeshDev m, TurbDev t, const double *q, const double *z, Ctrl *ctrl,
                                                    int stage)
{
    const int nf = m.nf;
    FOR_ACTIVE_FACES(m.act, i) {
        const int sid = m.face_sid[i];
        if (!t.hkt[sid] || !t.stress[sid]) continue;
        const Ctrl &ct = ctrl[sid];
        if (stage && skip_stage(ct, stage)) continue;
        const int a = m.owner[i], b = m.neighbour[i];
        double ox = 0., oy = 0.;
        if (b >= 0 && q[a] > ct.dry && q[b] > ct.dry) rotor_stress(m, t, q, z, i, a, b, m.normal[i], m.normal[nf + i], ox, oy);
        t.sface[i] = ox; t.sface[nf + i] = oy;
    }
}

// Balanced pressure correction of an interior face between two wet cells
// (river_turbine_flow.h:54-82), from the cells' depths, stages and beds, the
// face's reconstructed depths sl, sr over the common bed top, its normal
// velocities and speeds. Returns the magnitude along the normal, zero outside
// the fully wet, small-surface-jump, consistent-pressure scope.
struct FaceTrace { double hl, hr, top, ul, ur, hul, hvl, hur, hvr; };
__device__ __forceinline__ double balanced_pressure(const MeshDev &m, const TurbDev &t, int i, int a, int b,
                                                    const CellRec &ra, const CellRec &rb, const FaceTrace &s,
                                                    double gravity, double dry, double nx, double ny)
{
    const int n = m.nc, nf = m.nf;
    const double zmax = greater(ra.b, rb.b) ? ra.b : rb.b, bed = greater(s.top, zmax) ? s.top : zmax;
    const double ha = ra.eta - bed, hb = rb.eta - bed, hl = (s.hl + s.top) - bed, hr = (s.hr + s.top) - bed;
    if (!greater(ha, dry) || !greater(hb, dry) || !greater(hl, dry) || !greater(hr, dry)) return 0.;
    const double h = .5 * (hl + hr);
    if (magnitude(hr - hl) > __double_as_longlong(.005 * h)) return 0.;
    const double l2 = hl * hl, r2 = hr * hr, old = .25 * gravity * (l2 + r2);
    double po = old, pn = old;
    if (ra.flags & 1) po += .5 * gravity * (ha * ha - l2);
    if (rb.flags & 1) pn += .5 * gravity * (hb * hb - r2);
    if (po != pn && fabs(po - pn) > 128. * EPS * fmax(1., fmax(fabs(po), fabs(pn)))) return 0.;
    const double da = m.distance[i], db = m.distance[nf + i], d = da + db, rd = reciprocal(d);
    const double wa = quotient(db, d, rd), wb = quotient(da, d, rd);
    const double sx = wa * t.mdisp[i] + wb * t.mdisp[2 * nf + i];
    const double sy = wa * t.mdisp[nf + i] + wb * t.mdisp[3 * nf + i];
    double pressure = .5 * gravity * (wa * ha * ha + wb * hb * hb);
    pressure += gravity * sx * (wa * ha * t.grad[4 * n + a] + wb * hb * t.grad[4 * n + b]);
    pressure += gravity * sy * (wa * ha * t.grad[5 * n + a] + wb * hb * t.grad[5 * n + b]);
    // the actuator sink is zero outside the rotors' support cells
    if (t.foot[a] | t.foot[b])
        pressure += quotient(da * db, d, rd) * ((t.raw[a] - t.raw[b]) * nx + (t.raw[n + a] - t.raw[n + b]) * ny);
    double delta = .5 * (po + pn) - pressure;
    const double rl = reciprocal(s.hl), rr = reciprocal(s.hr);
    const double al = quotient(hypot(s.hul, s.hvl), s.hl, rl), ar = quotient(hypot(s.hur, s.hvr), s.hr, rr);
    const double speed = sqrt(gravity * h), sum = hl + hr;
    double theta = quotient(greater(al, ar) ? al : ar, speed, reciprocal(speed));
    if (greater(theta, 1.)) theta = 1.;
    delta -= .5 * (1. - theta) * speed * quotient(2. * hl * hr, sum, reciprocal(sum)) * (s.ur - s.ul);
    return delta;
}

}  // namespace brx
