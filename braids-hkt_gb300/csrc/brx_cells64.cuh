// FP64 cell sweep of the f-wave step for cells of at most four faces, and the
// tables it reads. The records equal k_cells' (brx_kernels.cuh), which stays
// for cells of up to 32 faces and for the allocation-free residual.
//
// What bounds it: FP64 instructions. A GB300 sub-partition issues one FP64
// warp instruction every 64-76 clocks, whatever the parallelism (a DFMA chain
// measures 65 clocks per step from one warp, 76 per warp from sixteen warps
// per SM), so a sweep's time is its FP64 instruction count. A division or a
// square root is ten of them, fmax 2.3, a comparison 1.7, a conversion one;
// integer and FP32 instructions are some thirty times cheaper. k_cells spent
// about 1,350 FP64 issue slots per cell and up to 3,700 on a warp whose lanes
// took different branches. This sweep takes about 250:
//   * velocities are formed once per cell by the kernel that writes a stage's
//     input (prim), not again by each neighbour;
//   * the limited bed gradient depends on the bed alone (except beside a stage
//     outlet): a table, rebuilt from the bed at the start of every call;
//   * divisions by mesh constants use the stored correctly rounded reciprocal
//     and one exact remainder (quotient());
//   * minima, maxima, signs and thresholds are integer operations on the bit
//     patterns (ordered());
//   * the projection of the surface gradient is reached only where a product
//     form of its bounds cannot rule it out, and there an FP32 pass discards
//     the candidates that rounding cannot make nearest or feasible; the FP64
//     arithmetic of the rest is k_cells'.
// Per launch, before -> after (CUDA events): 360 cells 122 -> 33 us, 50k cells
// 227 -> 49 us, 302k cells 901 -> 190 us; squares, 4k cells 167 -> 41 us.
#pragma once
#include "brx_num64.cuh"

namespace brx {

struct Cells64 {
    double4_32a *ls;          // (nc) A, B, C, D: gradient = ((A bx + B by) / D, (B bx + C by) / D); D = 0: none
    double *lsr;              // (nc) RN(1 / D)
    int2 *cidx;               // (nadj) other cell (-1 none); flags bit0 open face, bit1 stage outlet, bit2 wall
    int *ccls;                // (nc) bit0 the cell has a stage outlet face
    unsigned char *par;       // (nc) bit per pair of entries (0,1) (0,2) (1,2) (0,3) (1,3) (2,3): parallel
    double4_32a *ent;         // (nadj) LS weight * offset x, y; face displacement x, y
    double4_32a *unit;        // (nadj) displacement direction x, y, its length, RN(1 / length)
    double2 *gbed;            // (nc) limited bed gradient
    Prim64 *prim[2];          // (nc) primitives of the two stage inputs
};

// The mesh tables of Cells64 (at set-up, and when the boundary modes change).
__global__ void __launch_bounds__(256) k64_tables(MeshDev m, Cells64 g)
{
    const int nc = m.nc, nf = m.nf;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        const double a11 = m.ls_matrix[c], a12 = m.ls_matrix[nc + c], a22 = m.ls_matrix[2 * nc + c],
                     det = m.ls_matrix[3 * nc + c], tr = a11 + a22;
        double4_32a v = make_double4_32a(0., 0., 0., 0.);
        if (tr > 0.0)
            v = det > 1.e-12 * (tr * tr) ? make_double4_32a(a22, -a12, a11, det) : make_double4_32a(a11, a12, a22, tr * tr);
        g.ls[c] = v;
        g.lsr[c] = v.w != 0. ? 1. / v.w : 0.;
        int cls = 0;
        unsigned par = 0u;
        const int k0 = m.offset[c], deg = m.offset[c + 1] - k0;
        for (int e = 0; e < deg; ++e) {
            const int k = k0 + e, f = m.faces[k], nb = m.neighbour[f];
            const bool own = m.signs[k] > 0;
            const size_t a = own ? f : (size_t)nf + f, b = a + 2 * (size_t)nf;
            int flags = 0;
            if (m.bid[f] >= 0) flags |= 1;
            if (nb < 0 && m.bmode[f] == 2) { flags |= 2; cls = 1; }
            if (nb < 0 && m.bid[f] < 0) flags |= 4;
            g.cidx[k] = make_int2(own ? nb : m.owner[f], flags);
            g.ent[k] = make_double4_32a(m.ls_weight[k] * m.ls_delta[k], m.ls_weight[k] * m.ls_delta[m.nadj + k],
                                        m.disp[a], m.disp[b]);
            const double len = m.disp_len[a], ux = m.disp_unit[a], uy = m.disp_unit[b];
            g.unit[k] = make_double4_32a(ux, uy, len, len > 0. ? 1. / len : 0.);
            for (int o = 0; o < e; ++o) {
                const int fo = m.faces[k0 + o];
                const size_t ao = m.signs[k0 + o] > 0 ? fo : (size_t)nf + fo;
                if (fabs(ux * m.disp_unit[ao + 2 * (size_t)nf] - uy * m.disp_unit[ao]) < 1.e-12)
                    par |= 1u << (e * (e - 1) / 2 + o);
            }
        }
        g.ccls[c] = cls;
        g.par[c] = (unsigned char)par;
    }
}

// The slabs -bm[j] <= u[j] . g <= bp[j] of one cell's entries.
template <int D>
struct Slab64 {
    double ux[D], uy[D], bp[D], bm[D];
    unsigned mask;            // enabled entries
    unsigned par;             // parallel pairs
};

template <int D>
__device__ __forceinline__ bool inside64(const Slab64<D> &S, double x, double y)
{
    bool ok = true;
#pragma unroll
    for (int j = 0; j < D; ++j)
        if (S.mask >> j & 1u) {
            const double t = S.ux[j] * x + S.uy[j] * y;
            if (greater(t, S.bp[j] + 2.e-14) || greater(-t, S.bm[j] + 2.e-14)) ok = false;
        }
    return ok;
}

// project_pair's result for the slabs of one cell: the first candidate of
// least distance among the projections on one side and the vertices of two,
// in its order and with its FP64 arithmetic. An FP32 pass over all candidates
// first discards those that are infeasible, or farther than one that is
// surely feasible, by more than the FP32 error of the comparison (bounds on
// inputs truncated to 2^-23, 1 / |det| for a vertex; vertices of nearly
// parallel sides are not judged). Two sides whose bounds are both zero meet in
// the origin, the starting candidate, and are skipped.
template <int D>
__device__ __noinline__ void project64(double &x, double &y, const Slab64<D> &S)
{
    constexpr int NC = 2 * D * D;            // 2D singles, 2D(D-1) pairs of different entries
    const double rx = x, ry = y;
    if (inside64<D>(S, rx, ry)) return;
    float fx = truncated(rx), fy = truncated(ry);
    float ux[D], uy[D], bp[D], bm[D];
#pragma unroll
    for (int j = 0; j < D; ++j) {
        ux[j] = truncated(S.ux[j]); uy[j] = truncated(S.uy[j]);
        bp[j] = truncated(S.bp[j]); bm[j] = truncated(S.bm[j]);
    }
    unsigned zero = 0u;                      // sides whose bound is exactly zero
#pragma unroll
    for (int j = 0; j < D; ++j) {
        if (__double_as_longlong(S.bp[j]) == 0) zero |= 1u << (2 * j);
        if (__double_as_longlong(S.bm[j]) == 0) zero |= 2u << (2 * j);
    }
    // least distance that cannot be improved on: the origin's, then any surely feasible candidate's
    float bound = sqrtf(fx * fx + fy * fy) * (1.f + 4.e-6f) + 1.e-30f;
    float low[NC];
    unsigned keep = 0u;
    int id = 0;
#pragma unroll
    for (int i = 0; i < 2 * D; ++i) {
        const int e = i >> 1;
        const float ax = i & 1 ? -ux[e] : ux[e], ay = i & 1 ? -uy[e] : uy[e], b = i & 1 ? bm[e] : bp[e];
#pragma unroll
        for (int j = -1; j < i; ++j) {
            if (j >= 0 && (j >> 1) == e) continue;                   // the slab's other side: parallel
            float cx, cy, err;
            bool use = S.mask >> e & 1u, judged = true;
            if (j < 0) {
                const float dot = ax * fx + ay * fy - b;
                cx = fx - dot * ax; cy = fy - dot * ay;
                err = 4.e-6f * (fabsf(fx) + fabsf(fy) + b);
            } else {
                const int o = j >> 1;
                const float jx = j & 1 ? -ux[o] : ux[o], jy = j & 1 ? -uy[o] : uy[o], jb = j & 1 ? bm[o] : bp[o];
                use = use && (S.mask >> o & 1u) && !(S.par >> (e * (e - 1) / 2 + o) & 1u) &&
                      !((zero >> i & 1u) && (zero >> j & 1u));
                const float det = ax * jy - ay * jx, inv = __fdividef(1.f, det);
                cx = (b * jy - ay * jb) * inv; cy = (ax * jb - b * jx) * inv;
                judged = fabsf(det) > .05f;
                err = 4.e-6f * (b + jb + fabsf(cx) + fabsf(cy)) * fabsf(inv);
            }
            const float dx = cx - fx, dy = cy - fy, dist = sqrtf(dx * dx + dy * dy);
            err = err + 4.e-6f * dist + 1.e-13f;
            float worst = -3.e38f;           // how far the other sides are exceeded
#pragma unroll
            for (int k = 0; k < D; ++k)
                if ((S.mask >> k & 1u) && k != e && (j < 0 || k != (j >> 1))) {
                    const float t = ux[k] * cx + uy[k] * cy;
                    worst = fmaxf(worst, fmaxf(t - bp[k], -t - bm[k]) - 2.e-6f * (bp[k] + bm[k]));
                }
            // the candidate's own slabs: the far side of each
            {
                const float t = ux[e] * cx + uy[e] * cy;
                const float far = i & 1 ? t - bp[e] : -t - bm[e];
                worst = fmaxf(worst, far - 2.e-6f * (bp[e] + bm[e]));
                if (j >= 0) {
                    const int o = j >> 1;
                    const float to = ux[o] * cx + uy[o] * cy;
                    const float faro = j & 1 ? to - bp[o] : -to - bm[o];
                    worst = fmaxf(worst, faro - 2.e-6f * (bp[o] + bm[o]));
                }
            }
            const bool out = judged && worst > 2.f * err;
            low[id] = judged ? dist - 2.f * err : 0.f;
            if (use && !out) {
                keep |= 1u << id;
                // surely feasible: clear of the other sides (their bounds' own
                // rounding was taken off above), small enough that FP64
                // rounding stays below the 2e-14 of its own sides
                float span = 0.f;
#pragma unroll
                for (int k = 0; k < D; ++k) span = fmaxf(span, bp[k] + bm[k]);
                if (judged && worst + 4.e-6f * span < -2.f * err && fabsf(cx) + fabsf(cy) + b < 1.f)
                    bound = fminf(bound, dist + 2.f * err);
            }
            ++id;
        }
    }
#pragma unroll
    for (int k = 0; k < NC; ++k)
        if (low[k] > bound) keep &= ~(1u << k);
    double bx = 0., by = 0., best = rx * rx + ry * ry;
    while (keep) {
        int k = __ffs(keep) - 1, i = 0;
        keep &= keep - 1u;
        // candidates of side i: its projection, then the vertices with the sides below it
        for (int n = 1; k >= n; n = 1 + i - (i & 1)) { k -= n; ++i; }
        const int e = i >> 1;
        const double ax = i & 1 ? -S.ux[e] : S.ux[e], ay = i & 1 ? -S.uy[e] : S.uy[e], b = i & 1 ? S.bm[e] : S.bp[e];
        double cx, cy;
        if (k == 0) {
            const double dot = ax * rx + ay * ry - b;
            cx = rx - dot * ax; cy = ry - dot * ay;
        } else {
            const int j = k - 1, o = j >> 1;
            const double jx = j & 1 ? -S.ux[o] : S.ux[o], jy = j & 1 ? -S.uy[o] : S.uy[o],
                         jb = j & 1 ? S.bm[o] : S.bp[o];
            const double det = ax * jy - ay * jx, r = 1. / det;
            cx = quotient(b * jy - ay * jb, det, r);
            cy = quotient(ax * jb - b * jx, det, r);
        }
        const double d = (cx - rx) * (cx - rx) + (cy - ry) * (cy - ry);
        if (__double_as_longlong(d) < __double_as_longlong(best) && inside64<D>(S, cx, cy)) { bx = cx; by = cy; best = d; }
    }
    x = bx; y = by;
}

// Whether g lies within every slab of half-widths hp / len (up) and hm / len
// (down) for certain: |u . g| len below the half-width by more than the
// rounding of both sides. Five FP64 instructions per entry, no division.
template <int D>
__device__ __forceinline__ bool surely_inside(const double4_32a (&U)[D], unsigned mask, double hp, double hm, double x,
                                              double y)
{
    bool ok = true;
#pragma unroll
    for (int j = 0; j < D; ++j)
        if (mask >> j & 1u) {
            const double t = U[j].x * x + U[j].y * y;
            const double room = __double_as_longlong(t) < 0 ? hm : hp;
            if (magnitude(t * (U[j].z * (1. + 8. * EPS))) > __double_as_longlong(room)) ok = false;
        }
    return ok;
}

// Limit (x, y) to the slabs; hp, hm >= 0 are the variable's room up and down.
template <int D>
__device__ __forceinline__ void limit64(double &x, double &y, const double4_32a (&U)[D], unsigned mask, unsigned par,
                                        double hp, double hm)
{
    if (surely_inside<D>(U, mask, hp, hm, x, y)) return;
    Slab64<D> S;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        const bool on = mask >> j & 1u;
        S.ux[j] = on ? U[j].x : 0.; S.uy[j] = on ? U[j].y : 0.;
        S.bp[j] = on ? quotient(hp, U[j].z, U[j].w) : 0.;
        S.bm[j] = on ? quotient(hm, U[j].z, U[j].w) : 0.;
    }
    S.mask = mask; S.par = par;
    project64<D>(x, y, S);
}

// Limited bed gradients of the bed as it is now (before the first stage of a call).
template <int D>
__global__ void __launch_bounds__(128) k64_bed(MeshDev m, Cells64 g, const double *z)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < m.nc; c += gridDim.x * blockDim.x) {
        const int k0 = m.offset[c], deg = m.offset[c + 1] - k0;
        const double zc = z[c];
        const double4_32a L = g.ls[c];
        double bx = 0., by = 0.;
        long long lo = ordered(zc), hi = lo;
        double4_32a U[D];
        unsigned mask = 0u;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            U[j] = make_double4_32a(0., 0., 0., 0.);
            if (j >= deg) continue;
            const int2 id = g.cidx[k0 + j];
            U[j] = g.unit[k0 + j];
            if (U[j].z > 0. && !(id.y & 4)) mask |= 1u << j;         // walls do not bound the bed
            if (id.x < 0) continue;
            const double zn = z[id.x], d = zn - zc;
            const double4_32a ge = g.ent[k0 + j];
            bx += ge.x * d; by += ge.y * d;
            const long long k = ordered(zn);
            lo = min(lo, k); hi = max(hi, k);
        }
        double gx = 0., gy = 0.;
        if (L.w != 0.) {
            const double r = g.lsr[c];
            gx = quotient(L.x * bx + L.y * by, L.w, r);
            gy = quotient(L.y * bx + L.z * by, L.w, r);
            limit64<D>(gx, gy, U, mask, g.par[c], unordered(hi) - zc, zc - unordered(lo));
        }
        g.gbed[c] = make_double2(gx, gy);
    }
}

// First stage's primitives of a state placed in work directly (single residual).
// A nonfinite momentum of a dry cell, which a substep's drag has set to zero,
// fails the stage; the velocity that its neighbours see is zero.
__global__ void __launch_bounds__(256) k64_prim(MeshDev m, StateDev s, Ctrl *ctrl, Cells64 g)
{
    const int nc = m.nc;
    FOR_ACTIVE_CELLS(m.act, c) {
        Ctrl &ct = ctrl[m.cell_sid[c]];
        if (!ct.active || ct.done) continue;
        const double hu = s.work[nc + c], hv = s.work[2 * nc + c];
        if (!finite_bits(hu) || !finite_bits(hv)) raise_status(ct, 1, ST_SPATIAL);
        put_prim64(g.prim[0], c, s.work[c], hu, hv, s.z[c], ct.dry);
    }
}

template <int D>
__global__ void __launch_bounds__(128, 4) k64_cells(MeshDev m, StateDev s, Ctrl *ctrl, Work w, Cells64 g, int stage)
{
    const Prim64 *P = g.prim[stage == 1 ? 0 : 1];
    FOR_ACTIVE_CELLS(m.act, c) {
        Ctrl &ct = ctrl[m.cell_sid[c]];
        if (skip_stage(ct, stage)) continue;
        const int k0 = m.offset[c], deg = m.offset[c + 1] - k0;
        int2 id[D];
#pragma unroll
        for (int j = 0; j < D; ++j) id[j] = j < deg ? g.cidx[k0 + j] : make_int2(-1, 0);
        const Prim64 p = P[c];
        const double dry = ct.dry, zc = s.z[c];
        if (negative(p.h)) raise_status(ct, stage, ST_SPATIAL);
        if (!finite_bits(p.h) || !finite_bits(p.eta) || !finite_bits(p.u) || !finite_bits(p.v))
            raise_status(ct, stage, ST_SPATIAL);
        const bool wet = greater(p.h, dry), outlet = g.ccls[c] & 1;
        bool active = wet;
        const double centre[3] = {p.eta, p.u, p.v};
        double bx[3] = {0., 0., 0.}, by[3] = {0., 0., 0.}, zx = 0., zy = 0.;
        long long lo[3], hi[3], zlo = ordered(zc), zhi = zlo;
#pragma unroll
        for (int k = 0; k < 3; ++k) lo[k] = hi[k] = ordered(centre[k]);
#pragma unroll
        for (int j = 0; j < D; ++j) {
            const int n = id[j].x;
            if (n < 0) { if (id[j].y & 1) active = true; continue; }
            const Prim64 pn = P[n];
            const double4_32a ge = g.ent[k0 + j];
            const bool wetn = greater(pn.h, dry);
            if (wetn) active = true;
            double adj[3] = {pn.eta, pn.u, pn.v};
            // a dry neighbour whose bed rises above the wet surface contributes
            // the surface (the depths here are eta - b, as in k_cells)
            if (!(wet && greater(pn.h, 2. * dry))) {
                const double zn = s.z[n];
                if (p.eta - zc > dry && pn.eta - zn <= dry && zn >= p.eta) adj[0] = p.eta;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double d = adj[k] - centre[k];
                bx[k] += ge.x * d; by[k] += ge.y * d;
                const long long v = ordered(adj[k]);
                lo[k] = min(lo[k], v); hi[k] = max(hi[k], v);
            }
            if (outlet) {
                const double zn = s.z[n], d = zn - zc;
                zx += ge.x * d; zy += ge.y * d;
                const long long v = ordered(zn);
                zlo = min(zlo, v); zhi = max(zhi, v);
            }
        }
        double gx[4] = {0., 0., 0., 0.}, gy[4] = {0., 0., 0., 0.};
        const double4_32a L = g.ls[c];
        if (active && L.w != 0.) {
            const double r = g.lsr[c];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                gx[k] = quotient(L.x * bx[k] + L.y * by[k], L.w, r);
                gy[k] = quotient(L.y * bx[k] + L.z * by[k], L.w, r);
            }
            if (wet)
#pragma unroll
                for (int j = 0; j < D; ++j)
                    if (id[j].y & 4) {                       // a wall mirrors the velocity
                        const int f = m.faces[k0 + j];
                        const double nx = m.normal[f], ny = m.normal[m.nf + f];
                        const double un = p.u * nx + p.v * ny;
                        const long long mx = ordered(p.u - 2. * un * nx), my = ordered(p.v - 2. * un * ny);
                        lo[1] = min(lo[1], mx); hi[1] = max(hi[1], mx);
                        lo[2] = min(lo[2], my); hi[2] = max(hi[2], my);
                    }
            double4_32a U[D];
            unsigned bounded = 0u, kept = 0u;                // entries that bound the surface; that keep a bed slope
            if (outlet) {
                gx[3] = quotient(L.x * zx + L.y * zy, L.w, r);
                gy[3] = quotient(L.y * zx + L.z * zy, L.w, r);
                const double hh = p.eta - zc;
                const double sq = hh > dry ? sqrt(ct.grav * hh) : 0.;
                const double bedtol = 64.0 * EPS * fmax(1.0, fabs(zc));
                for (int j = 0; j < deg; ++j) {
                    // an open stage outlet with a subcritical wet owner keeps its bed slope
                    if (!(g.cidx[k0 + j].y & 2) || !(hh > dry)) continue;
                    const int f = m.faces[k0 + j];
                    const double4_32a ge = g.ent[k0 + j];
                    if (fabs(p.u * m.normal[f] + p.v * m.normal[m.nf + f]) < sq &&
                        fabs(gx[3] * ge.z + gy[3] * ge.w) > bedtol) kept |= 1u << j;
                }
            } else {
                const double2 gb = g.gbed[c];
                gx[3] = gb.x; gy[3] = gb.y;
            }
#pragma unroll
            for (int j = 0; j < D; ++j) {
                U[j] = make_double4_32a(0., 0., 0., 0.);
                if (j >= deg) continue;
                U[j] = g.unit[k0 + j];
                if (U[j].z > 0. && !(kept >> j & 1u)) bounded |= 1u << j;
            }
#pragma unroll
            for (int k = 1; k < 3; ++k) {
                const double up = unordered(hi[k]) - centre[k], down = unordered(lo[k]) - centre[k];
                const long long one = 0x3ff0000000000000LL;
                const long long scale = max(one, max(magnitude(centre[k]), max(magnitude(unordered(lo[k])),
                                                                               magnitude(unordered(hi[k])))));
                const long long tol = __double_as_longlong(64.0 * EPS * __longlong_as_double(scale));
                double th = 1.;
#pragma unroll
                for (int j = 0; j < D; ++j) {
                    if (j >= deg || (kept >> j & 1u)) continue;
                    const double4_32a ge = g.ent[k0 + j];
                    const double d = gx[k] * ge.z + gy[k] * ge.w;
                    if (magnitude(d) <= tol) continue;
                    const double room = __double_as_longlong(d) < 0 ? down : up;
                    // room / d >= 1 leaves the factor as it is; otherwise divide
                    // unless FP32 shows a quotient above the factor already held
                    if (magnitude(room) >= magnitude(d)) continue;
                    if (truncated(room) * __fdividef(1.f, truncated(d)) > truncated(th) * (1.f + 4.e-6f)) continue;
                    const double q = room / d;
                    if (magnitude(q) < __double_as_longlong(th)) th = fabs(q);
                }
                gx[k] *= th; gy[k] *= th;
            }
            const unsigned par = g.par[c];
            limit64<D>(gx[0], gy[0], U, bounded, par, unordered(hi[0]) - p.eta, p.eta - unordered(lo[0]));
            if (outlet) {
                unsigned bed = 0u;                           // walls do not bound the bed
#pragma unroll
                for (int j = 0; j < D; ++j)
                    if ((bounded >> j & 1u) && !(id[j].y & 4)) bed |= 1u << j;
                limit64<D>(gx[3], gy[3], U, bed, par, unordered(zhi) - zc, zc - unordered(zlo));
            }
        }
        bool flatten = !wet;
        if (wet) {
            // the reconstructed depth stays positive at every face: FP32 bounds
            // settle it unless the depth is of the order of the increments
            float rise = 0.f, bed = 0.f;
            const float f0 = fabsf(truncated(gx[0])), f1 = fabsf(truncated(gy[0])), f2 = fabsf(truncated(gx[3])),
                        f3 = fabsf(truncated(gy[3]));
#pragma unroll
            for (int j = 0; j < D; ++j) {
                if (j >= deg) continue;
                const double4_32a ge = g.ent[k0 + j];
                const float rx = fabsf(truncated(ge.z)), ry = fabsf(truncated(ge.w));
                rise = fmaxf(rise, f0 * rx + f1 * ry);
                bed = fmaxf(bed, f2 * rx + f3 * ry);
            }
            const float slack = 1.e-14f * (fabsf(truncated(p.eta)) + fabsf(truncated(zc)));
            if (!((rise + bed) * 1.00001f + slack + 1.00001f * truncated(dry) < truncated(p.h) * .99999f))
                for (int k = k0; k < k0 + deg; ++k) {
                    const double4_32a ge = g.ent[k];
                    const double eta = (p.eta + gx[0] * ge.z) + gy[0] * ge.w;
                    const double zb = (zc + gx[3] * ge.z) + gy[3] * ge.w;
                    if (eta - zb <= dry || fabs(zb - zc) >= p.h) { flatten = true; break; }
                }
        }
        CellRec o;
        o.h = p.h; o.eta = p.eta; o.u = p.u; o.v = p.v; o.b = zc;
#pragma unroll
        for (int k = 0; k < 4; ++k) { o.gx[k] = gx[k]; o.gy[k] = gy[k]; }
        o.flags = (flatten ? 1 : 0) | (active ? 2 : 0);
        o.pad = 0; o.pad2 = 0.;
        w.rec[c] = o;
    }
}

}  // namespace brx
