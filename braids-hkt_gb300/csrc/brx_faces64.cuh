// FP64 face sweep of the f-wave step: traces, hydrostatic reconstruction,
// augmented f-wave, flux assembly.
//
// What bounds it: FP64 instructions (brx_num64.cuh). Nearly every face joins
// two wet states; for those the solve is written out with the terms that
// vanish or repeat taken out, each remaining operation being the reference's
// own with the same operands (a quotient to the bound of quotient()), so the
// fluxes of all compared faces are the same bits:
//   * the hydrostatic reconstruction gives both sides one bed, so the bed
//     jump is zero and with it the steady-state correction of the depth and
//     momentum jumps (their clamps hold zero in place);
//   * the eigenvector matrix has unit and zero entries: Cramer's determinants
//     reduce to one to five products;
//   * the quotients by one depth share its reciprocal (quotient()), as do the
//     three wave strengths, whose divisor is lam0 - lam2;
//   * the middle state's characteristics matter only to a flow near critical;
//     bounds on its three wave patterns leave it out elsewhere, and with it the
//     branch in which a warp ran all three. Where it is formed, its square
//     roots of g h are those of the wave speeds, the first trial depth of a
//     mixed pattern gives the function value already known, and of a double
//     shock's two terms one is zero.
// About 300 FP64 instructions per wet face instead of 970. Per launch, before
// -> after: 302k cells 831 -> 306 us, 50k 158 -> 70 us, 360 cells 53 -> 29 us.
// A face with a dry side, or with a state whose solution is not finite, takes the
// general solver (dry_face64), which keeps the reference's whole sequence: its
// extrema pass over a NaN, so such a face has the reference's status and speed.
#pragma once
#include "brx_num64.cuh"
#include "brx_turbine.cuh"

namespace brx {

struct Side64 { double h, hu, hv, b, raw; };

__device__ __forceinline__ Side64 trace64(const CellRec &r, double rx, double ry, double dry, bool dryface,
                                          unsigned &bad)
{
    double eta = (r.eta + r.gx[0] * rx) + r.gy[0] * ry, u = (r.u + r.gx[1] * rx) + r.gy[1] * ry,
           v = (r.v + r.gx[2] * rx) + r.gy[2] * ry, b = (r.b + r.gx[3] * rx) + r.gy[3] * ry;
    const bool constant = r.flags & 1;
    if (constant) {
        eta = r.eta; u = r.u; v = r.v;
        if (r.eta - r.b <= dry) b = r.b;
    }
    if (!finite_bits(eta) || !finite_bits(u) || !finite_bits(v) || !finite_bits(b)) bad = 1;
    Side64 o = {0., 0., 0., 0., 0.};
    if (dryface) return o;
    double depth = eta - b;
    if (__double_as_longlong(depth) < 0) depth = 0.;
    o.raw = depth;
    if (!greater(r.h, dry) || (constant && !greater(depth, dry))) depth = 0.;
    o.h = depth; o.hu = depth * u; o.hv = depth * v; o.b = b;
    return o;
}

// Left- and right-side fluxes of a face in its own frame, the speeds' maximum.
struct Solve64 {
    double l[3], r[3], speed;
    double ul, ur;             // normal velocities of the two states (wet faces)
};

// The augmented f-wave solution of two wet states with equal beds
// (augmented_fwave.cu:28-334). in: h, hu, hv of both sides.
__device__ __forceinline__ bool wet_face64(double hL, double huL, double hvL, double hR, double huR, double hvR,
                                           double g, double g16r, Solve64 &o)
{
    bool bad = !(finite_bits(hL) && finite_bits(huL) && finite_bits(hvL) && finite_bits(hR) && finite_bits(huR) &&
                 finite_bits(hvR));
    const double hg = .5 * g;
    const double rL = reciprocal(hL), rR = reciprocal(hR);
    const double uL = quotient(huL, hL, rL), vL = quotient(hvL, hL, rL);
    const double uR = quotient(huR, hR, rR), vR = quotient(hvR, hR, rR);
    const double phiL = hg * (hL * hL) + quotient(huL * huL, hL, rL);
    const double phiR = hg * (hR * hR) + quotient(huR * huR, hR, rR);
    const double sqL = sqrt(g * hL), sqR = sqrt(g * hR), sq = sqR + sqL;
    const double mean = hg * (hR + hL);
    const double uhat = quotient(sqL * uL + sqR * uR, sq, reciprocal(sq)), chat = sqrt(mean);
    const double e1 = uhat - chat, e2 = uhat + chat, sL = uL - sqL, sR = uR + sqR;
    double lam0 = greater(sL, e1) ? e1 : sL, lam2 = greater(e2, sR) ? e2 : sR;
    // The speeds are lam0 = min(lam0, s2m) and lam2 = max(lam2, s1m) with the
    // middle state's characteristics s1m = u - c, s2m = u + c (riemann_type,
    // brx_fwave.cuh). Only a flow near critical reaches s2m below lam0 or s1m
    // above lam2; bounds on the three wave patterns rule that out in a dozen
    // instructions, by a margin far above their rounding:
    //   two rarefactions: the middle celerity is root / 4;
    //   two shocks: the middle depth is at least the deeper side's;
    //   a shock and a rarefaction: it lies between the two sides'.
    const bool right = __double_as_longlong(hR) >= __double_as_longlong(hL);       // R is the deeper side
    const double sqmin = right ? sqL : sqR, sqmax = right ? sqR : sqL;
    const double delu = uR - uL;
    const double fmn = delu + 2. * (sqmin - sqmax);
    const double aL = uL + 2. * sqL, aR = uR - 2. * sqR, slack = 1.e-6 * sq;
    const double up = lam0 + slack, down = lam2 - slack;
    bool clear;
    if (greater(fmn, 0.)) {
        const double root = 2. * sq - delu, q = .75 * root;
        clear = __double_as_longlong(root) > 0 && greater(aR + q, up) && greater(down, aL - q);
    } else {
        const double q = 3. * sqmin;
        clear = greater(uR + sqmax, up) && greater(down, uL - sqmax) && (right ? greater(aR + q, up) : greater(down, aL - q));
    }
    if (!clear) {
        const double hmin = right ? hL : hR, hmax = right ? hR : hL;
        double s1m, s2m;
        if (greater(fmn, 0.)) {
            const double root0 = -delu + 2. * (sqL + sqR), root = __double_as_longlong(root0) < 0 ? 0. : root0;
            const double c = sqrt(g * (g16r * (root * root)));
            s1m = aL - 3. * c;
            s2m = aR + 3. * c;
        } else {
            const double fmx = delu + (hmax - hmin) * sqrt(mean / (hmax * hmin));
            if (!greater(fmx, 0.)) {
                const double iL = 1. / hL, iR = 1. / hR, rmax = right ? iR : iL, rmin = right ? iL : iR;
                const double gM = sqrt(hg * (rmax + rmax)), gm = sqrt(hg * (rmax + rmin)), gap = hmax - hmin;
                const double F0 = delu + gap * gm;
                const double q = (g * gap) / (4. * (hmax * hmax) * gm);
                // ((gL - qL) + gR) - qR with the deeper side's q zero
                const double dfdh = right ? (gm - q) + gM : (gM + gm) - q;
                const double h0 = sqrt(hmax), root = h0 - F0 / (2. * h0 * dfdh);
                const double hm = root * root, rm = 1. / hm, c = sqrt(g * hm);
                s1m = uL - (hm - hL) * sqrt(hg * (rm + iL)) - c;
                s2m = uR + (hm - hR) * sqrt(hg * (rm + iR)) + c;
            } else {
                const double slope = (fmx - fmn) / (hmax - hmin);
                const double c = sqrt(g * (hmin - fmn / slope));
                if (!right) { s1m = aL - 3. * c; s2m = aL - c; }
                else { s2m = aR + 3. * c; s1m = aR + c; }
            }
        }
        if (greater(lam0, s2m)) lam0 = s2m;
        if (greater(s1m, lam2)) lam2 = s1m;
    }
    // wave strengths
    const double d0 = hR - hL, d1 = huR - huL, d2 = phiR - phiL;
    const double r20 = lam0 * lam0, r22 = lam2 * lam2;
    const double det = lam0 - lam2, rdet = reciprocal(det);
    const double b0 = quotient(d1 - d0 * lam2, det, rdet);
    const double b1 = quotient(((d1 * r22 - lam2 * d2) - d0 * (lam0 * r22 - lam2 * r20)) + (lam0 * d2 - d1 * r20), det, rdet);
    const double b2 = quotient(d0 * lam0 - d1, det, rdet);
    const double f00 = b0 * lam0, f01 = b0 * r20, f20 = b2 * lam2, f21 = b2 * r22;
    double f02 = f00 * vL, f22 = f20 * vR;
    const double rest = hR * uR * vR - hL * uL * vL - f02 - f22;
    if (!greater(huL + f00, 0.)) f02 = f02 + rest; else f22 = f22 + rest;
    const double lam1 = .5 * (lam0 + lam2);
    // left- and right-going parts; a wave that stands still gives half to each side
    const bool n0 = greater(-1.e-14, lam0), p0 = greater(lam0, 1.e-14), n1 = greater(-1.e-14, lam1),
               p1 = greater(lam1, 1.e-14), n2 = greater(-1.e-14, lam2), p2 = greater(lam2, 1.e-14);
    double am0, am1, am2, ap0, ap1, ap2;
    if (n0 && p2 && (n1 || p1)) {
        am0 = f00; ap0 = f20; am2 = f02; ap2 = f22;
        am1 = f01; ap1 = f21;
        if (n1) am1 = f01 + b1; else ap1 = b1 + f21;
    } else {
        const double w0 = n0 ? 1. : p0 ? 0. : .5, w1 = n1 ? 1. : p1 ? 0. : .5, w2 = n2 ? 1. : p2 ? 0. : .5;
        const double x0 = n0 ? 0. : p0 ? 1. : .5, x1 = n1 ? 0. : p1 ? 1. : .5, x2 = n2 ? 0. : p2 ? 1. : .5;
        am0 = w0 * f00 + w2 * f20; ap0 = x0 * f00 + x2 * f20;
        am1 = (w0 * f01 + w1 * b1) + w2 * f21; ap1 = (x0 * f01 + x1 * b1) + x2 * f21;
        am2 = w0 * f02 + w2 * f22; ap2 = x0 * f02 + x2 * f22;
    }
    bad = bad || !finite_bits(f00) || !finite_bits(f01) || !finite_bits(f02) || !finite_bits(b1) || !finite_bits(f20) ||
          !finite_bits(f21) || !finite_bits(f22) || !finite_bits(lam0) || !finite_bits(lam2) || !finite_bits(lam1) ||
          !finite_bits(am0) || !finite_bits(am1) || !finite_bits(am2) || !finite_bits(ap0) || !finite_bits(ap1) ||
          !finite_bits(ap2);
    o.speed = __longlong_as_double(max(magnitude(lam0), max(magnitude(lam1), magnitude(lam2))));
    o.l[0] = huL + am0; o.l[1] = phiL + am1; o.l[2] = quotient(huL * hvL, hL, rL) + am2;
    o.r[0] = huR - ap0; o.r[1] = phiR - ap1; o.r[2] = quotient(huR * hvR, hR, rR) - ap2;
    o.ul = uL; o.ur = uR;
    return bad;
}

// A face with a dry or nonfinite state: whether it is closed, the general augmented
// solver with its reflecting wall at a dry side, and the closed face's speed.
// loc: h, un, ut, b of both reconstructed states (brx_fwave.cuh's order).
__device__ __noinline__ bool dry_face64(const double *loc, double hc, double zc, double hn, double zn, int kind,
                                        double hL, double bL, double unL, double hR, double bR, double unR, double dc,
                                        double dn, double dry, double g, bool &closed, Solve64 &o)
{
    closed = false;
    if (kind == 1 && !(fmin(hc, hn) > dry)) {
        double shared;
        if (dc + dn > DBL_MIN_)
            shared = (dn * (zc + hc) + dc * (zn + hn)) / (dc + dn) - fmax(zc, zn);
        else
            shared = 0.5 * ((zc + hc) + (zn + hn)) - fmax(zc, zn);
        closed = shared <= dry;
        if (closed) {
            bool opens = false;
            if (hL > dry && hR <= dry && unL / hL > 0.0) {
                const RType<double> t = riemann_type<double>(hL, hL, unL / hL, -unL / hL, dry, g);
                opens = t.hm > hL + dry && t.hm + bL > bR + dry;
            } else if (hR > dry && hL <= dry && -unR / hR > 0.0) {
                const RType<double> t = riemann_type<double>(hR, hR, -unR / hR, unR / hR, dry, g);
                opens = t.hm > hR + dry && t.hm + bR > bL + dry;
            }
            closed = !opens;
        }
    }
    FWaveOut<double> w;
    double in[8];
    for (int j = 0; j < 8; ++j) in[j] = loc[j];
    const bool bad = fwave<double>(in, g, dry, w) != 0;
    o.speed = 0.;
    if (closed) {
        if (hL > dry) o.speed = fmax(o.speed, fabs(loc[1] / hL) + sqrt(g * hL));
        if (hR > dry) o.speed = fmax(o.speed, fabs(loc[5] / hR) + sqrt(g * hR));
        return bad;
    }
    for (int j = 0; j < 3; ++j) { o.l[j] = 0.; o.r[j] = 0.; }
    if (loc[0] > dry) {
        o.l[0] = loc[1]; o.l[1] = loc[1] * loc[1] / loc[0] + 0.5 * g * (loc[0] * loc[0]); o.l[2] = loc[1] * loc[2] / loc[0];
    }
    if (loc[4] > dry) {
        o.r[0] = loc[5]; o.r[1] = loc[5] * loc[5] / loc[4] + 0.5 * g * (loc[4] * loc[4]); o.r[2] = loc[5] * loc[6] / loc[4];
    }
    for (int j = 0; j < 3; ++j) { o.l[j] += w.amdq[j]; o.r[j] -= w.apdq[j]; }
    o.speed = fmax(fabs(w.s[0]), fmax(fabs(w.s[1]), fabs(w.s[2])));
    return bad;
}

// Four resident blocks of 128 threads (at most 128 registers): a single
// 75k-face scenario then fits the 152 SMs in one wave of 16 warps each.
// ROTOR: a solver with rotors, whose face terms (balanced pressure, ambient
// stress) are formed here from the traces in registers; they need the stage's
// wet gradients and actuator sink first.
template <bool ROTOR>
__global__ void __launch_bounds__(128, 4) k64_faces(MeshDev m, StateDev s, BoundaryDev b, Ctrl *ctrl, Work w, int stage,
                                                    TurbDev t)
{
    const int nf = m.nf, nc = m.nc;
    FOR_ACTIVE_FACES(m.act, f) {
        Ctrl &ct = ctrl[m.face_sid[f]];
        if (skip_stage(ct, stage)) continue;
        const double dry = ct.dry, grav = ct.grav, hg = .5 * grav;
        const int c = m.owner[f], n = m.neighbour[f];
        const double nx = m.normal[f], ny = m.normal[nf + f];
        const CellRec rc = w.rec[c];
        const double pc = hg * rc.h * rc.h;
        const int slot = m.bslot[f];
        if (slot >= 0) {
            // open face: the exterior owner's flux, owner/exterior CFL speed
            const double *q = stage == 1 ? s.work : s.q1;
            const double fl0 = b.flux[slot], fl1 = b.flux[(size_t)b.nslot + slot], fl2 = b.flux[2 * (size_t)b.nslot + slot];
            const double hb = b.trace[slot];
            const double hq = q[c];
            const double a = hq > dry ? fabs((q[nc + c] * nx + q[2 * nc + c] * ny) / hq) + sqrt(grav * hq) : 0.;
            const double bb = hb > dry ? fabs((b.trace[(size_t)b.nslot + slot] * nx + b.trace[2 * (size_t)b.nslot + slot] * ny) / hb) +
                                             sqrt(grav * hb) : 0.;
            w.ws[f] = make_double2(fl0, fmax(a, bb));
            w.gf[f] = make_double4_32a(fl1 - pc * nx, fl2 - pc * ny, 0., 0.);
            continue;
        }
        // a wall reads its owner on both sides: interior and wall faces then go
        // one way through the solve (a branch here splits the warp to the end)
        const bool inner = n >= 0;
        const CellRec rn = w.rec[inner ? n : c];
        const bool wetc = greater(rc.h, dry), wetn = greater(rn.h, dry);
        const bool idle = !wetc && !wetn;
        unsigned bad = 0;
        const Side64 L = trace64(rc, m.disp[f], m.disp[2 * nf + f], dry, idle, bad);
        const int other = inner ? nf : 0;
        const Side64 R = trace64(rn, m.disp[other + f], m.disp[2 * nf + other + f], dry, idle, bad);
        double water = 0., speed = 0., l1 = 0., l2 = 0., r1 = 0., r2 = 0.;
        const bool rotor = ROTOR && inner && t.hkt[m.face_sid[f]];
        double pressure = 0.;          // the rotors' balanced pressure along the normal
        if (!idle) {
            // rotation to the face frame; a wall mirrors the state
            const double unL = L.hu * nx + L.hv * ny, utL = L.hu * (-ny) + L.hv * nx;
            const double twice = inner ? 0. : 2.0 * unL;
            const double xR = R.hu - twice * nx, yR = R.hv - twice * ny;
            const double unR = xR * nx + yR * ny, utR = xR * (-ny) + yR * nx;
            const double hL = L.h, bL = L.b, hR = R.h, bR = R.b;
            const double top = greater(bL, bR) ? bL : bR, eL = hL + bL, eR = hR + bR;
            const long long big = max(__double_as_longlong(dry), max(magnitude(top), max(magnitude(eL), magnitude(eR))));
            const double thin = dry + 16. * EPS * __longlong_as_double(big);
            double hl = eL - top, hr = eR - top;
            if (!greater(hl, thin)) hl = 0.;
            if (!greater(hr, thin)) hr = 0.;
            const double kl = greater(hL, dry) ? quotient(hl, hL, reciprocal(hL)) : 0.;
            const double kr = greater(hR, dry) ? quotient(hr, hR, reciprocal(hR)) : 0.;
            const double loc[8] = {inner ? hl : hL, inner ? unL * kl : unL, inner ? utL * kl : utL, inner ? top : bL,
                                   inner ? hr : hR, inner ? unR * kr : unR, inner ? utR * kr : utR, inner ? top : bR};
            Solve64 o{};
            bool closed = false;
            const bool wet = greater(loc[0], dry) && greater(loc[4], dry);
            bool general = !wet;
            if (wet) general = wet_face64(loc[0], loc[1], loc[2], loc[4], loc[5], loc[6], grav, ct.g16r, o);
            if (general) {
                double in[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) in[j] = loc[j];
                Solve64 d;
                bool shut;
                if (dry_face64(in, rc.h, rc.b, rn.h, rn.b, inner ? 1 : 2, hL, bL, unL, hR, bR, unR,
                               m.distance[f], m.distance[nf + f], dry, grav, shut, d)) bad = 1;
                d.ul = o.ul; d.ur = o.ur;
                o = d;
                closed = shut;
            }
            if constexpr (ROTOR)
                if (rotor && wet && wetc && wetn)
                    pressure = balanced_pressure(m, t, f, c, n, rc, rn,
                                                 FaceTrace{loc[0], loc[4], loc[3], o.ul, o.ur, loc[1], loc[2], loc[5], loc[6]},
                                                 grav, dry, nx, ny);
            speed = o.speed;
            if (closed) {
                const double p = hg * (hL * hL), q = hg * (hR * hR);
                l1 = p * nx; l2 = p * ny; r1 = q * nx; r2 = q * ny;
            } else {
                // left / right mass fluxes agree to the solve's precision
                const long long top = max(0x3ff0000000000000LL, max(magnitude(o.l[0]), magnitude(o.r[0])));
                if (magnitude(o.l[0] - o.r[0]) > __double_as_longlong(1.e-10 * __longlong_as_double(top))) bad = 1;
                if (!inner) {
                    const double pressure = wall_pressure<double>(hL, loc[1], grav, dry);
                    l1 = pressure * nx; l2 = pressure * ny;
                } else {
                    water = 0.5 * (o.l[0] + o.r[0]);
                    l1 = o.l[1] * nx + o.l[2] * (-ny); l2 = o.l[1] * ny + o.l[2] * nx;
                    r1 = o.r[1] * nx + o.r[2] * (-ny); r2 = o.r[1] * ny + o.r[2] * nx;
                    const double cl = hg * (hL * hL - loc[0] * loc[0]), cr = hg * (hR * hR - loc[4] * loc[4]);
                    l1 += cl * nx; l2 += cl * ny; r1 += cr * nx; r2 += cr * ny;
                }
            }
            if (wetc) {
                const double corr = (rc.flags & 1) ? hg * (rc.h * rc.h - hL * hL) : hg * (rc.h + L.raw) * (bL - rc.b);
                l1 += corr * nx; l2 += corr * ny;
            }
            if (inner) {
                if (wetn) {
                    const double corr = (rn.flags & 1) ? hg * (rn.h * rn.h - hR * hR) : hg * (rn.h + R.raw) * (bR - rn.b);
                    r1 += corr * nx; r2 += corr * ny;
                }
            } else { r1 = l1; r2 = l2; }
            if (!finite_bits(water) || !finite_bits(l1) || !finite_bits(l2) || !finite_bits(r1) || !finite_bits(r2)) bad = 1;
        }
        if constexpr (ROTOR)
            if (rotor) {
                t.pface[f] = pressure * nx; t.pface[nf + f] = pressure * ny;
                if (t.stress[m.face_sid[f]]) {
                    double ox = 0., oy = 0.;
                    if (wetc && wetn) rotor_stress(m, t, stage == 1 ? s.work : s.q1, s.z, f, c, n, nx, ny, ox, oy);
                    t.sface[f] = ox; t.sface[nf + f] = oy;
                }
            }
        if (bad) raise_status(ct, stage, ST_SPATIAL);
        w.ws[f] = make_double2(water, speed);
        if (inner) {
            const double pn = hg * rn.h * rn.h;
            w.gf[f] = make_double4_32a(l1 - pc * nx, l2 - pc * ny, r1 - pn * nx, r2 - pn * ny);
        } else w.gf[f] = make_double4_32a(l1 - pc * nx, l2 - pc * ny, r1, r2);
    }
}

}  // namespace brx
