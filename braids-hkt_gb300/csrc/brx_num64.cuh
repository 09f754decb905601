// FP64 helpers that keep work off the FP64 pipe: on GB300 a sub-partition
// issues one FP64 warp instruction every 64-76 clocks, integer and FP32
// instructions some thirty times as often. Measured per dependent operation
// of one warp (clocks): FMA 65, division 640, square root 610, fmax 150,
// comparison 110, round trip through float 127.
#pragma once
#include "brx_common.cuh"

namespace brx {

// Order-preserving integer image of a double (its own inverse): signed 64-bit
// order of the images is the order of the values (-0 before +0, NaN outside).
__device__ __forceinline__ long long ordered(double x)
{
    const long long b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double unordered(long long k)
{
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}
// |x| as an integer that orders like |x|
__device__ __forceinline__ long long magnitude(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffLL; }
__device__ __forceinline__ bool greater(double a, double b) { return ordered(a) > ordered(b); }
// x < 0, false for -0 (which greater() orders below 0) and for a NaN
__device__ __forceinline__ bool negative(double x)
{
    const unsigned long long b = __double_as_longlong(x);
    return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull;
}
__device__ __forceinline__ bool finite_bits(double x)
{
    return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

// x / y from r, 1 / y to an ulp (stored and correctly rounded, or reciprocal()): a
// first quotient and one remainder (P. Markstein, IBM J. Res. Dev. 34(1):111,
// 1990). The result is the rounding of x / y (1 + d) with |d| < 2^-102, so RN(x / y)
// unless x / y lies that close to the middle of two numbers. Three FP64
// instructions instead of ten. Finite x, y and r, x r and the remainder without
// overflow or underflow; an infinite operand, or a y whose reciprocal overflows or
// vanishes, gives no number (any_quotient() where such states are accepted).
__device__ __forceinline__ double quotient(double x, double y, double r)
{
    const double q = __dmul_rn(x, r);
    return __fma_rn(__fma_rn(-y, q, x), r, q);
}

// 1 / y to about an ulp, for quotient(): the hardware's approximation (PTX
// rcp.approx.ftz.f64, relative error below 2^-20) and two Newton-Raphson steps;
// four FP64 instructions instead of a division's ten. 2^-1022 <= |y| <= 2^1022.
__device__ __forceinline__ double reciprocal(double y)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(y));
    r = __fma_rn(__fma_rn(-y, r, 1.), r, r);
    return __fma_rn(__fma_rn(-y, r, 1.), r, r);
}

// x / y as quotient() gives it, or by a division where that is not finite: an
// infinite operand, a divisor outside reciprocal()'s range, an overflow.
static __device__ __noinline__ double plain_quotient(double x, double y) { return x / y; }
__device__ __forceinline__ double any_quotient(double x, double y, double r)
{
    const double q = quotient(x, y, r);
    return finite_bits(q) ? q : plain_quotient(x, y);
}

// FP32 image of a double by truncation, on the integer pipe (a conversion
// instruction runs on the FP64 pipe): relative error below 2^-23, values
// below the FP32 normal range become 0, those above it the largest float.
__device__ __forceinline__ float truncated(double x)
{
    const unsigned hi = __double2hiint(x), lo = __double2loint(x), a = hi & 0x7fffffffu;
    unsigned f = __funnelshift_l(lo, a - 0x38000000u, 3);
    if (a < 0x38100000u) f = 0u;
    if (a >= 0x47f00000u) f = 0x7f7fffffu;
    return __uint_as_float(f | (hi & 0x80000000u));
}

// Primitives of one stage input, one sector per cell.
struct __align__(32) Prim64 {
    double eta, u, v, h;
};

__device__ __forceinline__ void put_prim64(Prim64 *P, int c, double h, double hu, double hv, double z, double dry)
{
    Prim64 p;
    p.eta = h + z; p.h = h;
    if (greater(h, dry)) {
        const double r = reciprocal(h);
        p.u = quotient(hu, h, r); p.v = quotient(hv, h, r);
    } else p.u = p.v = 0.;
    P[c] = p;
}

// Momentum terms of a rotor array, in the reference's add_momentum order
// (river_turbine_flow.py:230-239): ambient stress, actuator sink, balanced
// pressure; face terms gathered as sum(s len flux) / area
// (flow2dh_fixed_bed_kernels.h:54-60 with unit depth weights). The HLLC
// owner's rotor hook has no balanced pressure (river_turbines.py:27-36):
// balanced = false. rarea = RN(1 / area).
__device__ __forceinline__ void add_rotor_momentum(const MeshDev &m, const TurbDev &t, int sid, int c, double area,
                                                   double &r1, double &r2, bool balanced, double rarea)
{
    const int nc = m.nc, nf = m.nf;
    if (t.stress[sid]) {
        double x = 0., y = 0.;
        for (int k = m.offset[c]; k < m.offset[c + 1]; ++k) {
            const int f = m.faces[k];
            x += m.signs[k] * m.length[f] * t.sface[f];
            y += m.signs[k] * m.length[f] * t.sface[nf + f];
        }
        r1 += quotient(x, area, rarea); r2 += quotient(y, area, rarea);
    }
    r1 += t.raw[c]; r2 += t.raw[nc + c];
    if (!balanced) return;
    double x = 0., y = 0.;
    for (int k = m.offset[c]; k < m.offset[c + 1]; ++k) {
        const int f = m.faces[k];
        x += m.signs[k] * m.length[f] * t.pface[f];
        y += m.signs[k] * m.length[f] * t.pface[nf + f];
    }
    r1 += quotient(x, area, rarea); r2 += quotient(y, area, rarea);
}

}  // namespace brx
