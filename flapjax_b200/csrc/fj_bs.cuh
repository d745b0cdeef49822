// fj_bs.cuh -- the reference's Biot-Savart segment kernels in FP64, split into a
// per-(target, vertex) part and a per-(target, filament) part so that chains of
// filaments can share vertex work.  The formulas of each filament are those of
// aero/utils.py:580-648 without their common factor 1 / (4 pi), which the callers apply
// once per sum (kInv4Pi).
//
// The sums are bound by the FP64 pipe (64 lanes per SM; the other pipes and the issue
// slots have room), so the pair is written for the fewest FP64 operations: 11 per vertex
// and 25 (cutoff) or 26 (epsilon) per filament.
//   * One reciprocal square root per vertex and one reciprocal per filament.  Both start
//     from PTX's approximate forms (rsqrt/rcp.approx.ftz.f64, about 20 bits) and take one
//     step of third order by Householder's method (1970), which cubes the seed's error to
//     below the rounding of FP64: within 1.6 and 1.3 halves of a unit in the last place of
//     1 / sqrt and 1 / x (tests/test_gpu_pair_functions.py, beside CUDA's own).
//   * dot = r0.(u1 - u2) as inv1 (r0.r1) - inv2 (r0.r2): no unit vectors.
//   * The cutoff kernel's radius test |c|^2 > rc^2 |r0|^2 runs on the integer pipe, on the
//     leading bits of the two sides; pairs within about 1 % of the core radius take the
//     reference's own radial distance (with its division), so that no pair changes side.
// 25 800 targets x 55 600 filaments: cutoff 7.86 -> 3.9 ms (3.7e11 pairs/s), epsilon 5.92 ->
// 3.5 ms (4.1e11 pairs/s, 0.8 of the FP64 pipe at 37 operations a pair) against the form with
// unit vectors, one division per filament and a second one for the radial distance.
#pragma once

#include "fj_common.cuh"

namespace fj {

constexpr double kInv4Pi = 1.0 / kFourPi;

// 1 / sqrt(x) for normal x > 0: with h = x y, e = 1 - h y Householder's step for 1 / y^2 - x is
// y (1 + e / 2 + 3 e^2 / 8), the binomial series of (1 - e)^(-1/2) to its third term.
__device__ __forceinline__ double rsqrt_normal(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1 / x for normal x below 2^1022: with e = 1 - x y Householder's step for 1 / y - x is y (1 + e + e^2), the
// geometric series to its third term.
__device__ __forceinline__ double rcp_normal(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// x, or a number near 2^1021 for an infinite x (on the integer pipe): a pair so far away that its
// |c|^2 overflows adds next to nothing, where 0 (1 / x of infinity) times infinity would be NaN.
__device__ __forceinline__ double capped(double x) {
    return __hiloint2double(min(__double2hiint(x), 0x7fcfffff), __double2loint(x));
}

template <int KER>
struct Vtx64 {
    double d[3];  // x - y
    double inv;   // 1 / ||x - y||_eps  (plain kernel: 1 / ||x - y||)
};

template <int KER>
__device__ __forceinline__ void vtx64(const double x[3], double yx, double yy, double yz,
                                      Vtx64<KER>& o) {
    o.d[0] = x[0] - yx;
    o.d[1] = x[1] - yy;
    o.d[2] = x[2] - yz;
    // r / jnp.linalg.norm(r) (plain, aero/utils.py:591); r / ||r||_eps (make_unit_epsilon,
    // :603, and the epsilon kernel's rsqrt, :617-618), whose argument is at least eps^2
    if (KER == FJ_KERNEL_PLAIN) {
        o.inv = rsqrt(o.d[0] * o.d[0] + o.d[1] * o.d[1] + o.d[2] * o.d[2]);
    } else {
        o.inv = rsqrt_normal(fma(o.d[2], o.d[2], fma(o.d[1], o.d[1], fma(o.d[0], o.d[0], kEps * kEps))));
    }
}

// The reference's radial distance test of the cutoff kernel (aero/utils.py:637-648).
__device__ __forceinline__ bool outside_core(const double d[3], double r0x, double r0y, double r0z, double rc2) {
    const double sm = (r0x * d[0] + r0y * d[1] + r0z * d[2]) / (r0x * r0x + r0y * r0y + r0z * r0z);
    const double mx = d[0] - sm * r0x, my = d[1] - sm * r0y, mz = d[2] - sm * r0z;
    return mx * mx + my * my + mz * mz > rc2;
}

// |c|^2 > rq = rc2 |r0|^2 with the reference's decision.  The leading words (sign, exponent
// and 8 mantissa bits) decide where they are not within one of each other; c2's rounding is
// far below that wherever the pair's velocity matters.  Within one, with no core radius or no
// length, or where c2 is not finite (a NaN of either sign), `close` is set: the reference's test
// decides, which keeps no NaN.
__device__ __forceinline__ bool outside_core(double c2, double rq, bool& close) {
    const int hc = __double2hiint(c2) >> 12, hq = __double2hiint(rq) >> 12;
    close = close || hq == 0 || (unsigned)hc >= 0x7ff00u || (unsigned)(hc - hq + 1) <= 2u;
    return hc > hq;
}

// acc[j] += 4 pi g K(x_j; y0 -> y1) for T targets.  q: EPSILON |r0|^4 (epsilon kernel),
// rc2 |r0|^2 (cutoff) or unused (plain).
template <int KER, int T>
__device__ __forceinline__ void link64(const Vtx64<KER> (&a)[T], const Vtx64<KER> (&b)[T], double g, double r0x,
                                       double r0y, double r0z, double q, double rc2, double (&acc)[T][3]) {
    double c[T][3], val[T];
    bool keep[T], close = false;
#pragma unroll
    for (int j = 0; j < T; ++j) {
        // r1 = a.d (x - y0), r2 = b.d (x - y1), r0 = y1 - y0
        const double *r1 = a[j].d, *r2 = b[j].d;
        c[j][0] = r1[1] * r2[2] - r1[2] * r2[1];
        c[j][1] = r1[2] * r2[0] - r1[0] * r2[2];
        c[j][2] = r1[0] * r2[1] - r1[1] * r2[0];
        const double c2 = c[j][0] * c[j][0] + c[j][1] * c[j][1] + c[j][2] * c[j][2];
        if (KER == FJ_KERNEL_PLAIN) {  // aero/utils.py:587-592
            const double dot = r0x * (r1[0] * a[j].inv - r2[0] * b[j].inv) + r0y * (r1[1] * a[j].inv - r2[1] * b[j].inv) +
                               r0z * (r1[2] * a[j].inv - r2[2] * b[j].inv);
            val[j] = g * (dot / c2);
        } else {
            const double s1 = r0x * r1[0] + r0y * r1[1] + r0z * r1[2];
            const double s2 = r0x * r2[0] + r0y * r2[1] + r0z * r2[2];
            const double dot = fma(a[j].inv, s1, -(b[j].inv * s2));
            // aero/utils.py:619-623 (epsilon), :637-648 (cutoff)
            val[j] = (g * dot) * rcp_normal(capped(KER == FJ_KERNEL_EPSILON ? c2 + q : c2));
            if (KER == FJ_KERNEL_CUTOFF) keep[j] = outside_core(c2, q, close);
        }
    }
    if (KER == FJ_KERNEL_CUTOFF) {
        if (close) {
#pragma unroll
            for (int j = 0; j < T; ++j) {
                keep[j] = outside_core(a[j].d, r0x, r0y, r0z, rc2);
                if (!keep[j]) c[j][0] = c[j][1] = c[j][2] = 0.0;  // (they may be NaN)
            }
        }
#pragma unroll
        for (int j = 0; j < T; ++j) val[j] = keep[j] ? val[j] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < T; ++j) {
        acc[j][0] = fma(c[j][0], val[j], acc[j][0]);
        acc[j][1] = fma(c[j][1], val[j], acc[j][1]);
        acc[j][2] = fma(c[j][2], val[j], acc[j][2]);
    }
}

// A link's q from its vector (see link64).
template <int KER>
__device__ __forceinline__ double link_q(double r0sq, double rc2) {
    return KER == FJ_KERNEL_EPSILON ? kEps * r0sq * r0sq : KER == FJ_KERNEL_CUTOFF ? rc2 * r0sq : r0sq;
}

// 4 pi K(x; y0 -> y1) of one unit-strength filament.
template <int KER>
__device__ __forceinline__ void segment64(const double x[3], const double y0[3], const double y1[3], double rc2,
                                          double (&k)[3]) {
    Vtx64<KER> a[1], b[1];
    vtx64<KER>(x, y0[0], y0[1], y0[2], a[0]);
    vtx64<KER>(x, y1[0], y1[1], y1[2], b[0]);
    const double r0x = y1[0] - y0[0], r0y = y1[1] - y0[1], r0z = y1[2] - y0[2];
    double acc[1][3] = {{0.0, 0.0, 0.0}};
    link64<KER, 1>(a, b, 1.0, r0x, r0y, r0z, link_q<KER>(r0x * r0x + r0y * r0y + r0z * r0z, rc2), rc2, acc);
    k[0] = acc[0][0];
    k[1] = acc[0][1];
    k[2] = acc[0][2];
}

}  // namespace fj
