// fj_bsgrad.cuh -- derivatives of one Biot-Savart filament (FP64), shared by the
// adjoint sums (fj_adjoint.cu) and the dense influence Jacobians (fj_jac.cu).
//
// With r1 = x - y0, r2 = x - y1, r0 = y1 - y0 = r1 - r2, c = r1 x r2, n_i = sqrt(|r_i|^2 + eps^2),
// dot = r0.(r1 / n1 - r2 / n2), D = |c|^2 + eps|r0|^4 (epsilon kernel, aero/utils.py:606-623) or
// |c|^2 (cutoff kernel, :626-648, whose pairs within the cutoff radius of the filament line
// contribute nothing, derivative included), s = dot / D, b = (lam.c) / D and w = lam - 2 b c, the
// derivatives of 4 pi lam.K = s (lam.c) are
//   d/dr1 = s (r2 x w) + b [r1/n1 - r2/n2 + r0/n1 - (r0.r1/n1^3) r1] - 4 eps b s |r0|^2 r0
//   d/dr2 = s (w x r1) - b [r1/n1 - r2/n2 + r0/n2 - (r0.r2/n2^3) r2] + 4 eps b s |r0|^2 r0
// (w carries both the cross products' and |c|^2's), and for the target
//   d/dr1 + d/dr2 = s (w x r0) + b [(1/n1 - 1/n2) r0 - (r0.r1/n1^3) r1 + (r0.r2/n2^3) r2].
// x_bar = d/dr1 + d/dr2, y0_bar = -d/dr1, y1_bar = -d/dr2.
//
// As the sums themselves these are bound by the FP64 pipe and written for few operations: per
// pair 80 for the target and 114 for the filament's two ends and strength (which has both
// vertices to itself), one reciprocal square root a vertex and one reciprocal a filament
// (fj_bs.cuh), the cutoff's radius test on the integer pipe.
//
// dot: a target on the filament's line but beyond its ends has r1 / n1 = r2 / n2, and its
// derivative, unlike its velocity, keeps dot's rounding whole, over a D of eps|r0|^4 alone.  With
// P = r1.r2 + eps^2, dot = (1/n1 + 1/n2) (n1 n2 - P), and where P > 0 (no end between)
// n1 n2 - P = (|c|^2 + eps^2 |r0|^2) / (n1 n2 + P), in which nothing cancels.
#pragma once

#include "fj_bs.cuh"

namespace fj {

// Whether a coordinate is finite and 2^160 or more: where none is, a pair's products stay in range.
__device__ __forceinline__ bool beyond(double x, double y, double z) {
    constexpr unsigned kHi = (1023u + 160u) << 20;
    auto far = [](double v) { return ((unsigned)__double2hiint(v) & 0x7fffffffu) - kHi < 0x7ff00000u - kHi; };
    return far(x) || far(y) || far(z);
}

template <int KER>
struct VtxGrad {
    double d[3], inv, inv2, n;  // x - y; 1 / n, 1 / n^2, n
};

template <int KER>
__device__ __forceinline__ void vtx_grad(const double x[3], double yx, double yy, double yz, VtxGrad<KER>& o) {
    o.d[0] = x[0] - yx;
    o.d[1] = x[1] - yy;
    o.d[2] = x[2] - yz;
    const double n2 = fma(o.d[2], o.d[2], fma(o.d[1], o.d[1], fma(o.d[0], o.d[0], kEps * kEps)));
    o.inv = rsqrt_normal(n2);
    o.inv2 = o.inv * o.inv;
    o.n = n2 * o.inv;
}

// (Written out: the two passes' products are to round alike, see LinkGrad.)
__device__ __forceinline__ void cross_grad(const double a[3], const double b[3], double (&o)[3]) {
    o[0] = fma(a[1], b[2], -(a[2] * b[1]));
    o[1] = fma(a[2], b[0], -(a[0] * b[2]));
    o[2] = fma(a[0], b[1], -(a[1] * b[0]));
}

__device__ __forceinline__ double dot_grad(const double a[3], const double b[3], double c) {
    return fma(a[2], b[2], fma(a[1], b[1], fma(a[0], b[0], c)));
}

// A filament: vector, strength / (4 pi), the kernel's q (see link64), eps^2 |r0|^2.
struct FilGrad {
    double r0[3], g, q, e2;
};

// What both derivatives take from a pair: g s, g b, w; s1, s2 = r0.r_i / n_i^2; k = s (lam.c).
struct PairGrad {
    double gs, gb, s1, s2, w[3], s, k;
};

// False for a pair within the core radius, which adds nothing: the callers leave it out, since its
// other factors may be NaN.  kFar: den D, of the sixth power of a distance, may leave FP64's range
// before D and K do (from 1e51, where they do from 1e77): divisions one by one.
template <int KER, bool kFar>
__device__ __forceinline__ bool pair_grad(const VtxGrad<KER>& A, const VtxGrad<KER>& B, const FilGrad& f, double rc2,
                                          const double lam[3], PairGrad& o) {
    static_assert(KER != FJ_KERNEL_PLAIN, "the plain kernel has no adjoint");
    double c[3];
    cross_grad(A.d, B.d, c);
    const double c2 = dot_grad(c, c, 0.0);
    const double P = dot_grad(A.d, B.d, kEps * kEps), Z = fma(A.n, B.n, fabs(P));
    const bool ahead = __double2hiint(P) > 0;
    const double D = KER == FJ_KERNEL_EPSILON ? c2 + f.q : c2;
    const double num = ahead ? c2 + f.e2 : Z, den = ahead ? Z : 1.0;
    const double a = dot_grad(lam, c, 0.0);
    double b;
    if (kFar) {
        const double inv = 1.0 / D;
        b = a * inv;
        o.s = D == INFINITY ? 0.0 : (A.inv + B.inv) * (num / den * inv);
    } else {
        const double inv = rcp_normal(den * D);
        b = a * (den * inv);
        o.s = (A.inv + B.inv) * num * inv;
    }
    o.s1 = A.inv2 * dot_grad(f.r0, A.d, 0.0);
    o.s2 = B.inv2 * dot_grad(f.r0, B.d, 0.0);
    if (KER == FJ_KERNEL_CUTOFF) {
        bool close = false, keep = outside_core(c2, f.q, close);
        if (close) keep = outside_core(A.d, f.r0[0], f.r0[1], f.r0[2], rc2);
        if (!keep) return false;
    }
    o.k = o.s * a;
    o.gs = f.g * o.s;
    o.gb = f.g * b;
    const double b2 = -2.0 * b;
#pragma unroll
    for (int k = 0; k < 3; ++k) o.w[k] = fma(b2, c[k], lam[k]);
    return true;
}

// acc += g d(lam.K)/dx, the pair's terms added up before (acc may be of the size of 1 / (eps
// |r0|^3), see LinkGrad, and a rounding of that size a pair is enough).
template <int KER, bool kFar>
__device__ __forceinline__ void target_grad(const VtxGrad<KER>& A, const VtxGrad<KER>& B, const FilGrad& f, double rc2,
                                            const double lam[3], double (&acc)[3]) {
    PairGrad p;
    if (!pair_grad<KER, kFar>(A, B, f, rc2, lam, p)) return;
    const double f1 = p.gb * A.inv, f2 = p.gb * B.inv, h0 = f1 - f2, h1 = f1 * p.s1, h2 = f2 * p.s2;
    double t[3];
    cross_grad(p.w, f.r0, t);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        acc[i] += fma(p.gs, t[i], fma(h0, f.r0[i], fma(-h1, A.d[i], h2 * B.d[i])));
}

// The sums over targets of one filament's derivatives, but for its vector in the terms along
// it: g d(lam.K)/dr1 = d1 + e1 r0, likewise d2, e2; k: 4 pi lam.K.  g goes into s and b first, as
// for the target: a filament of a surface and the target at its middle, which moves with it,
// have derivatives of 1 / (eps |r0|^3) that cancel, and so do their roundings where both are
// made of the same products.
struct LinkGrad {
    double d1[3], d2[3], e1, e2, k;
};

// e4 = 4 eps |r0|^2 (epsilon kernel).
template <int KER, bool kFar>
__device__ __forceinline__ void link_grad(const VtxGrad<KER>& A, const VtxGrad<KER>& B, const FilGrad& f, double rc2,
                                          double e4, const double lam[3], LinkGrad& o) {
    PairGrad p;
    if (!pair_grad<KER, kFar>(A, B, f, rc2, lam, p)) return;
    const double f1 = p.gb * A.inv, f2 = p.gb * B.inv;
    const double se = KER == FJ_KERNEL_EPSILON ? p.s * e4 : 0.0;
    const double h1 = fma(-f1, p.s1, f1), h2 = fma(f2, p.s2, f2);
    double t[3];
    cross_grad(B.d, p.w, t);
#pragma unroll
    for (int i = 0; i < 3; ++i) o.d1[i] += fma(p.gs, t[i], fma(h1, A.d[i], -f2 * B.d[i]));
    o.e1 = KER == FJ_KERNEL_EPSILON ? fma(p.gb, A.inv - se, o.e1) : o.e1 + f1;
    cross_grad(p.w, A.d, t);
#pragma unroll
    for (int i = 0; i < 3; ++i) o.d2[i] += fma(p.gs, t[i], fma(-f1, A.d[i], h2 * B.d[i]));
    o.e2 = KER == FJ_KERNEL_EPSILON ? fma(p.gb, se - B.inv, o.e2) : o.e2 - f2;
    o.k += p.k;
}

// The same derivatives for the linearisation, by the unit vectors and per end in full.  It adds
// the targets' to the vertices' (fj_vertex_jacobian) where a target moves with a filament, and
// the entries of 1 / (eps |r0|^3) that cancel there leave 1e-9 of themselves: one arithmetic for
// both, whose cost (180 operations a pair) its host work hides.
struct VtxA {
    double d[3];  // x - y
    double u[3];  // d / n
    double rn;    // 1 / n, n = sqrt(|d|^2 + eps^2)
};

__device__ __forceinline__ void vtxa(const double x[3], double yx, double yy, double yz, VtxA& o) {
    o.d[0] = x[0] - yx;
    o.d[1] = x[1] - yy;
    o.d[2] = x[2] - yz;
    o.rn = rsqrt(o.d[0] * o.d[0] + o.d[1] * o.d[1] + o.d[2] * o.d[2] + kEps * kEps);
    o.u[0] = o.d[0] * o.rn;
    o.u[1] = o.d[1] * o.rn;
    o.u[2] = o.d[2] * o.rn;
}

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double o[3]) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// d(lam . K)/dr1 -> g1, d(lam . K)/dr2 -> g2 (each scaled by g), and lam . K (unit g).
// KER: FJ_KERNEL_EPSILON (D = |c|^2 + eps |r0|^4) or FJ_KERNEL_CUTOFF (D = |c|^2, zero
// within rc2 of the filament line, aero/utils.py:637-648).
template <int KER>
__device__ __forceinline__ void link_vjp(const VtxA& A, const VtxA& B, const double r0[3], double g,
                                         const double lam[3], double rc2, double g1[3], double g2[3], double& lk) {
    double c[3];
    cross3(A.d, B.d, c);
    const double du[3] = {A.u[0] - B.u[0], A.u[1] - B.u[1], A.u[2] - B.u[2]};
    const double dot = dot3(r0, du);
    const double r0sq = dot3(r0, r0);
    if (KER == FJ_KERNEL_CUTOFF) {
        const double sm = dot3(r0, A.d) / r0sq;
        const double mx = A.d[0] - sm * r0[0], my = A.d[1] - sm * r0[1], mz = A.d[2] - sm * r0[2];
        if (!(mx * mx + my * my + mz * mz > rc2)) {
            g1[0] = g1[1] = g1[2] = g2[0] = g2[1] = g2[2] = 0.0;
            lk = 0.0;
            return;
        }
    }
    const double eps_term = KER == FJ_KERNEL_EPSILON ? kEps * r0sq * r0sq : 0.0;
    const double D = dot3(c, c) + eps_term;
    const double inv = 1.0 / (kFourPi * D);
    const double s = dot * inv;
    const double a = dot3(lam, c);
    lk = s * a;
    const double r0u1 = dot3(r0, A.u), r0u2 = dot3(r0, B.u);
    double t1[3], t2[3], dD1[3], dD2[3];
    cross3(B.d, lam, t1);  // r2 x lam
    cross3(lam, A.d, t2);  // lam x r1
    double r2c[3], cr1[3];
    cross3(B.d, c, r2c);
    cross3(c, A.d, cr1);
    const double e4 = KER == FJ_KERNEL_EPSILON ? 4.0 * kEps * r0sq : 0.0;
    for (int k = 0; k < 3; ++k) {
        dD1[k] = 2.0 * r2c[k] + e4 * r0[k];
        dD2[k] = 2.0 * cr1[k] - e4 * r0[k];
    }
    const double q = kFourPi * s;  // dot / D
    for (int k = 0; k < 3; ++k) {
        const double dd1 = du[k] + (r0[k] - r0u1 * A.u[k]) * A.rn;
        const double dd2 = -du[k] - (r0[k] - r0u2 * B.u[k]) * B.rn;
        g1[k] = g * (s * t1[k] + a * (dd1 - q * dD1[k]) * inv);
        g2[k] = g * (s * t2[k] + a * (dd2 - q * dD2[k]) * inv);
    }
}

}  // namespace fj
