// fj_adjoint.cu -- hand-written adjoints of the induced-velocity sum and of the solve.
//
// The reference differentiates its UVLM by reverse-mode AD (jax.vjp through
// solve_prescribed_dynamic / the residuals of aero/uvlm.py:1529-1940).  Here the two
// operators that carry the cost have hand-written adjoints:
//   * the Biot-Savart sum v(x) = sum_s K(x; y0_s, y1_s) g_s (compute_v_ind,
//     aero/aic.py:248-310) -- cotangent lam(x) -> x_bar, vertex adjoints of every source
//     lattice, ring-circulation adjoints (FP64; epsilon kernel aero/utils.py:606-623, and
//     the cutoff kernel :626-648, whose D is |c|^2 and whose pairs within the cutoff
//     radius of the filament line contribute nothing, derivative included);
//   * the dense solve (aero/uvlm.py:985) -- A^T mu = lam with the getrf factors of A.
// K's derivative is in fj_bsgrad.cuh; g_bar = lam.K.
// 2531 targets x 14 118 filaments (cutoff): targets 419 -> 229 us, filaments 467 -> 287 us, of
// which the FP64 pipe's own 158 and 226 us; 768 x 9 800 (epsilon): 103 -> 63, 106 -> 86 us,
// against the form with unit vectors and divisions that link_vjp keeps.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "fj_bsgrad.cuh"
#include "fj_trsv.cuh"
#include "fj_vind.cuh"

namespace fj {

constexpr int kAdjBlock = 128;
constexpr int kAdjCtas = 4;  // per SM: 8 make two waves; 3 to 6 measured within 5 %, two pairs at a time 10 % faster

// Pass 1: target adjoints.  Walks the stream as the forward sum does.  kAlone: of a call for
// these only, with the linearisation's arithmetic (link_vjp).
template <int KER, bool kAlone>
__global__ void __launch_bounds__(kAdjBlock, kAdjCtas)
    vjp_targets_kernel(const double* __restrict__ tgt, const double* __restrict__ lam, int64_t n_t,
                       const Elem64* __restrict__ st, int64_t n_elem, int n_split, double rc2,
                       double* __restrict__ part) {
    __shared__ Elem64 sh[kAdjBlock];
    __shared__ double se2[kAdjBlock];
    const int split = blockIdx.y;
    const int64_t per = (n_elem + n_split - 1) / n_split;
    const int64_t e0 = (int64_t)split * per;
    const int64_t e1 = min(n_elem, e0 + per);
    const int64_t vend = min(e1, n_elem - 1);
    const int64_t ti = (int64_t)blockIdx.x * kAdjBlock + threadIdx.x;
    const int64_t tc = min(ti, n_t - 1);
    const double x[3] = {tgt[tc * 3], tgt[tc * 3 + 1], tgt[tc * 3 + 2]};
    const double lm[3] = {lam[tc * 3], lam[tc * 3 + 1], lam[tc * 3 + 2]};
    double acc[3] = {0.0, 0.0, 0.0};
    if (e0 < e1) {
        std::conditional_t<kAlone, VtxA, VtxGrad<KER>> prev, v;
        auto vertex = [&](const Elem64& e, auto& o) {
            if constexpr (kAlone) vtxa(x, e.x, e.y, e.z, o);
            else vtx_grad<KER>(x, e.x, e.y, e.z, o);
        };
        auto scaled = [&](Elem64 e) {  // (a break's q stays negative)
            if (kAlone) return e;
            e.g *= kInv4Pi;
            if (KER == FJ_KERNEL_CUTOFF) e.q = e.q >= 0.0 ? rc2 * e.q : e.q;
            return e;
        };
        auto e2_of = [](const Elem64& e) { return kEps * kEps * (e.r0x * e.r0x + e.r0y * e.r0y + e.r0z * e.r0z); };
        Elem64 pl = scaled(st[e0]);
        double pe2 = e2_of(pl);
        vertex(pl, prev);
        bool far = beyond(x[0], x[1], x[2]) || beyond(pl.x, pl.y, pl.z);
        // (told per element staged, for the CTA: told per pair it cost 2 to 4 %)
        auto pairs = [&](int cnt, auto is_far) {
#pragma unroll 2
            for (int i = 0; i < cnt; ++i) {
                const Elem64 cur = sh[i];
                vertex(cur, v);
                if (pl.q >= 0.0) {
                    if constexpr (kAlone) {
                        const double r0[3] = {pl.r0x, pl.r0y, pl.r0z};
                        double g1[3], g2[3], lk;
                        link_vjp<KER>(prev, v, r0, pl.g, lm, rc2, g1, g2, lk);
                        for (int k = 0; k < 3; ++k) acc[k] += g1[k] + g2[k];
                    } else {
                        const FilGrad f = {{pl.r0x, pl.r0y, pl.r0z}, pl.g, pl.q, pe2};
                        target_grad<KER, decltype(is_far)::value>(prev, v, f, rc2, lm, acc);
                    }
                }
                prev = v;
                pl = cur;
                pe2 = se2[i];
            }
        };
        for (int64_t c0 = e0 + 1; c0 <= vend; c0 += kAdjBlock) {
            const int cnt = (int)min((int64_t)kAdjBlock, vend + 1 - c0);
            __syncthreads();
            if (threadIdx.x < cnt) {
                const Elem64 e = scaled(st[c0 + threadIdx.x]);
                sh[threadIdx.x] = e;
                se2[threadIdx.x] = e2_of(e);
                far = far || beyond(e.x, e.y, e.z);
            }
            far = __syncthreads_or(far);
            if (!kAlone && far) pairs(cnt, std::true_type());
            else pairs(cnt, std::false_type());
        }
    }
    if (ti < n_t) {
        double* o = part + ((int64_t)split * n_t + ti) * 3;
        for (int k = 0; k < 3; ++k) o[k] = acc[k];
    }
}

// Pass 2: filament adjoints.  Thread per stream element e (the link e -> e+1); targets
// of this CTA's split staged through shared memory.  Output per element and split:
// [y0_bar(3), y1_bar(3), g_bar].
template <int KER>
__global__ void __launch_bounds__(kAdjBlock, kAdjCtas)
    vjp_links_kernel(const double* __restrict__ tgt, const double* __restrict__ lam, int64_t n_t,
                     const Elem64* __restrict__ st, int64_t n_elem, int n_split, double rc2,
                     double* __restrict__ part) {
    __shared__ __align__(16) double sx[kAdjBlock][6];
    const int split = blockIdx.y;
    const int64_t per = (n_t + n_split - 1) / n_split;
    const int64_t t0 = (int64_t)split * per;
    const int64_t t1 = min(n_t, t0 + per);
    const int64_t e = (int64_t)blockIdx.x * kAdjBlock + threadIdx.x;
    const bool live = e + 1 < n_elem && st[min(e, n_elem - 1)].q >= 0.0;
    Elem64 a, b;
    if (live) {
        a = st[e];
        b = st[e + 1];
    } else {
        memset(&a, 0, sizeof(a));
        memset(&b, 0, sizeof(b));
    }
    const double r0sq = a.r0x * a.r0x + a.r0y * a.r0y + a.r0z * a.r0z, e4 = 4.0 * kEps * r0sq;
    const FilGrad f = {{a.r0x, a.r0y, a.r0z}, kInv4Pi * a.g, KER == FJ_KERNEL_CUTOFF ? rc2 * a.q : a.q,
                       kEps * kEps * r0sq};
    // (a filament of no length: a c of nothing but rounding would give its ends a direction)
    const bool counts = live && r0sq > 0.0;
    LinkGrad l;
    memset(&l, 0, sizeof(l));
    auto pairs = [&](int cnt, auto is_far) {
#pragma unroll 2
        for (int i = 0; i < cnt; ++i) {
            const double x[3] = {sx[i][0], sx[i][1], sx[i][2]};
            const double lm[3] = {sx[i][3], sx[i][4], sx[i][5]};
            VtxGrad<KER> A, B;
            vtx_grad<KER>(x, a.x, a.y, a.z, A);
            vtx_grad<KER>(x, b.x, b.y, b.z, B);
            link_grad<KER, decltype(is_far)::value>(A, B, f, rc2, e4, lm, l);
        }
    };
    bool far = beyond(a.x, a.y, a.z) || beyond(b.x, b.y, b.z);
    for (int64_t c0 = t0; c0 < t1; c0 += kAdjBlock) {
        const int cnt = (int)min((int64_t)kAdjBlock, t1 - c0);
        __syncthreads();
        if (threadIdx.x < cnt) {
            const int64_t t = c0 + threadIdx.x;
            for (int k = 0; k < 3; ++k) {
                sx[threadIdx.x][k] = tgt[t * 3 + k];
                sx[threadIdx.x][3 + k] = lam[t * 3 + k];
            }
            far = far || beyond(sx[threadIdx.x][0], sx[threadIdx.x][1], sx[threadIdx.x][2]);
        }
        far = __syncthreads_or(far);
        if (counts && far) pairs(cnt, std::true_type());
        else if (counts) pairs(cnt, std::false_type());
    }
    if (e < n_elem) {
        double* o = part + ((int64_t)split * n_elem + e) * 7;
        for (int k = 0; k < 3; ++k) {
            o[k] = l.e1 != 0.0 ? -fma(l.e1, f.r0[k], l.d1[k]) : -l.d1[k];  // (r0 may be infinite)
            o[3 + k] = l.e2 != 0.0 ? -fma(l.e2, f.r0[k], l.d2[k]) : -l.d2[k];
        }
        o[6] = kInv4Pi * l.k;
    }
}

__global__ void sum_splits_kernel(const double* __restrict__ part, int n_split, int64_t n, double* __restrict__ out,
                                  int accumulate) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    for (int k = 0; k < n_split; ++k) s += part[(int64_t)k * n + i];
    out[i] = accumulate ? out[i] + s : s;
}

// Element adjoints -> lattice vertex and ring-circulation adjoints (accumulated).
struct UnpackArgs {
    LatticeRef lat[kMaxPack];
    int64_t offset[kMaxPack + 1];
    double* zeta_bar[kMaxPack];   // per packed lattice (images point at their original)
    double* gamma_bar[kMaxPack];
    int n_lat;
    MirrorPlane mirror;
};

__global__ void unpack_vertices_kernel(UnpackArgs u, const double* __restrict__ el, int li) {
    const LatticeRef& L = u.lat[li];
    const int R = L.rows, C = L.cols;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= (int64_t)(R + 1) * (C + 1)) return;
    const int k = (int)(v / (C + 1)), l = (int)(v % (C + 1));
    const int64_t off = u.offset[li];
    const int64_t n_chord = (int64_t)(C + 1) * (R + 1);
    const int64_t ec = off + (int64_t)l * (R + 1) + k;        // chordwise chain element
    const int64_t es = off + n_chord + (int64_t)k * (C + 1) + l;  // spanwise chain element
    double y[3];
    for (int d = 0; d < 3; ++d) {
        double s = el[ec * 7 + d] + el[es * 7 + d];          // vertex as link start
        if (k > 0) s += el[(ec - 1) * 7 + 3 + d];             // vertex as end of chordwise link
        if (l > 0) s += el[(es - 1) * 7 + 3 + d];             // vertex as end of spanwise link
        y[d] = s;
    }
    if (L.mirrored) {  // y' = y - 2((y - p).n) n  =>  y_bar += (I - 2 n n^T) y'_bar
        const double* nn = u.mirror.nrm;
        const double dn = y[0] * nn[0] + y[1] * nn[1] + y[2] * nn[2];
        for (int d = 0; d < 3; ++d) y[d] -= 2.0 * dn * nn[d];
    }
    double* zb = u.zeta_bar[li] + v * 3;
    for (int d = 0; d < 3; ++d) zb[d] += y[d];
}

__global__ void unpack_gamma_kernel(UnpackArgs u, const double* __restrict__ el, int li) {
    const LatticeRef& L = u.lat[li];
    const int R = L.rows, C = L.cols;
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= (int64_t)R * C || u.gamma_bar[li] == nullptr) return;
    const int k = (int)(r / C), l = (int)(r % C);
    const int64_t off = u.offset[li];
    const int64_t n_chord = (int64_t)(C + 1) * (R + 1);
    auto gm = [&](int kk, int ll) { return el[(off + (int64_t)ll * (R + 1) + kk) * 7 + 6]; };
    auto gn = [&](int kk, int ll) { return el[(off + n_chord + (int64_t)kk * (C + 1) + ll) * 7 + 6]; };
    // G_eff_m[k,l] = G[k,l] - G[k,l-1];  G_eff_n[k,l] = G[k-1,l] - G[k,l]  (aero/aic.py:284-287)
    const double gbar = gm(k, l) - gm(k, l + 1) - gn(k, l) + gn(k + 1, l);
    u.gamma_bar[li][r] += (double)L.sign * gbar;
}

static int64_t vjp_elems(const int* rows, const int* cols, int n_lattices, int img) {
    int64_t n = 0;
    for (int i = 0; i < n_lattices; ++i) n += img * stream_len(rows[i], cols[i]);
    return n;
}

static int vjp_splits_t(int64_t n_t) { return (int)std::max<int64_t>(1, std::min<int64_t>(64, 1184 / std::max<int64_t>(1, (n_t + kAdjBlock - 1) / kAdjBlock))); }
// Targets per split of the links' sums, at least: 300 targets, 190 links 33 us with 64, 24 us with
// 16; more than 2000 targets the same.
constexpr int kMinTargets = 16;

static int vjp_splits_l(int64_t n_elem, int64_t n_t) {
    const int64_t ctas = (n_elem + kAdjBlock - 1) / kAdjBlock;
    return (int)std::max<int64_t>(1, std::min<int64_t>({64, 1184 / std::max<int64_t>(1, ctas), std::max<int64_t>(1, n_t / kMinTargets)}));
}

}  // namespace fj

using namespace fj;

extern "C" {

int fj_vind_vjp_workspace_size(int64_t n_targets, const int* rows, const int* cols, int n_lattices, int mirror,
                               size_t* bytes) {
    if (bytes == nullptr || n_targets < 0 || n_lattices < 0 || n_lattices > FJ_MAX_SURF * 2)
        return fail(FJ_ERR_SHAPE, "vind_vjp workspace: bad arguments");
    const int64_t ne = vjp_elems(rows, cols, n_lattices, mirror ? 2 : 1);
    const int64_t nt = std::max<int64_t>(n_targets, 1);
    Arena a(nullptr, 0);
    a.carve<Elem64>(ne);
    a.carve<double>((int64_t)vjp_splits_t(nt) * nt * 3);
    a.carve<double>((int64_t)vjp_splits_l(ne, nt) * std::max<int64_t>(ne, 1) * 7);
    a.carve<double>(std::max<int64_t>(ne, 1) * 7);
    *bytes = a.used + 256;
    return FJ_OK;
}

int fj_vind_vjp(const double* d_targets, int64_t n_targets, const double* const* d_zetas,
                const double* const* d_gammas, const int* rows, const int* cols, int n_lattices,
                const double* mirror_point, const double* mirror_normal, int kernel, double r_cut,
                const double* d_lam, double* d_targets_bar, double* const* d_zetas_bar, double* const* d_gammas_bar,
                void* d_ws, size_t ws_bytes, fj_stream_t stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (kernel != FJ_KERNEL_EPSILON && kernel != FJ_KERNEL_CUTOFF)
        return fail(FJ_ERR_UNSUPPORTED, "fj_vind_vjp: the epsilon and cutoff kernels have hand-written adjoints");
    const double rc2 = r_cut * r_cut;
    const int mirror = mirror_point != nullptr && mirror_normal != nullptr;
    const int img = mirror ? 2 : 1;
    size_t need;
    FJ_TRY(fj_vind_vjp_workspace_size(n_targets, rows, cols, n_lattices, mirror, &need));
    if (ws_bytes < need) return fail(FJ_ERR_NOMEM, "vind_vjp workspace %zu < %zu", ws_bytes, need);
    if (n_targets == 0) return FJ_OK;
    const int64_t ne = vjp_elems(rows, cols, n_lattices, img);
    if (ne == 0) return FJ_OK;  // nothing to accumulate
    const int st_split = vjp_splits_t(n_targets), l_split = vjp_splits_l(ne, n_targets);
    Arena a(d_ws, ws_bytes);
    Elem64* st = a.carve<Elem64>(ne);
    double* part_t = a.carve<double>((int64_t)st_split * n_targets * 3);
    double* part_l = a.carve<double>((int64_t)l_split * ne * 7);
    double* el = a.carve<double>(ne * 7);
    PackArgs pa;
    UnpackArgs ua;
    memset(&pa, 0, sizeof(pa));
    memset(&ua, 0, sizeof(ua));
    pa.kernel = kernel;
    pa.r_cut = r_cut;
    if (mirror)
        for (int d = 0; d < 3; ++d) {
            pa.mirror.p[d] = mirror_point[d];
            pa.mirror.nrm[d] = mirror_normal[d];
        }
    ua.mirror = pa.mirror;
    int n = 0;
    for (int i = 0; i < n_lattices; ++i) {
        for (int k = 0; k < img; ++k) {
            LatticeRef& L = pa.lat[n];
            L.zeta = d_zetas[i];
            L.gamma = d_gammas[i];
            L.rows = rows[i];
            L.cols = cols[i];
            L.sign = k ? -1.0f : 1.0f;
            L.mirrored = k;
            pa.offset[n + 1] = pa.offset[n] + stream_len(rows[i], cols[i]);
            ua.lat[n] = L;
            ua.offset[n] = pa.offset[n];
            ua.zeta_bar[n] = d_zetas_bar ? d_zetas_bar[i] : nullptr;
            ua.gamma_bar[n] = d_gammas_bar ? d_gammas_bar[i] : nullptr;
            ++n;
        }
    }
    pa.n_lat = n;
    ua.n_lat = n;
    ua.offset[n] = pa.offset[n];
    FJ_TRY(pack_stream64(pa, st, s));
    if (d_targets_bar) {
        dim3 g((unsigned)((n_targets + kAdjBlock - 1) / kAdjBlock), (unsigned)st_split);
        const bool alone = d_zetas_bar == nullptr && d_gammas_bar == nullptr;
        auto* fn = kernel == FJ_KERNEL_EPSILON
                       ? (alone ? vjp_targets_kernel<FJ_KERNEL_EPSILON, true>
                                : vjp_targets_kernel<FJ_KERNEL_EPSILON, false>)
                       : (alone ? vjp_targets_kernel<FJ_KERNEL_CUTOFF, true>
                                : vjp_targets_kernel<FJ_KERNEL_CUTOFF, false>);
        fn<<<g, kAdjBlock, 0, s>>>(d_targets, d_lam, n_targets, st, ne, st_split, rc2, part_t);
        note_launch();
        sum_splits_kernel<<<(unsigned)((n_targets * 3 + 255) / 256), 256, 0, s>>>(part_t, st_split, n_targets * 3,
                                                                                 d_targets_bar, 1); note_launch();
    }
    if (d_zetas_bar || d_gammas_bar) {
        dim3 g((unsigned)((ne + kAdjBlock - 1) / kAdjBlock), (unsigned)l_split);
        if (kernel == FJ_KERNEL_EPSILON)
            vjp_links_kernel<FJ_KERNEL_EPSILON><<<g, kAdjBlock, 0, s>>>(d_targets, d_lam, n_targets, st, ne, l_split,
                                                                        rc2, part_l);
        else
            vjp_links_kernel<FJ_KERNEL_CUTOFF><<<g, kAdjBlock, 0, s>>>(d_targets, d_lam, n_targets, st, ne, l_split,
                                                                       rc2, part_l);
        note_launch();
        FJ_TRY(reduce_sums(part_l, l_split, ne * 7, el, 0, 1.0, s));
        for (int li = 0; li < n; ++li) {
            const int64_t nv = (int64_t)(ua.lat[li].rows + 1) * (ua.lat[li].cols + 1);
            if (ua.zeta_bar[li]) {
                unpack_vertices_kernel<<<(unsigned)((nv + 255) / 256), 256, 0, s>>>(ua, el, li); note_launch();
            }
            const int64_t nr = (int64_t)ua.lat[li].rows * ua.lat[li].cols;
            if (ua.gamma_bar[li] && nr > 0) {
                unpack_gamma_kernel<<<(unsigned)((nr + 255) / 256), 256, 0, s>>>(ua, el, li); note_launch();
            }
        }
    }
    FJ_LAUNCH_CHECK("fj_vind_vjp");
    return FJ_OK;
}

int fj_lu_solve_t(const double* d_lu, int n, const int32_t* d_piv, double* d_b, void* d_ws, size_t ws_bytes,
                  fj_stream_t stream) {
    if (ws_bytes < 256 + (size_t)n * sizeof(double)) return fail(FJ_ERR_NOMEM, "lu_solve_t workspace too small");
    if (n <= 0) return fail(FJ_ERR_SHAPE, "lu_solve_t: n=%d", n);
    // A = P^T L U  =>  U^T L^T (P x) = b
    return lu_substitute64(d_lu, n, d_piv, d_b, (double*)((char*)d_ws + 256), true, (cudaStream_t)stream);
}

}  // extern "C"
