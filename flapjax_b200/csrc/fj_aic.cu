// fj_aic.cu -- bound-on-collocation influence matrix (compute_aic_solve, aero/aic.py:11-205).
//
// A CTA takes kAicT collocation points (rows of the AIC).  For each source surface it evaluates
// the influence of every chordwise and spanwise filament at c_i, projects it on the area normal
// n_i (aero/aic.py:47-54) into shared memory, and combines filaments into rings as
// -diff(m, axis=1) + diff(n, axis=0) (aero/aic.py:55-57), so each filament is evaluated once per
// target, in FP64.  Mirror images are assembled the same way and subtracted ring by ring
// (aero/aic.py:101-110).  In the static solve the wake rings' influence, summed over wake
// rows, is added to the trailing-edge column (add_wake_influence, aero/aic.py:190-205).
//
// What bounds it: the FP64 pipe at large counts, else the latency of a thread's few pairs.
//   * A thread per vertex evaluates the filaments to its right and downstream neighbours, for
//     two targets: the vertex's work is shared by two filaments, its loads by both targets, and
//     the two targets' chains overlap.  One target where two exceed shared memory.
//   * Down a strip of the wake neighbouring rings share their spanwise filament with opposite
//     signs, so the sum over rows is the chordwise filaments' plus the first and the last
//     spanwise one: a quarter of the rings' evaluations.  Every thread takes a stretch of a
//     chordwise column, whose chain shares its vertices.
// Assembly with its geometry, epsilon (cutoff) kernel: 12 x 64 rings 20.6 -> 16.5 us (22.7 -> 16.5),
// 16 x 128 80 -> 60 us (93 -> 61); with the wake's lumping, 8 x 32 + 64 rows 135 -> 16.5 us
// (160 -> 16.5), 12 x 64 + 120 rows 507 -> 57 us (610 -> 60), against a thread per filament and a
// thread per strip over all its rings.  At 16 x 128, one target a CTA: 67 (69) us; four: 79 (81);
// two or four CTAs on an SM for three: 61 (64) and 68 (84).
#include "fj_aic.cuh"
#include "fj_bs.cuh"

namespace fj {

constexpr int kAicThreads = 256;
constexpr int kAicT = 2;  // targets of a CTA

__device__ __forceinline__ void load_vertex(const double* zeta, int64_t v, bool mirrored, const MirrorPlane& mp,
                                            double (&o)[3]) {
    o[0] = zeta[v * 3];
    o[1] = zeta[v * 3 + 1];
    o[2] = zeta[v * 3 + 2];
    if (mirrored) {
        const double dn = (o[0] - mp.p[0]) * mp.nrm[0] + (o[1] - mp.p[1]) * mp.nrm[1] + (o[2] - mp.p[2]) * mp.nrm[2];
#pragma unroll
        for (int d = 0; d < 3; ++d) o[d] -= 2.0 * dn * mp.nrm[d];
    }
}

// The targets of a CTA, their normals over 4 pi (the sums' common factor).
template <int T>
struct AicTargets {
    double x[T][3], nrm[T][3];
};

// Influence of the filament p0 -> p1 projected on the normals; A, B: its ends as the targets see them.
template <int KER, int T>
__device__ __forceinline__ void influence(const AicTargets<T>& t, const double (&p0)[3], const double (&p1)[3],
                                          const Vtx64<KER> (&A)[T], const Vtx64<KER> (&B)[T], double rc2,
                                          double (&inf)[T]) {
    const double r0x = p1[0] - p0[0], r0y = p1[1] - p0[1], r0z = p1[2] - p0[2];
    double k[T][3];
#pragma unroll
    for (int j = 0; j < T; ++j) k[j][0] = k[j][1] = k[j][2] = 0.0;
    link64<KER, T>(A, B, 1.0, r0x, r0y, r0z, link_q<KER>(r0x * r0x + r0y * r0y + r0z * r0z, rc2), rc2, k);
#pragma unroll
    for (int j = 0; j < T; ++j) inf[j] = k[j][0] * t.nrm[j][0] + k[j][1] * t.nrm[j][1] + k[j][2] * t.nrm[j][2];
}

template <int KER, int T>
__device__ __forceinline__ void see(const AicTargets<T>& t, const double (&p)[3], Vtx64<KER> (&o)[T]) {
#pragma unroll
    for (int j = 0; j < T; ++j) vtx64<KER>(t.x[j], p[0], p[1], p[2], o[j]);
}

// The wake of one surface lumped onto its trailing-edge column (static solve).
template <int KER, int T>
__device__ __forceinline__ void lump_wake(const AicArgs& a, const AicTargets<T>& t, int64_t i0, int sb, double* sm) {
    const int W = a.m_star[sb], C = a.n[sb], C1 = C + 1, n_img = a.mirror ? 2 : 1;
    const double* zw = a.zeta_w[sb];
    const int n_part = max(1, kAicThreads / C1), per = (W + n_part - 1) / n_part;
    double* chord = sm;                    // [n_part][T][C1]: a stretch's chordwise filaments
    double* span = sm + n_part * T * C1;   // [2][T][C]: the first and the last spanwise ones
    for (int u = threadIdx.x; u < n_part * C1 + 2 * C; u += kAicThreads) {
        double sum[T], inf[T], p0[3], p1[3];
#pragma unroll
        for (int j = 0; j < T; ++j) sum[j] = 0.0;
        const bool column = u < n_part * C1;
        const int v = u - n_part * C1, part = u / C1, l = column ? u % C1 : v % C;
        // the chain of vertices, `step` apart
        const int r0 = column ? part * per : v / C * W, r1 = column ? min(W, r0 + per) : r0 + 1;
        const int step = column ? C1 : 1;
        for (int img = 0; img < n_img && r0 < r1; ++img) {
            Vtx64<KER> A[T], B[T];
            int64_t q = (int64_t)r0 * C1 + l;
            load_vertex(zw, q, img == 1, a.mp, p0);
            see<KER, T>(t, p0, A);
            for (int r = r0; r < r1; ++r) {
                q += step;
                load_vertex(zw, q, img == 1, a.mp, p1);
                see<KER, T>(t, p1, B);
                influence<KER, T>(t, p0, p1, A, B, a.rc2, inf);
#pragma unroll
                for (int j = 0; j < T; ++j) {
                    sum[j] += img == 0 ? inf[j] : -inf[j];
                    A[j] = B[j];
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) p0[d] = p1[d];
            }
        }
#pragma unroll
        for (int j = 0; j < T; ++j) {
            if (column) chord[(part * T + j) * C1 + l] = sum[j];
            else span[(v / C * T + j) * C + l] = sum[j];
        }
    }
    __syncthreads();
    for (int u = threadIdx.x; u < T * C; u += kAicThreads) {
        const int j = u / C, l = u % C;
        if (i0 + j >= a.n_rows) continue;
        double total = span[(T + j) * C + l] - span[j * C + l];
        for (int q = 0; q < n_part; ++q) total -= chord[(q * T + j) * C1 + l + 1] - chord[(q * T + j) * C1 + l];
        a.aic[(i0 + j) * a.ld + a.col_off[sb] + (a.m[sb] - 1) * C + l] += total;
    }
}

template <int KER, int T>
__device__ __forceinline__ void aic_rows(const AicArgs& a, int64_t i0, double* sm_inf) {
    AicTargets<T> t;
#pragma unroll
    for (int j = 0; j < T; ++j)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int64_t i = min(i0 + j, a.n_rows - 1);
            t.x[j][d] = a.c[i * 3 + d];
            t.nrm[j][d] = kInv4Pi * a.nc[i * 3 + d];
        }
    const int n_img = a.mirror ? 2 : 1;

    for (int sb = 0; sb < a.n_surf; ++sb) {
        const int R = a.m[sb], C = a.n[sb], C1 = C + 1;
        const int nm = R * C1;
        const double* zeta = a.zeta_b[sb];
        __syncthreads();
        for (int v = threadIdx.x; v < (R + 1) * C1; v += kAicThreads) {
            const int k = v / C1, l = v % C1;
            for (int img = 0; img < n_img; ++img) {
                double* buf = sm_inf + img * T * a.max_fil;
                double p0[3], p1[3], inf[T];
                Vtx64<KER> A[T], B[T];
                load_vertex(zeta, v, img == 1, a.mp, p0);
                see<KER, T>(t, p0, A);
                if (k < R) {  // chordwise, m[k][l]
                    load_vertex(zeta, v + C1, img == 1, a.mp, p1);
                    see<KER, T>(t, p1, B);
                    influence<KER, T>(t, p0, p1, A, B, a.rc2, inf);
#pragma unroll
                    for (int j = 0; j < T; ++j) buf[j * a.max_fil + v] = inf[j];
                }
                if (l < C) {  // spanwise, n[k][l]
                    load_vertex(zeta, v + 1, img == 1, a.mp, p1);
                    see<KER, T>(t, p1, B);
                    influence<KER, T>(t, p0, p1, A, B, a.rc2, inf);
#pragma unroll
                    for (int j = 0; j < T; ++j) buf[j * a.max_fil + nm + v - k] = inf[j];
                }
            }
        }
        __syncthreads();
        for (int r = threadIdx.x; r < R * C; r += kAicThreads) {
            const int k = r / C;
#pragma unroll
            for (int j = 0; j < T; ++j) {
                if (i0 + j >= a.n_rows) continue;
                double v = 0.0;
                for (int img = 0; img < n_img; ++img) {
                    const double* m_inf = sm_inf + (img * T + j) * a.max_fil + r + k;  // m[k][l]
                    const double* n_inf = sm_inf + (img * T + j) * a.max_fil + nm + r;  // n[k][l]
                    const double ring = -(m_inf[1] - m_inf[0]) + (n_inf[C] - n_inf[0]);
                    v = img == 0 ? ring : v - ring;
                }
                a.aic[(i0 + j) * a.ld + a.col_off[sb] + r] = v;
            }
        }
        if (a.zeta_w[sb] != nullptr && a.m_star[sb] > 0) {
            __syncthreads();
            lump_wake<KER, T>(a, t, i0, sb, sm_inf);
        }
    }
}

// (Two CTAs on an SM here and three below: with the arguments read from the table three spill, 167 us
// for 147 on 16 wings.)
template <int KER, int T>
__global__ void __launch_bounds__(kAicThreads, 2) aic_jobs_kernel(const AicArgs* __restrict__ tab) {
    const AicArgs& a = tab[blockIdx.y];
    if ((int64_t)blockIdx.x * T >= a.n_rows) return;
    if (a.run_flag != nullptr && *a.run_flag == 0) return;
    extern __shared__ double sm_inf[];
    aic_rows<KER, T>(a, (int64_t)blockIdx.x * T, sm_inf);
}

template <int KER, int T>
__global__ void __launch_bounds__(kAicThreads, 3) aic_kernel(AicArgs a, const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;
    extern __shared__ double sm_inf[];  // [images][T][max filaments], or the wake's partial sums
    aic_rows<KER, T>(a, (int64_t)blockIdx.x * T, sm_inf);
}

// Targets of a CTA: two, unless their filaments leave no room for two CTAs on an SM.
static int aic_targets(int n_img, int max_fil, size_t* smem) {
    auto bytes = [&](int t) { return (size_t)t * ((size_t)n_img * max_fil + kAicThreads) * sizeof(double); };
    const int t = bytes(kAicT) <= 100 * 1024 ? kAicT : 1;
    *smem = bytes(t);
    return t;
}

static int aic_check(int n_img, int max_fil) {
    if ((size_t)n_img * max_fil * sizeof(double) > 200 * 1024)
        return fail(FJ_ERR_UNSUPPORTED, "aic: a surface with %d filaments exceeds shared memory", max_fil);
    return FJ_OK;
}

int aic_launch_jobs(const AicArgs* d_tab, int n_jobs, int64_t max_rows, int max_fil, int any_mirror, int kernel,
                    cudaStream_t s) {
    const int n_img = any_mirror ? 2 : 1;
    FJ_TRY(aic_check(n_img, max_fil));
    if (n_jobs == 0 || max_rows == 0) return FJ_OK;
    size_t smem;
    const int t = aic_targets(n_img, max_fil, &smem);
    void (*fn)(const AicArgs*) = nullptr;
    switch (kernel) {
        case FJ_KERNEL_EPSILON:
            fn = t == 1 ? aic_jobs_kernel<FJ_KERNEL_EPSILON, 1> : aic_jobs_kernel<FJ_KERNEL_EPSILON, kAicT>;
            break;
        case FJ_KERNEL_CUTOFF:
            fn = t == 1 ? aic_jobs_kernel<FJ_KERNEL_CUTOFF, 1> : aic_jobs_kernel<FJ_KERNEL_CUTOFF, kAicT>;
            break;
        case FJ_KERNEL_PLAIN:
            fn = t == 1 ? aic_jobs_kernel<FJ_KERNEL_PLAIN, 1> : aic_jobs_kernel<FJ_KERNEL_PLAIN, kAicT>;
            break;
        default:
            return fail(FJ_ERR_UNSUPPORTED, "aic: unknown kernel %d", kernel);
    }
    FJ_TRY(allow_dynamic_smem((const void*)fn, smem));
    fn<<<dim3((unsigned)((max_rows + t - 1) / t), (unsigned)n_jobs), kAicThreads, smem, s>>>(d_tab); note_launch();
    FJ_LAUNCH_CHECK("aic_jobs_kernel");
    return FJ_OK;
}

int aic_launch(const AicArgs& a, const int* d_run_flag, cudaStream_t s) {
    const int n_img = a.mirror ? 2 : 1;
    FJ_TRY(aic_check(n_img, a.max_fil));
    if (a.n_rows == 0) return FJ_OK;
    size_t smem;
    const int t = aic_targets(n_img, a.max_fil, &smem);
    void (*fn)(AicArgs, const int*) = nullptr;
    switch (a.kernel) {
        case FJ_KERNEL_EPSILON:
            fn = t == 1 ? aic_kernel<FJ_KERNEL_EPSILON, 1> : aic_kernel<FJ_KERNEL_EPSILON, kAicT>;
            break;
        case FJ_KERNEL_CUTOFF:
            fn = t == 1 ? aic_kernel<FJ_KERNEL_CUTOFF, 1> : aic_kernel<FJ_KERNEL_CUTOFF, kAicT>;
            break;
        case FJ_KERNEL_PLAIN:
            fn = t == 1 ? aic_kernel<FJ_KERNEL_PLAIN, 1> : aic_kernel<FJ_KERNEL_PLAIN, kAicT>;
            break;
        default:
            return fail(FJ_ERR_UNSUPPORTED, "aic: unknown kernel %d", a.kernel);
    }
    FJ_TRY(allow_dynamic_smem((const void*)fn, smem));
    fn<<<(unsigned)((a.n_rows + t - 1) / t), kAicThreads, smem, s>>>(a, d_run_flag); note_launch();
    FJ_LAUNCH_CHECK("aic_kernel");
    return FJ_OK;
}

}  // namespace fj
