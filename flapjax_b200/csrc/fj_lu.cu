// fj_lu.cu -- the dense AIC solve (jnp.linalg.solve, aero/uvlm.py:985).
//
// lu_factor*: blocked right-looking LU with partial pivoting (the LAPACK getrf
// algorithm family XLA calls).  Per panel of NB columns:
//   1. one CTA factors the (n-k) x NB panel held in shared memory (pivot search by
//      block arg-max with LAPACK's first-maximum tie rule, row swap, scale, rank-1);
//   2. the panel's row swaps are applied to the other columns, and U12 = L11^-1 A12;
//   3. the trailing matrix is updated, A22 -= L21 U12.
// lu_inverse32 + refine_solve: the mixed-precision solve.  FP32 factors give an FP32
// explicit inverse X once per factorisation; every solve is then GEMVs over all SMs:
// x = X b, r = b - A x in FP64, x += X r.
#include <climits>
#include <cstdlib>
#include <cstring>

#include "fj_lu.cuh"
#include "fj_panel.cuh"
#include "fj_tc.cuh"
#include "fj_trsv.cuh"

namespace fj {

template <typename T>
__device__ __forceinline__ T absval(T v) {
    return v < T(0) ? -v : v;
}

template <typename T, int NB>
__global__ void __launch_bounds__(1024) lu_panel_kernel(T* __restrict__ a, int n, int k,
                                                        int32_t* __restrict__ piv, int* __restrict__ info,
                                                        const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    T* P = reinterpret_cast<T*>(smraw);  // (n-k) x LDP, row-major; odd stride avoids bank conflicts
    constexpr int LDP = NB + 1;
    __shared__ T s_val[32];
    __shared__ int s_idx[32];
    const int rows = n - k;
    const int nb = min(NB, rows);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    // asynchronous copies of the panel: every element in flight at once (columns past nb
    // zero-filled)
    for (int idx = threadIdx.x; idx < rows * NB; idx += blockDim.x) {
        const int r = idx / NB, c = idx % NB;
        const T* src = a + (int64_t)(k + r) * n + k + min(c, nb - 1);
        const unsigned dst = (unsigned)__cvta_generic_to_shared(P + r * LDP + c);
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(sizeof(T)),
                     "r"(c < nb ? (int)sizeof(T) : 0)
                     : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int j = 0; j < nb; ++j) {
        T best = T(-1);
        int bi = INT_MAX;
        for (int r = j + threadIdx.x; r < rows; r += blockDim.x) {
            const T v = absval(P[r * LDP + j]);
            if (v > best) {
                best = v;
                bi = r;
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const T ov = __shfl_down_sync(0xffffffffu, best, off);
            const int oi = __shfl_down_sync(0xffffffffu, bi, off);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            s_val[warp] = best;
            s_idx[warp] = bi;
        }
        __syncthreads();
        // every warp reduces the partials itself: no second barrier
        best = lane < nwarps ? s_val[lane] : T(-1);
        bi = lane < nwarps ? s_idx[lane] : INT_MAX;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, best, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        const int p = (bi == INT_MAX) ? j : bi;  // all-NaN column: keep the diagonal
        if (threadIdx.x == 0) piv[k + j] = k + p;
        if (p != j && threadIdx.x < NB) {
            const T t = P[j * LDP + threadIdx.x];
            P[j * LDP + threadIdx.x] = P[p * LDP + threadIdx.x];
            P[p * LDP + threadIdx.x] = t;
        }
        __syncthreads();
        const T pv = P[j * LDP + j];
        if (pv == T(0)) {
            if (threadIdx.x == 0 && *info == 0) *info = k + j + 1;
        } else {
            for (int r = j + 1 + threadIdx.x; r < rows; r += blockDim.x) {
                const T l = P[r * LDP + j] / pv;
                P[r * LDP + j] = l;
                for (int c = j + 1; c < nb; ++c) P[r * LDP + c] -= l * P[j * LDP + c];
            }
        }
        __syncthreads();
    }
#pragma unroll 8
    for (int idx = threadIdx.x; idx < rows * NB; idx += blockDim.x) {
        const int r = idx / NB, c = idx % NB;
        if (c < nb) a[(int64_t)(k + r) * n + k + c] = P[r * LDP + c];
    }
}

// The same panel with its rows in registers, for panels of at most RPT * 1024 rows.  The
// panel comes in and goes out through shared memory (coalesced cp.async loads and row-
// contiguous stores, as lu_panel_kernel); between, thread t owns rows t + 1024 i (i < RPT)
// in registers, and a column costs two barriers: one to combine the warps' pivot
// candidates, one to exchange the pivot row and row j.  Pivots (first maximum, as getrf)
// and every arithmetic operation are those of lu_panel_kernel, so the factors are bitwise
// the same.
template <typename T, int NB, int RPT>
__global__ void __launch_bounds__(1024) lu_panel_reg_kernel(T* __restrict__ a, int n, int k,
                                                            int32_t* __restrict__ piv, int* __restrict__ info,
                                                            const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    T* P = reinterpret_cast<T*>(smraw);  // (n-k) x LDP staging
    constexpr int LDP = NB + 1;
    __shared__ T s_val[32];
    __shared__ int s_idx[32];
    __shared__ T s_rowp[NB], s_rowj[NB];
    const int rows = n - k;
    const int nb = min(NB, rows);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    for (int idx = tid; idx < rows * NB; idx += blockDim.x) {
        const int r = idx / NB, c = idx % NB;
        const T* src = a + (int64_t)(k + r) * n + k + min(c, nb - 1);
        const unsigned dst = (unsigned)__cvta_generic_to_shared(P + r * LDP + c);
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(sizeof(T)),
                     "r"(c < nb ? (int)sizeof(T) : 0)
                     : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    T v[RPT][NB];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = tid + i * (int)blockDim.x;
#pragma unroll
        for (int c = 0; c < NB; ++c) v[i][c] = r < rows ? P[r * LDP + c] : T(0);
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        if (j >= nb) break;  // uniform over the CTA
        T best = T(-1);
        int bi = INT_MAX;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + i * (int)blockDim.x;
            if (r >= j && r < rows) {
                const T x = absval(v[i][j]);
                if (x > best) {
                    best = x;
                    bi = r;
                }
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const T ov = __shfl_down_sync(0xffffffffu, best, off);
            const int oi = __shfl_down_sync(0xffffffffu, bi, off);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            s_val[warp] = best;
            s_idx[warp] = bi;
        }
        __syncthreads();
        best = lane < nwarps ? s_val[lane] : T(-1);
        bi = lane < nwarps ? s_idx[lane] : INT_MAX;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, best, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        const int p = (bi == INT_MAX) ? j : bi;  // all-NaN column: keep the diagonal
        if (tid == 0) piv[k + j] = k + p;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {  // the owners of rows p and j publish them
            const int r = tid + i * (int)blockDim.x;
            if (r == p) {
#pragma unroll
                for (int c = 0; c < NB; ++c) s_rowp[c] = v[i][c];
            }
            if (r == j) {
#pragma unroll
                for (int c = 0; c < NB; ++c) s_rowj[c] = v[i][c];
            }
        }
        __syncthreads();
        if (p != j) {  // the swap: row j takes the pivot row, row p takes row j
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = tid + i * (int)blockDim.x;
                if (r == j) {
#pragma unroll
                    for (int c = 0; c < NB; ++c) v[i][c] = s_rowp[c];
                }
                if (r == p) {
#pragma unroll
                    for (int c = 0; c < NB; ++c) v[i][c] = s_rowj[c];
                }
            }
        }
        const T pv = s_rowp[j];
        if (pv == T(0)) {
            if (tid == 0 && *info == 0) *info = k + j + 1;
        } else {
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = tid + i * (int)blockDim.x;
                if (r > j && r < rows) {
                    const T l = v[i][j] / pv;
                    v[i][j] = l;
#pragma unroll
                    for (int c = j + 1; c < NB; ++c)
                        if (c < nb) v[i][c] -= l * s_rowp[c];
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = tid + i * (int)blockDim.x;
        if (r < rows) {
#pragma unroll
            for (int c = 0; c < NB; ++c) P[r * LDP + c] = v[i][c];
        }
    }
    __syncthreads();
    for (int idx = tid; idx < rows * NB; idx += blockDim.x) {
        const int r = idx / NB, c = idx % NB;
        if (c < nb) a[(int64_t)(k + r) * n + k + c] = P[r * LDP + c];
    }
}

// One panel at column k: the register form where its rows fit (at most 2048), else the
// shared-memory form; both stage the panel in the same dynamic shared memory.
template <typename T, int NB>
static void launch_panel(T* a, int n, int k, int32_t* piv, int* info, const int* run_flag, cudaStream_t s) {
    const int rows = n - k;
    const size_t smem = (size_t)rows * (NB + 1) * sizeof(T);
    if (rows <= 1024)
        lu_panel_reg_kernel<T, NB, 1><<<1, 1024, smem, s>>>(a, n, k, piv, info, run_flag);
    else if (rows <= 2048)
        lu_panel_reg_kernel<T, NB, 2><<<1, 1024, smem, s>>>(a, n, k, piv, info, run_flag);
    else
        lu_panel_kernel<T, NB><<<1, 1024, smem, s>>>(a, n, k, piv, info, run_flag);
    note_launch();
}

// Row swaps of the panel at column k for every other column; U12 = L11^-1 A12 for the
// columns [k + nb, c_end).  The panel's swaps (applied in order, as getrf) compose to one
// permutation of the at most 2 NB rows they touch; thread 0 works it out in shared memory,
// then each column thread loads all the touched values before storing any, one memory
// round trip instead of one per swap.
template <typename T, int NB>
__global__ void lu_swap_trsm_kernel(T* __restrict__ a, int n, int k, const int32_t* __restrict__ piv, int c_end,
                                    const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;
    __shared__ int s_dst[2 * NB], s_src[2 * NB], s_piv[NB];
    __shared__ int s_cnt;
    __shared__ T s_l[NB][NB];  // the panel's unit-lower diagonal block, for the triangular solve
    const int nb = min(NB, n - k);
    if (threadIdx.x < nb) s_piv[threadIdx.x] = piv[k + threadIdx.x];
    for (int idx = threadIdx.x; idx < NB * NB; idx += blockDim.x) {
        const int r = idx / NB, c = idx % NB;
        s_l[r][c] = (r < nb && c < r) ? a[(int64_t)(k + r) * n + k + c] : T(0);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int cnt = 0;
        for (int jj = 0; jj < nb; ++jj) {
            const int r1 = k + jj, r2 = s_piv[jj];
            if (r1 == r2) continue;
            int i1 = -1, i2 = -1;
            for (int e = 0; e < cnt; ++e) {
                if (s_dst[e] == r1) i1 = e;
                if (s_dst[e] == r2) i2 = e;
            }
            if (i1 < 0) {
                i1 = cnt++;
                s_dst[i1] = r1;
                s_src[i1] = r1;
            }
            if (i2 < 0) {
                i2 = cnt++;
                s_dst[i2] = r2;
                s_src[i2] = r2;
            }
            const int tmp = s_src[i1];
            s_src[i1] = s_src[i2];
            s_src[i2] = tmp;
        }
        s_cnt = cnt;
    }
    __syncthreads();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n || (c >= k && c < k + nb)) return;
    const int cnt = s_cnt;
    T val[2 * NB];
#pragma unroll
    for (int e = 0; e < 2 * NB; ++e)
        if (e < cnt) val[e] = a[(int64_t)s_src[e] * n + c];
#pragma unroll
    for (int e = 0; e < 2 * NB; ++e)
        if (e < cnt) a[(int64_t)s_dst[e] * n + c] = val[e];
    if (c >= k + nb && c < c_end) {
        T u[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j)
            if (j < nb) u[j] = a[(int64_t)(k + j) * n + c];
#pragma unroll
        for (int j = 1; j < NB; ++j) {
            if (j < nb) {
                T s = u[j];
#pragma unroll
                for (int jj = 0; jj < j; ++jj) s -= s_l[j][jj] * u[jj];
                u[j] = s;
            }
        }
#pragma unroll
        for (int j = 1; j < NB; ++j)
            if (j < nb) a[(int64_t)(k + j) * n + c] = u[j];
    }
}

// A[r0.., c0..] -= L[., k..k+NB) U[k..k+NB, .] on one 64 x 64 tile, rows < r_end and
// columns < c_end.
template <typename T, int NB>
__device__ __forceinline__ void lu_update_tile(T* __restrict__ a, int n, int k, int r0, int c0, int r_end,
                                               int c_end) {
    __shared__ T Ls[64][NB + 1];
    __shared__ T Us[NB][64];
    for (int idx = threadIdx.x; idx < 64 * NB; idx += blockDim.x) {
        const int r = idx / NB, j = idx % NB;
        Ls[r][j] = (r0 + r < r_end) ? a[(int64_t)(r0 + r) * n + k + j] : T(0);
        const int jj = idx / 64, c = idx % 64;
        Us[jj][c] = (c0 + c < c_end) ? a[(int64_t)(k + jj) * n + c0 + c] : T(0);
    }
    // the 16 elements of this thread are loaded before any is computed: one memory round
    // trip per tile
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    T acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = ty + 16 * p, c = tx + 16 * q;
            acc[p][q] = (r0 + r < r_end && c0 + c < c_end) ? a[(int64_t)(r0 + r) * n + c0 + c] : T(0);
        }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = ty + 16 * p, c = tx + 16 * q;
#pragma unroll
            for (int j = 0; j < NB; ++j) acc[p][q] -= Ls[r][j] * Us[j][c];
        }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = ty + 16 * p, c = tx + 16 * q;
            if (r0 + r < r_end && c0 + c < c_end) a[(int64_t)(r0 + r) * n + c0 + c] = acc[p][q];
        }
}

// A22 -= L21 U12 over rows [k + NB, n) and columns [k + NB, c_end).
template <typename T, int NB>
__global__ void __launch_bounds__(256) lu_update_kernel(T* __restrict__ a, int n, int k, int c_end,
                                                        const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;
    const int k2 = k + NB;
    lu_update_tile<T, NB>(a, n, k, k2 + blockIdx.y * 64, k2 + blockIdx.x * 64, n, c_end);
}

template <typename T, int NB>
static int lu_factor_impl(T* a, int n, int32_t* piv, int* d_info, cudaStream_t s, const int* run_flag) {
    if (n <= 0) return fail(FJ_ERR_SHAPE, "lu_factor: n=%d", n);
    const size_t smem = (size_t)n * (NB + 1) * sizeof(T);
    if (smem > 220 * 1024) return fail(FJ_ERR_UNSUPPORTED, "lu_factor: n=%d too large for the shared-memory panel", n);
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_kernel<T, NB>, (size_t)smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_reg_kernel<T, NB, 1>, (size_t)smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_reg_kernel<T, NB, 2>, (size_t)smem));
    FJ_CUDA(cudaMemsetAsync(d_info, 0, sizeof(int), s));
    for (int k = 0; k < n; k += NB) {
        const int nb = min(NB, n - k);
        launch_panel<T, NB>(a, n, k, piv, d_info, run_flag, s);
        if (n > nb) {
            lu_swap_trsm_kernel<T, NB><<<(n + 255) / 256, 256, 0, s>>>(a, n, k, piv, n, run_flag); note_launch();
        }
        const int rem = n - k - nb;
        if (rem > 0) {
            dim3 g((rem + 63) / 64, (rem + 63) / 64);
            lu_update_kernel<T, NB><<<g, 256, 0, s>>>(a, n, k, n, run_flag); note_launch();
        }
    }
    FJ_LAUNCH_CHECK("lu_factor");
    return FJ_OK;
}

// Panel width: the widest whose (n x (NB + 1)) panel fits the shared-memory budget, so that
// the largest validated AIC order (6144) factors too.
template <typename T>
static bool panel_fits(int n, int nb) {
    return (size_t)n * (nb + 1) * sizeof(T) <= (size_t)220 * 1024;
}

int lu_solve64(const double* lu, int n, const int32_t* piv, double* b, double* work, cudaStream_t s) {
    if (n <= 0) return fail(FJ_ERR_SHAPE, "lu_solve: n=%d", n);
    return lu_substitute64(lu, n, piv, b, work, false, s);
}

int lu_factor32(float* a, int n, int32_t* piv, int* d_info, cudaStream_t s) {
    if (panel_fits<float>(n, 16)) return lu_factor_impl<float, 16>(a, n, piv, d_info, s, nullptr);
    return lu_factor_impl<float, 8>(a, n, piv, d_info, s, nullptr);
}

// ---------------------------------------------------------------------------------
// Explicit inverse from FP32 factors: each CTA solves for 16 columns of the identity.
constexpr int kInvCols = 16;

__global__ void __launch_bounds__(512) lu_inverse32_kernel(const float* __restrict__ lu, int n,
                                                           const int32_t* __restrict__ piv,
                                                           float* __restrict__ xout) {
    extern __shared__ float B[];  // n x kInvCols
    const int c0 = blockIdx.x * kInvCols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int idx = threadIdx.x; idx < n * kInvCols; idx += blockDim.x) {
        const int i = idx / kInvCols, c = idx % kInvCols;
        B[idx] = (i == c0 + c) ? 1.0f : 0.0f;
    }
    __syncthreads();
    if (threadIdx.x < kInvCols) {  // B <- P B, swaps in getrf order
        const int c = threadIdx.x;
        for (int i = 0; i < n; ++i) {
            const int p = piv[i];
            if (p != i) {
                const float t = B[i * kInvCols + c];
                B[i * kInvCols + c] = B[p * kInvCols + c];
                B[p * kInvCols + c] = t;
            }
        }
    }
    __syncthreads();
    const int r = threadIdx.x / kInvCols;  // 0..31
    const int c = threadIdx.x % kInvCols;
    // forward: unit lower
    for (int i0 = 0; i0 < n; i0 += 32) {
        const int bw = min(32, n - i0);
        if (r < bw) {
            const float* row = lu + (int64_t)(i0 + r) * n;
            float sacc = B[(i0 + r) * kInvCols + c];
            for (int j = 0; j < i0; ++j) sacc -= row[j] * B[j * kInvCols + c];
            B[(i0 + r) * kInvCols + c] = sacc;
        }
        __syncthreads();
        if (warp < kInvCols) {
            const int cc = warp;
            float v = lane < bw ? B[(i0 + lane) * kInvCols + cc] : 0.0f;
            for (int jj = 0; jj < bw; ++jj) {
                const float xj = __shfl_sync(0xffffffffu, v, jj);
                if (lane > jj && lane < bw) v -= lu[(int64_t)(i0 + lane) * n + i0 + jj] * xj;
            }
            if (lane < bw) B[(i0 + lane) * kInvCols + cc] = v;
        }
        __syncthreads();
    }
    // backward: upper
    for (int i0 = ((n - 1) / 32) * 32; i0 >= 0; i0 -= 32) {
        const int be = min(i0 + 32, n);
        const int bw = be - i0;
        if (r < bw) {
            const float* row = lu + (int64_t)(i0 + r) * n;
            float sacc = B[(i0 + r) * kInvCols + c];
            for (int j = be; j < n; ++j) sacc -= row[j] * B[j * kInvCols + c];
            B[(i0 + r) * kInvCols + c] = sacc;
        }
        __syncthreads();
        if (warp < kInvCols) {
            const int cc = warp;
            float v = lane < bw ? B[(i0 + lane) * kInvCols + cc] : 0.0f;
            for (int jj = bw - 1; jj >= 0; --jj) {
                if (lane == jj) v = v / lu[(int64_t)(i0 + jj) * n + i0 + jj];
                const float xj = __shfl_sync(0xffffffffu, v, jj);
                if (lane < jj) v -= lu[(int64_t)(i0 + lane) * n + i0 + jj] * xj;
            }
            if (lane < bw) B[(i0 + lane) * kInvCols + cc] = v;
        }
        __syncthreads();
    }
    for (int idx = threadIdx.x; idx < n * kInvCols; idx += blockDim.x) {
        const int i = idx / kInvCols, cc = idx % kInvCols;
        if (c0 + cc < n) xout[(int64_t)i * n + c0 + cc] = B[idx];
    }
}

int lu_inverse32(const float* lu, int n, const int32_t* piv, float* x, cudaStream_t s) {
    const size_t smem = (size_t)n * kInvCols * sizeof(float);
    if (smem > 220 * 1024) return fail(FJ_ERR_UNSUPPORTED, "lu_inverse32: n=%d too large", n);
    FJ_TRY(allow_dynamic_smem((const void*)lu_inverse32_kernel, (size_t)smem));
    lu_inverse32_kernel<<<(n + kInvCols - 1) / kInvCols, 512, smem, s>>>(lu, n, piv, x); note_launch();
    FJ_LAUNCH_CHECK("lu_inverse32_kernel");
    return FJ_OK;
}

// ---------------------------------------------------------------------------------
// Tensor-core factorisation and inverse (mixed path, n >= kTcMinN).
//
// lu_factor32_tc: the same partial-pivoting LU, blocked twice.  One launch factors each
// outer panel of 128 columns (panel_factor; the 16-column panels above where the rows
// exceed one cluster, their U rows and updates confined to the outer panel).  The columns to
// its right receive only the row swaps until the outer panel is done; then
//   U12 = L11^-1 A12        (lu_trsm32_kernel: forward substitution, CUDA cores, in place)
//   A22 -= L21 U12          (tensor cores, K = 128)
//
// lu_inverse32_tc: X = U^-1 L^-1 P by blocked substitution on the n x n right-hand side
// P (the getrf row swaps applied to the identity), 128 rows at a time:
//   forward   Y_i = L_ii^-1 Y_i,  Y_below -= L_below,i Y_i
//   backward  X_i = U_ii^-1 Y_i,  Y_above -= U_above,i X_i
// Every product is a tensor-core GEMM; 2 n^3 flop in all.
constexpr int kTcBlk = 128;

// tri: the 2 x nblk inverted diagonal blocks (L's, then U's), then the TMA products'
// operand-split scratch, enough for the largest product (m, n <= nblk x 128, K = 128).

static size_t tc_inv_floats(int n) {
    return (size_t)2 * ((n + kTcBlk - 1) / kTcBlk) * kTcBlk * kTcBlk;
}

static size_t tc_scratch_floats(int n) {
    const int np = (n + kTcBlk - 1) / kTcBlk * kTcBlk;
    return tc_gemm_scratch_floats(np, np, kTcBlk, 3);
}

size_t tc_tri_floats(int n) {
    return tc_inv_floats(n) + tc_scratch_floats(n);
}

// The rows that an outer panel's pivots move (panel_factor), as a list of (destination,
// source) global rows in shared memory: the panel's own rows, then the pivot rows below
// them (a row named by several pivots is listed as often, each time with the same source).
// Returns the list's length; the CTA's first 2 kb threads trace one row each.
template <int KB>
struct MoveList {
    int p[KB], dst[2 * KB], src[2 * KB];
    int count[2 * KB / 32];
};

template <int KB>
__device__ __forceinline__ int list_moves(const int32_t* __restrict__ piv, int k, int kb, MoveList<KB>& m) {
    constexpr int NW = 2 * KB / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t < kb) m.p[t] = piv[k + t] - k;
    __syncthreads();
    int pos = -1, src = -1;
    unsigned moved = 0;
    if (warp < NW) {
        if (t < kb) pos = t;
        else if (t >= KB && t < KB + kb && m.p[t - KB] >= kb) pos = m.p[t - KB];
        src = swap_source(m.p, kb, pos);
        moved = __ballot_sync(0xffffffffu, pos >= 0 && src != pos);
        if (lane == 0) m.count[warp] = __popc(moved);
    }
    __syncthreads();
    int total = 0, before = 0;
    for (int w = 0; w < NW; ++w) {
        if (w < warp) before += m.count[w];
        total += m.count[w];
    }
    if (warp < NW && ((moved >> lane) & 1u)) {
        const int o = before + __popc(moved & ((1u << lane) - 1u));
        m.dst[o] = k + pos;
        m.src[o] = k + src;
    }
    __syncthreads();
    return total;
}

// An outer panel's row moves for every column outside it: a CTA takes 32 columns, loads
// every moved row's values into shared memory, then stores them to their destinations (all
// loads before any store, so the permutation's cycles need no order).
__global__ void __launch_bounds__(256) lu_swap_rows_kernel(float* __restrict__ a, int n, int k, int kb,
                                                           const int32_t* __restrict__ piv) {
    __shared__ MoveList<kTcBlk> m;
    __shared__ float tile[2 * kTcBlk][33];
    const int cnt = list_moves<kTcBlk>(piv, k, kb, m);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    const bool col = c < n && (c < k || c >= k + kb);
#pragma unroll 8
    for (int e = warp; e < cnt; e += 8)
        if (col) tile[e][lane] = a[(int64_t)m.src[e] * n + c];
    __syncthreads();
    for (int e = warp; e < cnt; e += 8)
        if (col) a[(int64_t)m.dst[e] * n + c] = tile[e][lane];
}

// U12 = L11^-1 A12 for the mixed factorisation's outer panel at column k (kb <= 128
// rows, L11 unit lower from the factored panel), in place on the columns [c0, n).  A CTA
// of 16 warps takes 16 columns: L11 and the columns' panel rows come into shared memory
// (coalesced), then warp w substitutes column w, lane l holding rows l + 32 q (q < 4) in
// registers, each x_j reaching every lane by a shuffle.  Forward substitution in FP32,
// as the CUDA-core path's lu_swap_trsm_kernel computes its U rows.
constexpr int kTrsmCols = 16;
constexpr size_t kTrsm32Smem = (size_t)(kTcBlk * (kTcBlk + 1) + kTcBlk * (kTrsmCols + 1)) * sizeof(float);

__device__ __forceinline__ float pick4f(const float (&v)[4], int q) {
    return q == 0 ? v[0] : q == 1 ? v[1] : q == 2 ? v[2] : v[3];
}

constexpr int kTrsmThreads = 32 * kTrsmCols;

__global__ void __launch_bounds__(kTrsmThreads) lu_trsm32_kernel(float* __restrict__ a, int n, int k, int kb, int c0) {
    extern __shared__ __align__(16) float smt[];
    float* ls = smt;                               // [128][129]
    float* xs = smt + kTcBlk * (kTcBlk + 1);       // [128][17]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cb = c0 + blockIdx.x * kTrsmCols;
    for (int idx = threadIdx.x; idx < kTcBlk * kTcBlk; idx += blockDim.x) {
        const int r = idx >> 7, j = idx & 127;
        ls[r * (kTcBlk + 1) + j] = (r < kb && j < r) ? a[(int64_t)(k + r) * n + k + j] : 0.0f;
    }
    for (int idx = threadIdx.x; idx < kTcBlk * kTrsmCols; idx += blockDim.x) {
        const int r = idx / kTrsmCols, cc = idx % kTrsmCols, col = cb + cc;
        xs[r * (kTrsmCols + 1) + cc] = (r < kb && col < n) ? a[(int64_t)(k + r) * n + col] : 0.0f;
    }
    __syncthreads();
    const unsigned full = 0xffffffffu;
    {
        const int cc = warp;
        float x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = xs[(lane + 32 * q) * (kTrsmCols + 1) + cc];
#pragma unroll 4
        for (int j = 0; j < kb - 1; ++j) {
            const float xj = __shfl_sync(full, pick4f(x, j >> 5), j & 31);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = lane + 32 * q;
                if (r > j) x[q] -= ls[r * (kTcBlk + 1) + j] * xj;  // rows >= kb: zero multipliers
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) xs[(lane + 32 * q) * (kTrsmCols + 1) + cc] = x[q];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < kTcBlk * kTrsmCols; idx += blockDim.x) {
        const int r = idx / kTrsmCols, cc = idx % kTrsmCols, col = cb + cc;
        if (r >= 1 && r < kb && col < n) a[(int64_t)(k + r) * n + col] = xs[r * (kTrsmCols + 1) + cc];
    }
}

// The factorisation's and the inverse's products: the TMA-fed tensor-core GEMM, its
// operand split in the scratch that follows the diagonal-block inverses.
static int tc_mul(const float* a, int lda, const float* b, int ldb, float* c, int ldc, int m, int n, int k,
                  float alpha, float beta, int passes, float* tri, int nn, int* d_err, cudaStream_t s) {
    return tc_gemm_tf32_tma(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, passes, tri + tc_inv_floats(nn),
                            tc_scratch_floats(nn), d_err, s);
}

template <int NB>
static int lu_factor32_tc_impl(float* a, int n, int32_t* piv, int* d_info, int* d_err, float* tri_l, int passes,
                               cudaStream_t s) {
    static_assert(kTcBlk % NB == 0, "inner panels tile the outer one");
    if (n <= 0) return fail(FJ_ERR_SHAPE, "lu_factor: n=%d", n);
    const size_t smem = (size_t)n * (NB + 1) * sizeof(float);
    if (smem > 220 * 1024) return fail(FJ_ERR_UNSUPPORTED, "lu_factor: n=%d too large for the shared-memory panel", n);
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_kernel<float, NB>, smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_reg_kernel<float, NB, 1>, smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_reg_kernel<float, NB, 2>, smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_trsm32_kernel, kTrsm32Smem));
    FJ_CUDA(cudaMemsetAsync(d_info, 0, sizeof(int), s));
    const int panel_rows = panel_max_rows<float>();
    for (int k = 0; k < n; k += kTcBlk) {
        const int kb = min(kTcBlk, n - k), ke = k + kb;
        if (n - k <= panel_rows) {
            FJ_TRY(panel_factor<float>(a, n, k, kb, piv, d_info, nullptr, s));
            if (n > kb) {
                lu_swap_rows_kernel<<<(unsigned)((n + 31) / 32), 256, 0, s>>>(a, n, k, kb, piv);
                note_launch();
            }
        } else {
          for (int j = k; j < ke; j += NB) {
            const int nb = min(NB, n - j);
            launch_panel<float, NB>(a, n, j, piv, d_info, nullptr, s);
            if (n > nb) {
                lu_swap_trsm_kernel<float, NB><<<(n + 255) / 256, 256, 0, s>>>(a, n, j, piv, ke, nullptr);
                note_launch();
            }
            const int rows = n - j - nb, cols = ke - j - nb;
            if (nb == NB && rows > 0 && cols > 0) {
                lu_update_kernel<float, NB><<<dim3((cols + 63) / 64, (rows + 63) / 64), 256, 0, s>>>(a, n, j, ke, nullptr);
                note_launch();
            }
          }
        }
        const int rest = n - ke;
        if (rest > 0) {  // U12 = L11^-1 A12 (CUDA cores), then A22 -= L21 U12 (tensor cores)
            float* a12 = a + (int64_t)k * n + ke;
            lu_trsm32_kernel<<<(unsigned)((rest + kTrsmCols - 1) / kTrsmCols), kTrsmThreads, kTrsm32Smem, s>>>(a, n, k,
                                                                                                          kb, ke);
            note_launch();
            FJ_TRY(tc_mul(a + (int64_t)ke * n + k, n, a12, n, a + (int64_t)ke * n + ke, n, rest, rest, kb, -1.0f, 1.0f,
                          passes, tri_l, n, d_err, s));
        }
    }
    FJ_LAUNCH_CHECK("lu_factor32_tc");
    return FJ_OK;
}

int lu_factor32_tc(float* a, int n, int32_t* piv, int* d_info, int* d_err, float* tri_l, int passes,
                   cudaStream_t s) {
    if (panel_fits<float>(n, 16)) return lu_factor32_tc_impl<16>(a, n, piv, d_info, d_err, tri_l, passes, s);
    return lu_factor32_tc_impl<8>(a, n, piv, d_info, d_err, tri_l, passes, s);
}

// Y = P I: row i holds a one in column perm[i].  Y must be zero on entry.
__global__ void __launch_bounds__(1024) perm_identity_kernel(const int32_t* __restrict__ piv, int n,
                                                             float* __restrict__ y) {
    extern __shared__ int perm_sm[];
    __shared__ PermScratch<kPermChunk> S;
    build_perm(piv, n, perm_sm, S);
    for (int i = threadIdx.x; i < n; i += blockDim.x) y[(int64_t)i * n + perm_sm[i]] = 1.0f;
}

int lu_inverse32_tc(const float* lu, int n, const int32_t* piv, float* x, float* tri, int passes, int* d_err,
                    cudaStream_t s) {
    const int nblk = (n + kTcBlk - 1) / kTcBlk;
    float* tri_l = tri;
    float* tri_u = tri + (size_t)nblk * kTcBlk * kTcBlk;
    // the diagonal blocks' inverses, L's and U's, each set in one launch (a CTA per block);
    // L's blocks are final once their panel is factored (later swaps touch lower rows only)
    FJ_TRY(tri_inverse32_blocks(lu, n, 0, nblk, false, tri_l, s));
    FJ_TRY(tri_inverse32_blocks(lu, n, 0, nblk, true, tri_u, s));
    FJ_CUDA(cudaMemsetAsync(x, 0, (size_t)n * n * sizeof(float), s));
    FJ_TRY(allow_dynamic_smem((const void*)perm_identity_kernel, (size_t)n * sizeof(int)));
    perm_identity_kernel<<<1, 1024, (size_t)n * sizeof(int), s>>>(piv, n, x);
    note_launch();
    FJ_LAUNCH_CHECK("perm_identity_kernel");
    for (int b = 0; b < nblk; ++b) {  // forward: unit lower
        const int i0 = b * kTcBlk, ib = min(kTcBlk, n - i0), below = n - i0 - ib;
        float* yi = x + (int64_t)i0 * n;
        FJ_TRY(tc_mul(tri_l + (size_t)b * kTcBlk * kTcBlk, kTcBlk, yi, n, yi, n, ib, n, ib, 1.0f, 0.0f, passes, tri,
                      n, d_err, s));
        if (below > 0)
            FJ_TRY(tc_mul(lu + (int64_t)(i0 + ib) * n + i0, n, yi, n, yi + (int64_t)ib * n, n, below, n, ib, -1.0f,
                          1.0f, passes, tri, n, d_err, s));
    }
    for (int b = nblk - 1; b >= 0; --b) {  // backward: upper
        const int i0 = b * kTcBlk, ib = min(kTcBlk, n - i0);
        float* yi = x + (int64_t)i0 * n;
        FJ_TRY(tc_mul(tri_u + (size_t)b * kTcBlk * kTcBlk, kTcBlk, yi, n, yi, n, ib, n, ib, 1.0f, 0.0f, passes, tri,
                      n, d_err, s));
        if (i0 > 0) FJ_TRY(tc_mul(lu + i0, n, yi, n, x, n, i0, n, ib, -1.0f, 1.0f, passes, tri, n, d_err, s));
    }
    return FJ_OK;
}

// ---------------------------------------------------------------------------------
// FP64 factorisation (the plain path's getrf), blocked twice.  Outer panels of kDB = 64
// columns; where a panel's rows fit one launch (n - k <= panel_max_rows<double>())
// panel_factor factors it, else 2- to 8-column panels do, with their U rows and updates
// confined to the outer panel.  Then
//   lu_swap_trsm64_kernel: the outer panel's row swaps for every column outside it, and
//                          U12 = L11^-1 A12 for the columns to its right;
//   lu_gemm64_kernel:      A22 -= L21 U12 (K = 64, FP64 FMA).
// Pivots are getrf's (first maximum of the column below the diagonal); the trailing
// matrix is updated once per 64 columns instead of once per column, so the factors
// differ from a column-by-column getrf only by rounding.
constexpr int kDB = 64;
static_assert(kDB == kPanelCols<double> && kTcBlk == kPanelCols<float>, "the outer panels are panel_factor's");

// The outer panel's row moves for 32 columns per CTA, one per lane: the panel's own kb rows
// come from the rows whose values end there (swap_source), the rows below it that move are
// listed and loaded beside them, and every load precedes every store.  Then, for the CTA's
// columns right of the panel, the kb x kb unit-lower L11 solves the panel's rows: warp w (of
// 16) takes columns 2w and 2w + 1 side by side (their chains of shuffles overlap), lane l
// rows l and l + 32.  Latency-bound: one round trip to memory, then 64 substitution steps.
constexpr int kSwapTrsm64Warps = 16;

__global__ void __launch_bounds__(32 * kSwapTrsm64Warps)
    lu_swap_trsm64_kernel(double* __restrict__ a, int n, int k, int kb, const int32_t* __restrict__ piv,
                          int do_swaps, const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;
    extern __shared__ __align__(16) unsigned char sm64[];
    double* xs = reinterpret_cast<double*>(sm64);  // [kDB][33]
    double* ls = xs + kDB * 33;                    // [kDB][kDB + 1] L11
    __shared__ int p[kDB], src[kDB], down_dst[kDB], down_src[kDB];
    const unsigned full = 0xffffffffu;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int c0 = blockIdx.x * 32, c = c0 + lane;
    const bool solve = c0 + 31 >= k + kb && kb > 1;  // a column right of the panel (uniform over the CTA)
    if (t < kb) p[t] = do_swaps ? piv[k + t] - k : t;
    if (solve) {
#pragma unroll
        for (int idx = t; idx < kDB * kDB; idx += 32 * kSwapTrsm64Warps) {
            const int r = idx / kDB, j = idx % kDB;
            ls[r * (kDB + 1) + j] = (r < kb && j < r) ? a[(int64_t)(k + r) * n + k + j] : 0.0;
        }
    }
    __syncthreads();
    if (t < kb) {
        src[t] = do_swaps ? swap_source(p, kb, t) : t;
    } else if (t >= kDB && t < kDB + kb) {
        const int r = p[t - kDB];  // a row below the panel takes the values that end there
        down_dst[t - kDB] = r >= kb ? r : -1;
        down_src[t - kDB] = r >= kb ? swap_source(p, kb, r) : 0;
    }
    __syncthreads();
    const bool col = c < n && (c < k || c >= k + kb);
    double own[kDB / kSwapTrsm64Warps], down[kDB / kSwapTrsm64Warps];
#pragma unroll
    for (int i = 0; i < kDB / kSwapTrsm64Warps; ++i) {
        const int r = warp + i * kSwapTrsm64Warps;
        own[i] = r < kb && col ? a[(int64_t)(k + src[r]) * n + c] : 0.0;
        down[i] = r < kb && col && down_dst[r] >= 0 ? a[(int64_t)(k + down_src[r]) * n + c] : 0.0;
    }
    __syncthreads();  // the CTA has read what it is about to write
#pragma unroll
    for (int i = 0; i < kDB / kSwapTrsm64Warps; ++i) {
        const int r = warp + i * kSwapTrsm64Warps;
        if (r < kb && col && down_dst[r] >= 0) a[(int64_t)(k + down_dst[r]) * n + c] = down[i];
        if (solve) xs[r * 33 + lane] = own[i];
        else if (r < kb && col) a[(int64_t)(k + r) * n + c] = own[i];
    }
    if (!solve) return;
    __syncthreads();
    double x0[2], x1[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        x0[h] = xs[lane * 33 + 2 * warp + h];
        x1[h] = xs[(lane + 32) * 33 + 2 * warp + h];
    }
    const bool right0 = c0 + 2 * warp >= k + kb, right1 = c0 + 2 * warp + 1 >= k + kb;
    if (right0 || right1) {  // (columns left of the panel only move)
        const double *l0 = ls + lane * (kDB + 1), *l1 = ls + (lane + 32) * (kDB + 1);
        double y0[2] = {x0[0], x0[1]}, y1[2] = {x1[0], x1[1]};
#pragma unroll 4
        for (int j = 0; j < min(kb - 1, 32); ++j) {
            const double m0 = l0[j], m1 = l1[j];  // rows >= kb: zero multipliers
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double xj = __shfl_sync(full, y0[h], j);
                if (lane > j) y0[h] -= m0 * xj;
                y1[h] -= m1 * xj;
            }
        }
#pragma unroll 4
        for (int j = 32; j < kb - 1; ++j) {
            const double m1 = l1[j];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double xj = __shfl_sync(full, y1[h], j - 32);
                y1[h] -= m1 * xj;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (h == 0 ? right0 : right1) {
                xs[lane * 33 + 2 * warp + h] = y0[h];
                xs[(lane + 32) * 33 + 2 * warp + h] = y1[h];
            }
    }
    __syncthreads();
#pragma unroll
    for (int idx = t; idx < kDB * 32; idx += 32 * kSwapTrsm64Warps) {
        const int r = idx >> 5, cc = idx & 31, g = c0 + cc;
        if (r < kb && g < n && (g < k || g >= k + kb)) a[(int64_t)(k + r) * n + g] = xs[r * 33 + cc];
    }
}

constexpr size_t kSwapTrsm64Smem = (size_t)(kDB * 33 + kDB * (kDB + 1)) * sizeof(double);

// A22 -= L21 U12 with K = kDB, on one 64 x 64 tile of the trailing matrix per CTA: the
// CTA's 64 rows of L21 and 64 columns of U12 come into shared memory (cp.async, zero past
// the matrix), then thread (tx, ty) updates rows ty + 16 p and columns tx + 16 q (p, q < 4)
// with the 64 products in order, as the column-by-column update would.
__global__ void __launch_bounds__(256)
    lu_gemm64_kernel(double* __restrict__ a, int n, int k, const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;
    extern __shared__ __align__(16) unsigned char smg64[];
    double* as = reinterpret_cast<double*>(smg64);  // [64][kDB]: L21 rows
    double* bs = as + 64 * kDB;                      // [kDB][64]: U12 columns
    const int k2 = k + kDB;
    const int r0 = k2 + blockIdx.y * 64, c0 = k2 + blockIdx.x * 64;
    for (int idx = threadIdx.x; idx < 64 * kDB; idx += blockDim.x) {
        const int r = idx / kDB, j = idx % kDB;
        const bool oka = r0 + r < n;
        const double* srca = a + (int64_t)(oka ? r0 + r : 0) * n + k + j;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(as + idx)),
                     "l"(srca), "r"(oka ? 8 : 0)
                     : "memory");
        const int jb = idx / 64, cb = idx % 64;
        const bool okb = c0 + cb < n;
        const double* srcb = a + (int64_t)(k + jb) * n + (okb ? c0 + cb : 0);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(bs + idx)),
                     "l"(srcb), "r"(okb ? 8 : 0)
                     : "memory");
    }
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = r0 + ty + 16 * p, cc = c0 + tx + 16 * q;
            acc[p][q] = (r < n && cc < n) ? a[(int64_t)r * n + cc] : 0.0;
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll 8
    for (int j = 0; j < kDB; ++j) {
        double ar[4], br[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) ar[p] = as[(ty + 16 * p) * kDB + j];
#pragma unroll
        for (int q = 0; q < 4; ++q) br[q] = bs[j * 64 + tx + 16 * q];
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[p][q] -= ar[p] * br[q];
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = r0 + ty + 16 * p, cc = c0 + tx + 16 * q;
            if (r < n && cc < n) a[(int64_t)r * n + cc] = acc[p][q];
        }
}

constexpr size_t kGemm64Smem = (size_t)2 * 64 * kDB * sizeof(double);

// The outer panel at column k in NB-column panels (rows beyond one cluster): swaps over
// every column, U rows and updates inside the outer panel [k, ke).
template <int NB>
static int lu_outer_panel_narrow64(double* a, int n, int k, int ke, int32_t* piv, int* d_info, const int* run_flag,
                                   cudaStream_t s) {
    const size_t smem = (size_t)n * (NB + 1) * sizeof(double);
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_kernel<double, NB>, smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_reg_kernel<double, NB, 1>, smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_panel_reg_kernel<double, NB, 2>, smem));
    for (int j = k; j < ke; j += NB) {
        const int nb = min(NB, n - j);
        launch_panel<double, NB>(a, n, j, piv, d_info, run_flag, s);
        if (n > nb) {
            lu_swap_trsm_kernel<double, NB><<<(n + 255) / 256, 256, 0, s>>>(a, n, j, piv, ke, run_flag);
            note_launch();
        }
        const int rows = n - j - nb, cols = ke - j - nb;
        if (nb == NB && rows > 0 && cols > 0) {
            lu_update_kernel<double, NB><<<dim3((cols + 63) / 64, (rows + 63) / 64), 256, 0, s>>>(a, n, j, ke, run_flag);
            note_launch();
        }
    }
    return FJ_OK;
}

int lu_factor64(double* a, int n, int32_t* piv, int* d_info, cudaStream_t s, const int* run_flag) {
    if (n <= 0) return fail(FJ_ERR_SHAPE, "lu_factor: n=%d", n);
    int nb_narrow = 0;
    for (int nb : {8, 4, 2})
        if (nb_narrow == 0 && panel_fits<double>(n, nb)) nb_narrow = nb;
    const int panel_rows = panel_max_rows<double>();
    if (nb_narrow == 0 && n > panel_rows)
        return fail(FJ_ERR_UNSUPPORTED, "lu_factor: n=%d too large for the shared-memory panel", n);
    FJ_TRY(allow_dynamic_smem((const void*)lu_swap_trsm64_kernel, kSwapTrsm64Smem));
    FJ_TRY(allow_dynamic_smem((const void*)lu_gemm64_kernel, kGemm64Smem));
    FJ_CUDA(cudaMemsetAsync(d_info, 0, sizeof(int), s));
    for (int k = 0; k < n; k += kDB) {
        const int kb = min(kDB, n - k), ke = k + kb;
        const bool whole = n - k <= panel_rows;
        if (whole) {
            FJ_TRY(panel_factor<double>(a, n, k, kb, piv, d_info, run_flag, s));
        } else if (nb_narrow == 8) {
            FJ_TRY(lu_outer_panel_narrow64<8>(a, n, k, ke, piv, d_info, run_flag, s));
        } else if (nb_narrow == 4) {
            FJ_TRY(lu_outer_panel_narrow64<4>(a, n, k, ke, piv, d_info, run_flag, s));
        } else {
            FJ_TRY(lu_outer_panel_narrow64<2>(a, n, k, ke, piv, d_info, run_flag, s));
        }
        if (n > kb) {
            lu_swap_trsm64_kernel<<<(unsigned)((n + 31) / 32), 32 * kSwapTrsm64Warps, kSwapTrsm64Smem, s>>>(
                a, n, k, kb, piv, whole ? 1 : 0, run_flag);
            note_launch();
        }
        const int rest = n - ke;
        if (rest > 0) {  // kb == kDB here
            lu_gemm64_kernel<<<dim3((unsigned)((rest + 63) / 64), (unsigned)((rest + 63) / 64)), 256, kGemm64Smem, s>>>(
                a, n, k, run_flag);
            note_launch();
        }
    }
    FJ_LAUNCH_CHECK("lu_factor64");
    return FJ_OK;
}

// Factor path of the mixed solve.  FJ_MIXED_FACTOR selects it: "cuda" (FP32 CUDA cores),
// "tf32" (tensor cores, one TF32 pass) or the default "tf32x3" (three-pass split); the
// tensor-core paths apply from n >= kTcMinN.
constexpr int kTcMinN = 256;

int factor_inverse32(const double* a64, int n, float* a32, int32_t* piv, int* flags, float* x32, float* tri,
                     cudaStream_t s) {
    int passes = 3;
    if (const char* e = getenv("FJ_MIXED_FACTOR")) {
        if (!strcmp(e, "cuda")) passes = 0;
        else if (!strcmp(e, "tf32")) passes = 1;
        else if (strcmp(e, "tf32x3") != 0) return fail(FJ_ERR_SHAPE, "FJ_MIXED_FACTOR=%s (cuda, tf32 or tf32x3)", e);
    }
    FJ_TRY(convert64to32(a64, a32, (int64_t)n * n, s));
    if (passes == 0 || n < kTcMinN) {
        FJ_TRY(lu_factor32(a32, n, piv, flags, s));
        return lu_inverse32(a32, n, piv, x32, s);
    }
    FJ_CUDA(cudaMemsetAsync(flags + 3, 0, sizeof(int), s));
    FJ_TRY(lu_factor32_tc(a32, n, piv, flags, flags + 3, tri, passes, s));
    return lu_inverse32_tc(a32, n, piv, x32, tri, passes, flags + 3, s);
}

__global__ void convert64to32_kernel(const double* __restrict__ a, float* __restrict__ b, int64_t count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) b[i] = (float)a[i];
}

int convert64to32(const double* a, float* b, int64_t count, cudaStream_t s) {
    if (count == 0) return FJ_OK;
    convert64to32_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(a, b, count); note_launch();
    FJ_LAUNCH_CHECK("convert64to32_kernel");
    return FJ_OK;
}

// ---------------------------------------------------------------------------------
// Refinement GEMVs: one warp per row, FP64 accumulation.
//   mode 0: y = X v        mode 1: y += X v        (X FP32)
//   residual: r = b - A x  (A FP64)
// Row dot products of the refinement (HBM-bound: one pass over the matrix row).  A warp
// takes a row; where the row and the vector are 16-byte aligned and n a multiple of 4 (2
// for FP64 rows) each lane loads whole 16-byte vectors, four in flight, into four
// independent FP64 partial sums; else element by element.  The warp's sum comes back in
// every lane.
__device__ __forceinline__ double warp_sum(double a) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    return a;
}

__device__ __forceinline__ double row_dot32(const float* __restrict__ xr, const double* __restrict__ v, int n,
                                            int lane) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if ((n & 3) == 0 && (((uintptr_t)xr | (uintptr_t)v) & 15) == 0) {
        const float4* x4 = reinterpret_cast<const float4*>(xr);
        const double2* v2 = reinterpret_cast<const double2*>(v);
        const int n4 = n >> 2;
#pragma unroll 4
        for (int j = lane; j < n4; j += 32) {
            const float4 x = __ldg(x4 + j);
            const double2 p = v2[2 * j], q = v2[2 * j + 1];
            a0 = fma((double)x.x, p.x, a0);
            a1 = fma((double)x.y, p.y, a1);
            a2 = fma((double)x.z, q.x, a2);
            a3 = fma((double)x.w, q.y, a3);
        }
    } else {
        for (int j = lane; j < n; j += 32) a0 = fma((double)xr[j], v[j], a0);
    }
    return warp_sum((a0 + a1) + (a2 + a3));
}

__device__ __forceinline__ double row_dot64(const double* __restrict__ ar, const double* __restrict__ x, int n,
                                            int lane) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if ((n & 1) == 0 && (((uintptr_t)ar | (uintptr_t)x) & 15) == 0) {
        const double2* r2 = reinterpret_cast<const double2*>(ar);
        const double2* x2 = reinterpret_cast<const double2*>(x);
        const int n2 = n >> 1;
        int j = lane;
#pragma unroll 2
        for (; j + 32 < n2; j += 64) {
            const double2 p = __ldg(r2 + j), q = __ldg(r2 + j + 32);
            const double2 u = x2[j], w = x2[j + 32];
            a0 = fma(p.x, u.x, a0);
            a1 = fma(p.y, u.y, a1);
            a2 = fma(q.x, w.x, a2);
            a3 = fma(q.y, w.y, a3);
        }
        if (j < n2) {
            const double2 p = __ldg(r2 + j), u = x2[j];
            a0 = fma(p.x, u.x, a0);
            a1 = fma(p.y, u.y, a1);
        }
    } else {
        for (int j = lane; j < n; j += 32) a0 = fma(ar[j], x[j], a0);
    }
    return warp_sum((a0 + a1) + (a2 + a3));
}

__global__ void gemv32_kernel(const float* __restrict__ X, const double* __restrict__ v, int n,
                              double* __restrict__ y, int accumulate) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    const double acc = row_dot32(X + (int64_t)row * n, v, n, lane);
    if (lane == 0) y[row] = accumulate ? y[row] + acc : acc;
}

__global__ void residual64_kernel(const double* __restrict__ A, const double* __restrict__ x,
                                  const double* __restrict__ b, int n, double* __restrict__ r) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    const double acc = row_dot64(A + (int64_t)row * n, x, n, lane);
    if (lane == 0) r[row] = b[row] - acc;
}

__global__ void rel_resid_kernel(const double* __restrict__ r, const double* __restrict__ b, int n,
                                 double* __restrict__ out) {
    relative_residual(r, b, n, out);
}

int refine_solve(const double* a, const float* xinv, int n, const double* b, double* x, double* r_buf,
                 double* d_resid, int n_iter, cudaStream_t s) {
    const int wpb = 8;
    const unsigned grid = (unsigned)((n + wpb - 1) / wpb);
    gemv32_kernel<<<grid, wpb * 32, 0, s>>>(xinv, b, n, x, 0); note_launch();
    for (int it = 0; it < n_iter; ++it) {
        residual64_kernel<<<grid, wpb * 32, 0, s>>>(a, x, b, n, r_buf); note_launch();
        gemv32_kernel<<<grid, wpb * 32, 0, s>>>(xinv, r_buf, n, x, 1); note_launch();
    }
    residual64_kernel<<<grid, wpb * 32, 0, s>>>(a, x, b, n, r_buf); note_launch();
    rel_resid_kernel<<<1, 1024, 0, s>>>(r_buf, b, n, d_resid); note_launch();
    FJ_LAUNCH_CHECK("refine_solve");
    return FJ_OK;
}

// ---------------------------------------------------------------------------------
// Batched refinement sweeps (grid.y = system).
__global__ void gemv32_jobs_kernel(const RefineJob* __restrict__ jobs, int from_residual, int accumulate) {
    const RefineJob& J = jobs[blockIdx.y];
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= J.n) return;
    const double acc = row_dot32(J.xinv + (int64_t)row * J.n, from_residual ? J.r : J.b, J.n, lane);
    if (lane == 0) J.x[row] = accumulate ? J.x[row] + acc : acc;
}

__global__ void residual64_jobs_kernel(const RefineJob* __restrict__ jobs) {
    const RefineJob& J = jobs[blockIdx.y];
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= J.n) return;
    const double acc = row_dot64(J.a + (int64_t)row * J.n, J.x, J.n, lane);
    if (lane == 0) J.r[row] = J.b[row] - acc;
}

int refine_jobs(const RefineJob* d_jobs, int n_jobs, int max_n, int n_iter, cudaStream_t s) {
    if (n_jobs == 0 || max_n == 0) return FJ_OK;
    const int wpb = 8;
    dim3 g((unsigned)((max_n + wpb - 1) / wpb), (unsigned)n_jobs);
    gemv32_jobs_kernel<<<g, wpb * 32, 0, s>>>(d_jobs, 0, 0); note_launch();
    for (int it = 0; it < n_iter; ++it) {
        residual64_jobs_kernel<<<g, wpb * 32, 0, s>>>(d_jobs); note_launch();
        gemv32_jobs_kernel<<<g, wpb * 32, 0, s>>>(d_jobs, 1, 1); note_launch();
    }
    residual64_jobs_kernel<<<g, wpb * 32, 0, s>>>(d_jobs); note_launch();
    FJ_LAUNCH_CHECK("refine_jobs");
    return FJ_OK;
}

}  // namespace fj
