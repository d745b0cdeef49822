// fj_trsv.cuh -- getrf's row order, and the substitutions of getrs for one right-hand side
// (fj_trsv.cu).
#pragma once

#include "fj_common.cuh"

namespace fj {

// The pivots' row order in shared memory: perm[i] = the row that the swaps (i, piv[i]), applied
// in order, bring to row i.  Every thread of the CTA calls it.  Blocks of 64 swaps are
// composed side by side, a thread tracing one row back through its block, and then applied
// one after the other: one thread's walk through all swaps took 11 us for 256 and 80 us for
// 2048.  kChunk swaps at a time: kPermChunk, or fewer where the scratch has to make room for perm.
// perm may lie in global memory.
constexpr int kPermChunk = 2048, kPermChunkSmall = 512;
template <int kChunk>
struct PermScratch {
    int p[kChunk], src[2 * kChunk];
};

// The orders whose perm fits in shared memory beside its scratch.
template <int kChunk>
constexpr int kPermRows = (232448 - (int)sizeof(PermScratch<kChunk>)) / (int)sizeof(int);

template <int kChunk>
__device__ __forceinline__ void build_perm(const int32_t* __restrict__ piv, int n, int* perm, PermScratch<kChunk>& S) {
    const int t = threadIdx.x, nt = blockDim.x;
    for (int i = t; i < n; i += nt) perm[i] = i;
    for (int c0 = 0; c0 < n; c0 += kChunk) {
        const int cnt = min(kChunk, n - c0);
        __syncthreads();
        for (int i = t; i < cnt; i += nt) S.p[i] = min(max(piv[c0 + i], 0), n - 1);
        __syncthreads();
        const int blocks = (cnt + 63) / 64;
        for (int e = t; e < blocks * 128; e += nt) {  // a block's own rows, then its pivot rows
            const int b = e >> 7, i = b * 64 + (e & 63), len = min(64, cnt - b * 64);
            int x = -1;
            if (i < cnt) {
                x = e & 64 ? S.p[i] : c0 + i;
#pragma unroll 8
                for (int q = len - 1; q >= 0; --q) {
                    const int r = c0 + b * 64 + q, p = S.p[b * 64 + q];
                    x = x == r ? p : (x == p ? r : x);
                }
            }
            S.src[e] = x;
        }
        __syncthreads();
        if (t < 128) {
            for (int b = 0; b < blocks; ++b) {
                const int i = b * 64 + (t & 63), src = S.src[b * 128 + t];
                const int dst = i >= cnt ? -1 : t & 64 ? S.p[i] : c0 + i;
                const int v = src >= 0 ? perm[src] : 0;
                asm volatile("bar.sync 7, 128;" ::: "memory");
                if (dst >= 0) perm[dst] = v;  // (a row named twice gets the same value)
                asm volatile("bar.sync 7, 128;" ::: "memory");
            }
        }
    }
    __syncthreads();
}

// getrs from the factors of fj_lu_factor, single right-hand side, in place on b; work: n
// doubles.  transposed: A^T x = b.
int lu_substitute64(const double* lu, int n, const int32_t* piv, double* b, double* work, bool transposed,
                    cudaStream_t s);

}  // namespace fj
