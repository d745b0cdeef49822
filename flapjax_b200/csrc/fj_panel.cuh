// fj_panel.cuh -- the LU factorisations' outer panels (fj_panel.cu), and their row moves.
#pragma once

#include "fj_common.cuh"

namespace fj {

// Columns of an outer panel: 512 bytes of a row.
template <typename T>
constexpr int kPanelCols = 512 / (int)sizeof(T);

// Rows panel_factor takes on this device (0 where its cluster does not run).
template <typename T>
int panel_max_rows();

// Factors the columns [k, k + kb) (kb <= kPanelCols<T>) of the row-major n x n matrix, rows
// k .. n - 1, with getrf's pivots: L and U in place, 0-based pivot rows in piv[k ..], *info
// as lu_factor64's (or n + 1 where a bounded wait expired).  The swaps are not applied to
// the other columns.  run_flag (may be null): nothing happens when *run_flag == 0.
template <typename T>
int panel_factor(T* a, int n, int k, int kb, int32_t* piv, int* info, const int* run_flag, cudaStream_t s);

// The row whose values end at row x after the transpositions (t, p[t]), t = 0 .. cnt - 1, in
// order: x traced back through them, last first.  Every thread reads the same p[t] (a
// broadcast, and no read waits on the one before).
__device__ __forceinline__ int swap_source(const int* p, int cnt, int x) {
#pragma unroll 8
    for (int t = cnt - 1; t >= 0; --t) {
        const int q = p[t];
        x = x == t ? q : (x == q ? t : x);
    }
    return x;
}

}  // namespace fj
