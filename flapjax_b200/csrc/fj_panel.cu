// fj_panel.cu -- one outer panel of a partially pivoted LU (getrf's pivots and per-element
// operations) in one launch: 64 FP64 or 128 FP32 columns.
//
// A panel is a chain of columns, each a search over its rows, an exchange of the pivot row
// and a rank-1 update: what bounds it is the latency of one column, not arithmetic.  (Lanes
// that own columns need a shuffle per row for the search and another for the multiplier:
// 400 instructions per warp and column.)
//   * The panel lies in shared memory, column by column; a quarter of its columns (the
//     window) is in registers while they are eliminated, a lane of the column warps owning
//     one or two rows of it.  All eight warps load the panel, apply a finished window to the
//     panel's other columns as a product of tiles, and write the panel back.
//   * A column: every lane shows its magnitude's leading word; after one barrier every
//     column warp finds the maximum of all rows by itself (redux.sync), and the lane that
//     holds it copies its window to shared memory (only that lane: a store of 16 bytes by one
//     lane takes the load/store unit 11 cycles, and candidates from every warp took 350); after
//     a second barrier the window comes back as 16-byte broadcasts for at most 15 (FP64) or
//     31 (FP32) multiply-adds a row.  Every lane has its element's reciprocal ready meanwhile.
//   * Rows never move: a lane keeps its rows' current positions, and a swap exchanges two
//     positions.  Rows reach their places when the panel is written back.
//   * The column loop is not unrolled (an unrolled one would be fetched once and run once),
//     and still names every register at compile time: the update of window column c writes
//     the register of column c - 1, so the current column is always register 0.
//   * Up to 384 rows one CTA factors the panel.  More rows take a cluster of 128-row CTAs
//     (up to 16): each CTA's best window goes to every CTA by st.async, whose arrival an
//     mbarrier counts, so that no cluster barrier and no fence stand in the chain.  A CTA
//     sends column j + 2 only after it has every CTA's column j + 1, which each sends after
//     its last read of column j.  The exchange adds about 450 cycles to a column's 600.
// Measured, the FP64 LU of order 128, 256, 768 and 2048: 88, 209, 797 and 2547 us, against 187,
// 410, 1480 and 5070 us for lanes that own columns and a cluster barrier per column.  Rows per
// lane and warps: 4 x 1, 2 x 2 and 1 x 8 were slower for one CTA, 256-row CTAs of a cluster up
// to 12 %.
#include <climits>
#include <map>
#include <mutex>

#include <cooperative_groups.h>

#include "fj_panel.cuh"

namespace fj {
namespace {

namespace cg = cooperative_groups;

constexpr int kMaxCtas = 16;
constexpr int kThreads = 256, kWarps = kThreads / 32;

// Search keys (hi, lo), ordered as the magnitudes: hi is the leading word of the magnitude's
// bits + 2; 1 for NaN, which getrf never prefers; 0 for a row that is no candidate.
struct Key {
    uint32_t hi, lo;
};

// Whether key a at position pa goes before b at pb: the larger, the lower position of equals
// (getrf's first maximum).
__device__ __forceinline__ bool before(Key a, int pa, Key b, int pb) {
    const unsigned long long ka = ((unsigned long long)a.hi << 32) | a.lo, kb = ((unsigned long long)b.hi << 32) | b.lo;
    return ka > kb || (ka == kb && pa < pb);
}

template <typename T>
struct Elem;
template <>
struct Elem<double> {
    using Vec = double2;
    static constexpr uint32_t kInf = 0x7ff00000u;  // leading word of infinity
    __device__ static uint32_t lead(double x) { return (uint32_t)__double2hiint(x); }
    __device__ static Key key(double x) {
        const uint32_t hi = lead(x) & 0x7fffffffu, lo = (uint32_t)__double2loint(x);
        if (hi > kInf || (hi == kInf && lo != 0u)) return {1u, 0u};
        return {hi + 2u, lo};
    }
    // getrf scales by the reciprocal of a pivot that is normal (by hi, of its key)
    __device__ static bool normal(uint32_t hi) { return hi - 2u >= 0x00100000u; }
};
template <>
struct Elem<float> {
    using Vec = float4;
    static constexpr uint32_t kInf = 0x7f800000u;
    __device__ static uint32_t lead(float x) { return __float_as_uint(x); }
    __device__ static Key key(float x) {
        const uint32_t b = lead(x) & 0x7fffffffu;
        return {b > kInf ? 1u : b + 2u, 0u};
    }
    __device__ static bool normal(uint32_t hi) { return hi - 2u >= 0x00800000u; }
};

// Columns of the window, and a candidate: its window, and what goes with it.
template <typename T>
constexpr int kWin = kPanelCols<T> / 4;

template <typename T>
struct __align__(16) Cand {
    T row[kWin<T>];
    uint32_t hi, lo;  // key; hi = 0: no candidate
    int pos, idx;     // the row's position, and its place in its CTA's tile
    T rinv;           // 1 / row[0]
};
static_assert(sizeof(Cand<double>) == 160 && sizeof(Cand<float>) == 160, "10 16-byte words");

// The lane whose key goes before the others'.
__device__ __forceinline__ int best_lane(Key key, int pos, int lane) {
    constexpr unsigned full = 0xffffffffu;
    const uint32_t m = __reduce_max_sync(full, key.hi);
    unsigned e = __ballot_sync(full, key.hi == m);
    if (__popc(e) > 1) {  // (the same for every lane)
        const bool in = key.hi == m;
        const uint32_t ml = __reduce_max_sync(full, in ? key.lo : 0u);
        const bool tie = in && key.lo == ml;
        const int mp = __reduce_min_sync(full, tie ? pos : INT_MAX);
        e = __ballot_sync(full, tie && pos == mp);
    }
    return __ffs(e) - 1;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void send16(uint32_t dst, uint32_t bar, uint4 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void expect_bytes(uint32_t bar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ uint32_t in_cta(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

constexpr long long kWaitCycles = FJ_WAIT_CYCLES;

__device__ __forceinline__ bool try_phase(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Waits for the phase, about a second at most (far beyond any column); false on expiry.  From then on
// the CTA waits for nothing and expects nothing, works on whatever its slots hold (places and
// positions in range, since the slots begin with zeros), and writes none of its rows back.
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity) {
    if (kWaitCycles < 0) return false;
    if (try_phase(bar, parity)) return true;
    const long long t0 = clock64();
    while (!try_phase(bar, parity))
        if (clock64() - t0 > kWaitCycles) return false;
    return true;
}

// CW: column warps, RPL: rows per lane of them; 32 RPL CW rows per CTA.
template <typename T, int CW, int RPL, bool kCluster>
struct Shared {
    __align__(16) uint32_t lead[2][CW * RPL * 32];  // every row's magnitude, leading word
    uint4 key[CW];                             // ties: the column warps' best keys: hi, lo, position
    Cand<T> chosen[kWin<T>];                   // the window's pivot rows' windows
    Cand<T> mine[kCluster ? 2 : 1];            // this CTA's best row of a column
    Cand<T> slot[2][kCluster ? kMaxCtas : 1];  // every CTA's
    __align__(16) T u[kWin<T>][kPanelCols<T>]; // the window's pivot rows
    __align__(16) T zeros[kWin<T>];
    T spare[32];
    uint64_t bar[2], ubar;
    int piv[kPanelCols<T>], pos[CW * RPL * 32];
    int cta[kWin<T>];    // whose row each column of the window chose
    int owner[kWin<T>];  // its place in the tile where it is this CTA's, else -1
    int info, dead;
};

template <int RPL>
struct Rows {
    int pos[RPL];       // current positions
    uint32_t mask[RPL]; // of a leading word's magnitude: 0 for a row that is no candidate
};

template <int CW>
__device__ __forceinline__ void column_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(32 * CW) : "memory");
}

// Whether this thread holds the CTA's best row, and which of its rows that is (the column
// warps, together).  Every warp reads all rows' leading words: where one alone is the
// largest, it decides; ties, infinities and NaN are searched in full.
template <typename T, int CW, int RPL, bool kCluster>
__device__ __forceinline__ bool search(const T (&x)[RPL], const Rows<RPL>& row, Shared<T, CW, RPL, kCluster>& S,
                                       int par, int warp, int lane, int& num) {
    constexpr unsigned full = 0xffffffffu;
    constexpr int NQ = CW * RPL / 4;  // 16-byte words of leading words per lane
    uint32_t hi[RPL];
#pragma unroll
    for (int e = 0; e < RPL; ++e) {
        hi[e] = Elem<T>::lead(x[e]) & row.mask[e];
        S.lead[par][(warp * RPL + e) * 32 + lane] = hi[e];
    }
    column_barrier<CW>();
    uint4 w[NQ];
    uint32_t m = 0u;
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        w[i] = reinterpret_cast<const uint4*>(S.lead[par])[32 * i + lane];
        m = max(m, max(max(w[i].x, w[i].y), max(w[i].z, w[i].w)));
    }
    m = __reduce_max_sync(full, m);
    int c = 0;
#pragma unroll
    for (int i = 0; i < NQ; ++i) c += (w[i].x == m) + (w[i].y == m) + (w[i].z == m) + (w[i].w == m);
    const unsigned any = __ballot_sync(full, c != 0), more = __ballot_sync(full, c > 1);
    if ((any & (any - 1u)) == 0u && more == 0u && m < Elem<T>::kInf && m != 0u) {  // (the same for every thread)
        bool mine = false;
        num = 0;
#pragma unroll
        for (int e = 0; e < RPL; ++e)
            if (hi[e] == m) {
                mine = true;
                num = e;
            }
        return mine;
    }
    Key k = {0u, 0u};
    int p = INT_MAX;
    num = 0;
#pragma unroll
    for (int e = 0; e < RPL; ++e) {
        const Key ke = row.mask[e] ? Elem<T>::key(x[e]) : Key{0u, 0u};
        const int pe = row.mask[e] ? row.pos[e] : INT_MAX;
        if (e == 0 || before(ke, pe, k, p)) {
            k = ke;
            p = pe;
            num = e;
        }
    }
    const int b = best_lane(k, p, lane);
    if (lane == b) S.key[warp] = make_uint4(k.hi, k.lo, (uint32_t)p, 0u);
    column_barrier<CW>();
    uint4 best = S.key[0];
    int w0 = 0;
    for (int i = 1; i < CW; ++i) {
        const uint4 h = S.key[i];
        if (before({h.x, h.y}, (int)h.z, {best.x, best.y}, (int)best.z)) {
            best = h;
            w0 = i;
        }
    }
    column_barrier<CW>();  // S.key is free again
    return warp == w0 && lane == b;
}

template <typename T, int W>
__device__ __forceinline__ void store_window(Cand<T>& c, const T (&v)[kWin<T>], Key key, int pos, int idx, T rinv) {
    using Vec = typename Elem<T>::Vec;
    Vec* r = reinterpret_cast<Vec*>(c.row);
#pragma unroll
    for (int i = 0; i < W * (int)sizeof(T) / 16; ++i) r[i] = reinterpret_cast<const Vec*>(v)[i];
    *reinterpret_cast<uint4*>(&c.hi) = make_uint4(key.hi, key.lo, (uint32_t)pos, (uint32_t)idx);
    c.rinv = rinv;
}

// Columns [j0, j1) of the window that begins at s0, W of whose columns are left at most
// (the column warps).
template <int W, typename T, int CW, int RPL, bool kCluster>
__device__ __forceinline__ void columns(T (&v)[RPL][kWin<T>], Rows<RPL>& row, T* __restrict__ tile,
                                        Shared<T, CW, RPL, kCluster>& S, int s0, int j0, int j1, int q, int nc) {
    using E = Elem<T>;
    using Vec = typename E::Vec;
    constexpr int NV = 16 / (int)sizeof(T), LD = CW * RPL * 32 + 1, kWords = (int)sizeof(Cand<T>) / 16;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll 1
    for (int j = j0; j < j1; ++j) {
        const int par = j & 1;
        const bool dead = kCluster && *(volatile int*)&S.dead;
        T x[RPL];
#pragma unroll
        for (int e = 0; e < RPL; ++e) x[e] = v[e][0];
        T rinv[RPL];
#pragma unroll
        for (int e = 0; e < RPL; ++e) rinv[e] = T(1) / x[e];
        int num;
        const bool best = search<T, CW, RPL, kCluster>(x, row, S, par, warp, lane, num);
        Cand<T>& mine = kCluster ? S.mine[par] : S.chosen[j - s0];
        if (best) {
            const int idx = (warp * RPL + num) * 32 + lane;
#pragma unroll
            for (int e = 0; e < RPL; ++e)
                if (num == e)
                    store_window<T, W>(mine, v[e], row.mask[e] ? E::key(x[e]) : Key{0u, 0u}, row.pos[e], idx, rinv[e]);
        }
        if (kCluster && __any_sync(0xffffffffu, best)) {
            // lanes 0-9 send to CTAs 0, 3, 6; 10-19 to 1, 4, 7; 20-29 to 2, 5
            const int part = lane / kWords, word = lane - part * kWords;
            __syncwarp();
            if (part < 3) {
                const uint4 w = reinterpret_cast<const uint4*>(&mine)[word];
                const uint32_t bar = smem_addr(&S.bar[par]);
                const uint32_t dst = smem_addr(&S.slot[par][q]) + 16 * word;
                for (int t = part; t < nc; t += 3) send16(in_cta(dst, t), in_cta(bar, t), w);
            }
        }
        const Cand<T>* p = &mine;
        if (kCluster) {
            if (tid == 0 && !dead) expect_bytes(smem_addr(&S.bar[par]), nc * (int)sizeof(Cand<T>));
            if (!dead && !wait_phase(smem_addr(&S.bar[par]), (j >> 1) & 1)) S.dead = 1;
            const uint4 h = *reinterpret_cast<const uint4*>(&S.slot[par][lane & (kMaxCtas - 1)].hi);
            const int o = best_lane({lane < nc ? h.x : 0u, h.y}, lane < nc ? (int)h.z : INT_MAX, lane) & (kMaxCtas - 1);
            p = &S.slot[par][o];
            if (warp == CW - 1) {  // kept for the end of the window
                if (lane < kWords)
                    reinterpret_cast<uint4*>(&S.chosen[j - s0])[lane] = reinterpret_cast<const uint4*>(p)[lane];
                if (lane == 0) S.cta[j - s0] = o;
            }
        } else {
            column_barrier<CW>();
        }
        const uint4 h = *reinterpret_cast<const uint4*>(&p->hi);
        const T ri = p->rinv;
        const int ppos = (int)h.z;
        const T* r = p->row;
        T l[RPL], lm[RPL];
#pragma unroll
        for (int i = 0; i < RPL; ++i) lm[i] = l[i] = x[i] * ri;
        if (!E::normal(h.x)) {  // getrf divides by a subnormal pivot; a zero pivot updates nothing
            const T pv = p->row[0];
            const bool zero = pv == T(0);
            if (zero) r = S.zeros;
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                l[i] = zero ? x[i] : x[i] / pv;
                lm[i] = zero ? T(0) : l[i];
            }
        }
#pragma unroll
        for (int i = 0; i < W / NV; ++i) {
            const Vec u = reinterpret_cast<const Vec*>(r)[i];
            const T* t = reinterpret_cast<const T*>(&u);
#pragma unroll
            for (int g = 0; g < NV; ++g)
                if (i * NV + g > 0) {
#pragma unroll
                    for (int f = 0; f < RPL; ++f) v[f][i * NV + g - 1] = fma(-lm[f], t[g], v[f][i * NV + g]);
                }
        }
#pragma unroll
        for (int f = 0; f < RPL; ++f) {
            const bool is = row.pos[f] == ppos, active = row.mask[f] != 0u;
            const int at = (warp * RPL + f) * 32 + lane;
            *(active && !is ? tile + j * LD + at : S.spare + lane) = l[f];  // (no branch)
            row.pos[f] = !active ? row.pos[f] : is ? j : row.pos[f] == j ? ppos : row.pos[f];
            row.mask[f] = is ? 0u : row.mask[f];
        }
    }
}

// The NC columns right of the full window at s0: U = L11^-1 (its pivot rows) and, for the
// rows still candidates, the columns minus L U.  A warp takes NC / 8 neighbouring columns,
// a lane every 32nd row.
template <int NC, typename T, int CW, int RPL, bool kCluster>
__device__ __forceinline__ void update_right(T* __restrict__ tile, Shared<T, CW, RPL, kCluster>& S, int s0) {
    using Vec = typename Elem<T>::Vec;
    constexpr int KW = kWin<T>, NV = 16 / (int)sizeof(T), LD = CW * RPL * 32 + 1;
    constexpr int C = NC / kWarps, R = CW * RPL;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < NC) {
        const int c = s0 + KW + tid;
        T u[KW];
#pragma unroll
        for (int t = 0; t < KW; ++t) u[t] = S.u[t][c];
#pragma unroll
        for (int i = 0; i < KW; i += NV) {
#pragma unroll
            for (int t = i + 1; t < KW; ++t) {
                const Vec lv = *reinterpret_cast<const Vec*>(&S.u[t][s0 + i]);
                const T* l = reinterpret_cast<const T*>(&lv);
#pragma unroll
                for (int g = 0; g < NV; ++g)
                    if (i + g < t) u[t] = fma(-l[g], u[i + g], u[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < KW; ++t) S.u[t][c] = u[t];
    }
    __syncthreads();
    if (warp >= kWarps / 2) {  // the pivot rows of this CTA
        for (int t = warp - kWarps / 2; t < KW; t += kWarps / 2) {
            const int o = S.owner[t];
            if (o < 0) continue;
            for (int c = lane; c < NC; c += 32) tile[(s0 + KW + c) * LD + o] = S.u[t][s0 + KW + c];
        }
    }
    const int c0 = s0 + KW + warp * C;
    T acc[R][C];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int c = 0; c < C; ++c) acc[i][c] = tile[(c0 + c) * LD + lane + 32 * i];
#pragma unroll 2
    for (int t = 0; t < KW; ++t) {
        T l[R], u[C];
#pragma unroll
        for (int i = 0; i < R; ++i) l[i] = tile[(s0 + t) * LD + lane + 32 * i];
#pragma unroll
        for (int c = 0; c < C / NV; ++c)
            *reinterpret_cast<Vec*>(&u[c * NV]) = *reinterpret_cast<const Vec*>(&S.u[t][c0 + c * NV]);
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int c = 0; c < C; ++c) acc[i][c] = fma(-l[i], u[c], acc[i][c]);
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (S.pos[lane + 32 * i] >= 0) {  // still a candidate (see panel_kernel)
#pragma unroll
            for (int c = 0; c < C; ++c) tile[(c0 + c) * LD + lane + 32 * i] = acc[i][c];
        }
    __syncthreads();
}

template <typename T, int CW, int RPL, bool kCluster>
__global__ void __launch_bounds__(kThreads, 1)
    panel_kernel(T* __restrict__ a, int n, int k, int kb, int32_t* __restrict__ piv, int* __restrict__ info,
                 const int* __restrict__ run_flag) {
    if (run_flag != nullptr && *run_flag == 0) return;  // the same for every CTA of the cluster
    constexpr int KB = kPanelCols<T>, KW = kWin<T>, NR = CW * RPL * 32, LD = NR + 1, NV = 16 / (int)sizeof(T);
    extern __shared__ __align__(16) unsigned char panel_smem[];
    T* tile = reinterpret_cast<T*>(panel_smem);  // [KB][LD]: this CTA's rows, column by column
    __shared__ Shared<T, CW, RPL, kCluster> S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int q = 0, nc = 1;
    if (kCluster) {
        cg::cluster_group cl = cg::this_cluster();
        q = (int)cl.block_rank();
        nc = (int)cl.num_blocks();
    }
    const int rows = n - k, r0 = q * NR;
#pragma unroll 8
    for (int r = warp; r < NR; r += kWarps) {
        const T* src = a + (int64_t)(k + min(r0 + r, rows - 1)) * n + k;
#pragma unroll
        for (int c = lane; c < KB; c += 32) tile[c * LD + r] = (r0 + r < rows && c < kb) ? src[c] : T(0);
    }
    if (tid < KW) S.zeros[tid] = T(0);
    if (kCluster && tid < 2 * kMaxCtas)
        *reinterpret_cast<uint4*>(&S.slot[tid / kMaxCtas][tid % kMaxCtas].hi) = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
        S.info = INT_MAX;
        S.dead = 0;
        if (kCluster) {
            for (uint64_t* b : {&S.bar[0], &S.bar[1], &S.ubar})
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    if (kCluster) cg::this_cluster().sync();  // every CTA runs, its barriers ready
    else __syncthreads();
    const int base = warp * RPL * 32 + lane;  // a column warp's rows: base + 32 f
    Rows<RPL> row;
#pragma unroll
    for (int f = 0; f < RPL; ++f) {
        const bool has = warp < CW && r0 + base + 32 * f < rows;
        row.mask[f] = has ? 0x7fffffffu : 0u;
        row.pos[f] = has ? r0 + base + 32 * f : -1;
    }
#pragma unroll 1
    for (int s0 = 0; s0 < kb; s0 += KW) {
        const int end = min(kb, s0 + KW);
        const bool more = end < kb;
        if (kCluster && more && tid == kThreads - 1 && !S.dead) expect_bytes(smem_addr(&S.ubar), KW * KB * (int)sizeof(T));
        if (warp < CW) {
            __align__(16) T v[RPL][KW];
#pragma unroll
            for (int f = 0; f < RPL; ++f)
#pragma unroll
                for (int c = 0; c < KW; ++c) v[f][c] = tile[(s0 + c) * LD + base + 32 * f];
            columns<KW>(v, row, tile, S, s0, s0, min(end, s0 + KW / 2), q, nc);
            columns<KW / 2>(v, row, tile, S, s0, s0 + KW / 2, end, q, nc);
#pragma unroll
            for (int f = 0; f < RPL; ++f) S.pos[base + 32 * f] = row.mask[f] ? row.pos[f] : -1;
        }
        __syncthreads();
        // the pivots, and the pivot rows' windows to their places
        if (tid < end - s0) {
            const Cand<T>& c = S.chosen[tid];
            S.piv[s0 + tid] = k + max(c.pos, 0);  // (-1: a CTA without rows, after an expired wait)
            S.owner[tid] = !kCluster || S.cta[tid] == q ? c.idx : -1;
            if (c.row[0] == T(0)) atomicMin(&S.info, s0 + tid);
        }
        for (int i = tid; i < KW * KW; i += kThreads) {
            const int t = i / KW, g = i % KW;
            if (s0 + t < end && t + g < KW) {
                const Cand<T>& c = S.chosen[t];
                if (!kCluster || S.cta[t] == q) tile[(s0 + t + g) * LD + c.idx] = c.row[g];
            }
        }
        __syncthreads();
        if (!more) break;
        // every pivot row of the window to every CTA, for the other columns
        for (int t = warp; t < KW; t += kWarps) {
            const int o = S.owner[t];
            if (o < 0) continue;
            __align__(16) T part[NV];
#pragma unroll
            for (int g = 0; g < NV; ++g) part[g] = tile[(lane * NV + g) * LD + o];
            const uint4 w = *reinterpret_cast<const uint4*>(part);
            if (kCluster) {
                const uint32_t dst = smem_addr(&S.u[t][lane * NV]), bar = smem_addr(&S.ubar);
                for (int c = 0; c < nc; ++c) send16(in_cta(dst, c), in_cta(bar, c), w);
            } else {
                *reinterpret_cast<uint4*>(&S.u[t][lane * NV]) = w;
            }
        }
        if (kCluster && !*(volatile int*)&S.dead && !wait_phase(smem_addr(&S.ubar), (s0 / KW) & 1)) S.dead = 1;
        __syncthreads();
        switch (s0 / KW) {
            case 0: update_right<3 * KW>(tile, S, s0); break;
            case 1: update_right<2 * KW>(tile, S, s0); break;
            default: update_right<KW>(tile, S, s0); break;
        }
    }
    if (warp < CW)
#pragma unroll
        for (int f = 0; f < RPL; ++f) S.pos[base + 32 * f] = row.pos[f];
    __syncthreads();
    const bool dead = kCluster && S.dead != 0;
#pragma unroll 4
    for (int r = warp; r < NR; r += kWarps) {
        const int pos = S.pos[r];
        if (pos < 0 || dead) continue;
        T* dst = a + (int64_t)(k + pos) * n + k;
#pragma unroll
        for (int c = lane; c < KB; c += 32)
            if (c < kb) dst[c] = tile[c * LD + r];
    }
    if (q == 0)
        for (int j = tid; j < kb; j += kThreads) piv[k + j] = dead ? k + j : S.piv[j];
    if (tid == 0) {
        if (q == 0 && S.info != INT_MAX) atomicCAS(info, 0, k + S.info + 1);
        if (dead) atomicMax(info, n + 1);  // above any column's
    }
    if (kCluster) {
        if (dead) {
            const long long t0 = clock64();
            while (clock64() - t0 < kSettleCycles) {
            }
        }
        cg::this_cluster().sync();  // no CTA leaves while another may still send to it
        if (dead && tid == 0) a[(int64_t)k * n + k] = (T)NAN;  // so that no solution comes of the factors
    }
}

// The forms: column warps and rows per lane for panels of up to 128, 256 and 384 rows in one
// CTA, and for the CTAs of a cluster.
template <typename T>
using Kernel = void (*)(T*, int, int, int, int32_t*, int*, const int*);

constexpr int kCW[4] = {4, 4, 6, 4}, kRPL[4] = {1, 2, 2, 1};
constexpr int form_rows(int f) { return kCW[f] * kRPL[f] * 32; }
constexpr int kCluster = 3;

template <typename T, int F>
constexpr Kernel<T> kForm = panel_kernel<T, kCW[F], kRPL[F], F == kCluster>;

template <typename T>
constexpr int tile_bytes(int f) {
    return kPanelCols<T> * (form_rows(f) + 1) * (int)sizeof(T);
}

template <typename T>
Kernel<T> form(int f) {
    return f == 0 ? kForm<T, 0> : f == 1 ? kForm<T, 1> : f == 2 ? kForm<T, 2> : kForm<T, 3>;
}

template <typename T>
cudaLaunchConfig_t cluster_config(unsigned ctas, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = tile_bytes<T>(kCluster);
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim = {ctas, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// The rows the forms take on the current device, whose limits this sets (a kernel's attributes
// belong to a device).
template <typename T>
int limits_of_device() {
    for (int f = 0; f < 4; ++f)
        if (allow_dynamic_smem((const void*)form<T>(f), (size_t)tile_bytes<T>(f)) != FJ_OK) {
            cudaGetLastError();
            return 0;
        }
    const Kernel<T> many = form<T>(kCluster);
    const bool any_size =
        cudaFuncSetAttribute((const void*)many, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    cudaGetLastError();
    for (unsigned size : {(unsigned)kMaxCtas, 8u, 4u}) {
        if (size > 8 && !any_size) continue;
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = cluster_config<T>(size, &at);
        int clusters = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, many, &cfg);
        cudaGetLastError();
        if (e == cudaSuccess && clusters > 0) return (int)size * form_rows(kCluster);
    }
    return form_rows(2);
}

template <typename T>
int set_up() {
    static std::mutex mu;
    static std::map<int, int> rows;  // by device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    std::lock_guard<std::mutex> g(mu);
    const auto it = rows.find(dev);
    return it != rows.end() ? it->second : rows[dev] = limits_of_device<T>();
}

}  // namespace

template <typename T>
int panel_max_rows() {
    return set_up<T>();
}

template <typename T>
int panel_factor(T* a, int n, int k, int kb, int32_t* piv, int* info, const int* run_flag, cudaStream_t s) {
    const int rows = n - k;
    if (rows > set_up<T>() || kb > kPanelCols<T>) return fail(FJ_ERR_UNSUPPORTED, "panel: %d rows", rows);
    if (rows <= form_rows(2)) {
        const int f = rows <= form_rows(0) ? 0 : rows <= form_rows(1) ? 1 : 2;
        form<T>(f)<<<1, kThreads, tile_bytes<T>(f), s>>>(a, n, k, kb, piv, info, run_flag);
    } else {
        constexpr int per = form_rows(kCluster);
        cudaLaunchAttribute at;
        cudaLaunchConfig_t cfg = cluster_config<T>((unsigned)((rows + per - 1) / per), &at);
        cfg.stream = s;
        FJ_CUDA(cudaLaunchKernelEx(&cfg, form<T>(kCluster), a, n, k, kb, piv, info, run_flag));
    }
    note_launch();
    FJ_LAUNCH_CHECK("panel_kernel");
    return FJ_OK;
}

template int panel_max_rows<double>();
template int panel_max_rows<float>();
template int panel_factor<double>(double*, int, int, int, int32_t*, int*, const int*, cudaStream_t);
template int panel_factor<float>(float*, int, int, int, int32_t*, int*, const int*, cudaStream_t);

}  // namespace fj
