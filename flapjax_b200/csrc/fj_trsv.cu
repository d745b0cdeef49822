// fj_trsv.cu -- getrs for one right-hand side: the permutation, then both substitutions in one
// launch.
//
// A substitution is a chain of diagonal blocks, each waiting for the one before: what bounds
// it is that chain's latency, then the reading of the factors (n^2 doubles in all).  A
// cluster of up to 8 CTAs holds the right-hand side in shared memory, its blocks of 64 rows
// dealt out in turn.  Per block:
//   * One warp of the owner solves the diagonal block, four columns at a time: the four
//     values come to every lane by shuffles, which all lanes solve among themselves, so a
//     shuffle's latency is paid once in four columns.  It sends the 64 solved values to
//     every CTA (st.async, counted by an mbarrier).
//   * The 15 other warps apply them: first to the next block, so that its solve can begin,
//     then to the rest of the CTA's rows while it runs.  The diagonal and the next block's
//     off-diagonal tile come into shared memory by cp.async, two owned blocks ahead.
// A CTA owns one block in every n_cta (two at the turn between the substitutions), and sends
// it only after its warps have applied all but the block before: so when a slot of the ring
// of solved blocks comes round again, 2 n_cta + 2 <= kRing blocks on, every CTA has done
// with what it held.
// Measured, solve (transposed solve) of order 64, 256, 768 and 2048: 12-14, 33, 84 and 214 us
// (13-14, 35, 87, 222), against 40, 163, 494 and 1324 us (34, 150-168, 467-526, 1305-1434)
// for a launch per diagonal block and per update.  The solving warp's 3,100 to 4,000 cycles
// per block (column of the triangle: a shuffle's latency in four, then one DFMA's) are what
// remains on the chain below 768 rows; from 6144 rows (1285 us for 4100) the reading is.
#include <algorithm>

#include <cooperative_groups.h>

#include "fj_trsv.cuh"

namespace fj {
namespace {

namespace cg = cooperative_groups;

constexpr int kB = 64;               // block
constexpr int kPitch = kB + 2;       // of a tile's row in shared memory (16-byte aligned rows)
constexpr int kThreads = 512, kUpdateWarps = kThreads / 32 - 1, kUpdateThreads = 32 * kUpdateWarps;
constexpr int kMaxCtas = 8;
constexpr int kRing = 20;
constexpr int kTile = kB * kPitch;
constexpr int kMaxBuf = 3;           // owned blocks whose tiles are held
constexpr long long kWaitCycles = FJ_WAIT_CYCLES;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

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

struct Shared {
    uint64_t full[kRing];      // solved blocks
    uint64_t tiles[kMaxBuf];   // an owned block's tiles
    uint64_t ready;            // an owned block has every update
    __align__(16) double x[kRing][kB];
    double diag[kB];
    int dead;
};

// Waits for a phase, about a second at most; after the first expiry the CTA waits for nothing, and
// its solved blocks are NaN.  False unless the phase is complete.
__device__ __forceinline__ bool wait(Shared& S, const uint64_t& bar, int phase) {
    const uint32_t a = smem_addr(&bar), parity = (uint32_t)phase & 1u;
    if (kWaitCycles < 0) S.dead = 1;
    else if (try_phase(a, parity)) return true;
    const long long t0 = clock64();
    while (!*(volatile int*)&S.dead) {
        if (try_phase(a, parity)) return true;
        if (clock64() - t0 > kWaitCycles) S.dead = 1;
    }
    return false;
}

// tile[r][c] = lu[r0 + r][c0 + c], zero outside the matrix; two elements a copy where the
// matrix's rows begin 16-byte aligned (a bulk copy per row was slower: 16.5 us for 12.4 at
// 64 rows, 50 for 33 at 256, a single warp issuing 128 of them).
__device__ __forceinline__ void load_tile(const double* __restrict__ lu, int n, int r0, int c0, double* tile,
                                          bool vec, int t) {
    if (vec) {
        for (int i = t; i < kB * kB / 2; i += kUpdateThreads) {
            const int r = i / (kB / 2), c = i % (kB / 2) * 2;
            const bool in = r0 + r < n && c0 + c < n;  // n is even: both elements or neither
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(tile + r * kPitch + c)),
                         "l"(lu + (in ? (int64_t)(r0 + r) * n + c0 + c : 0)), "r"(in ? 16 : 0)
                         : "memory");
        }
        return;
    }
    for (int i = t; i < kB * kB; i += kUpdateThreads) {
        const int r = i / kB, c = i % kB;
        const bool in = r0 + r < n && c0 + c < n;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(tile + r * kPitch + c)),
                     "l"(lu + (in ? (int64_t)(r0 + r) * n + c0 + c : 0)), "r"(in ? 8 : 0)
                     : "memory");
    }
}

// A triangle's diagonal: of ones, or given by its reciprocals; or itself, where one of these would
// not be a normal number (a division stands in the chain: 64 of them in a block).
enum Diag { kOnes, kReciprocals, kDivisors };

__device__ __forceinline__ bool has_reciprocal(double d) {
    return ((unsigned)__double2hiint(d) & 0x7fffffffu) - 0x00100000u < 0x7fd00000u - 0x00100000u;
}

// Four columns of the block's triangle (kHigh: of its rows 32 ..): lower, ascending from
// j0 = 4 g, or upper, descending from 4 g + 3.  Their rows' lanes come to hold the solved
// values (times the diagonal, unless it is unit) by the same operations as every lane's x.
template <bool kTrans, bool kLower, Diag kDiag, bool kHigh>
__device__ __forceinline__ void solve4(const double* tile, const double* diag, double& v0, double& v1, int g, int lane) {
    constexpr unsigned full = 0xffffffffu;
    // M(r, c) lies at tile[r][c], or (kTrans) at tile[c][r]
    auto at = [&](int r, int c) { return kTrans ? tile[c * kPitch + r] : tile[r * kPitch + c]; };
    double x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = __shfl_sync(full, kHigh ? v1 : v0, (kLower ? 4 * g + i : 4 * g + 3 - i) & 31);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int j = kLower ? 4 * g + i : 4 * g + 3 - i;
        if (kDiag == kReciprocals) x[i] *= diag[j];
        if (kDiag == kDivisors) x[i] /= diag[j];
#pragma unroll
        for (int h = i + 1; h < 4; ++h)
            x[h] = fma(-at(kLower ? 4 * g + h : 4 * g + 3 - h, j), x[i], x[h]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int j = kLower ? 4 * g + i : 4 * g + 3 - i;
        if (kLower) {
            if (!kHigh && lane > j) v0 = fma(-at(lane, j), x[i], v0);
            if (!kHigh || lane + 32 > j) v1 = fma(-at(lane + 32, j), x[i], v1);
        } else {
            if (kHigh || lane < j) v0 = fma(-at(lane, j), x[i], v0);
            if (kHigh && lane + 32 < j) v1 = fma(-at(lane + 32, j), x[i], v1);
        }
    }
}

// One warp solves the block's triangle on v (rows lane, lane + 32).
template <bool kTrans, bool kLower, Diag kDiag>
__device__ __forceinline__ void solve_block(const double* tile, const double* diag, double& v0, double& v1, int lane) {
    if (kLower) {
#pragma unroll 2
        for (int g = 0; g < 8; ++g) solve4<kTrans, kLower, kDiag, false>(tile, diag, v0, v1, g, lane);
#pragma unroll 2
        for (int g = 8; g < 16; ++g) solve4<kTrans, kLower, kDiag, true>(tile, diag, v0, v1, g, lane);
    } else {
#pragma unroll 2
        for (int g = 15; g >= 8; --g) solve4<kTrans, kLower, kDiag, true>(tile, diag, v0, v1, g, lane);
#pragma unroll 2
        for (int g = 7; g >= 0; --g) solve4<kTrans, kLower, kDiag, false>(tile, diag, v0, v1, g, lane);
    }
    if (kDiag == kReciprocals) {
        v0 *= diag[lane];
        v1 *= diag[lane + 32];
    }
    if (kDiag == kDivisors) {
        v0 /= diag[lane];
        v1 /= diag[lane + 32];
    }
}

// The same by divisions, of a block with a diagonal element whose reciprocal is no normal number;
// n: the matrix's rows from this block's first.  (Not inlined: rare, and the solving warp's loop stays
// short.)
template <bool kTrans>
__device__ __noinline__ double2 divide_block(const double* tile, double* diag, double2 v, int lane, int n) {
    for (int r = lane; r < kB; r += 32) diag[r] = r < n ? tile[r * kPitch + r] : 1.0;
    __syncwarp();
    solve_block<kTrans, kTrans, kDivisors>(tile, diag, v.x, v.y, lane);
    return v;
}

// y -= M x for eight rows, 8 lanes per row: the lane group's rows begin at m and m + 4 stride
// (null: no such row); x: the lane's eight values.
template <bool kVec>
__device__ __forceinline__ void apply8(const double* m0, const double* m1, const double (&x)[8], int lane, double* y) {
    double s[2] = {0.0, 0.0};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const double* m = u ? m1 : m0;
        if (m == nullptr) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double* q = m + (lane & 7) * 2 + 16 * i;
            const double2 w = kVec ? *reinterpret_cast<const double2*>(q) : make_double2(q[0], q[1]);
            s[u] = fma(w.x, x[2 * i], s[u]);
            s[u] = fma(w.y, x[2 * i + 1], s[u]);
        }
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
        s[1] += __shfl_xor_sync(0xffffffffu, s[1], off);
    }
    if ((lane & 7) == 0) {
        y[lane / 8] -= s[0];
        y[4 + lane / 8] -= s[1];
    }
}

// y -= M^T x for a lane's row: column `m` of `len` rows, `stride` apart.
__device__ __forceinline__ void apply_column(const double* m, int64_t stride, int len, const double* x, double* y) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int j = 0;
#pragma unroll 4
    for (; j + 4 <= len; j += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = fma(m[(j + i) * stride], x[j + i], s[i]);
    }
    for (; j < len; ++j) s[0] = fma(m[j * stride], x[j], s[0]);
    *y -= (s[0] + s[1]) + (s[2] + s[3]);
}

template <bool kTrans>
__global__ void __launch_bounds__(kThreads, 1)
    substitute_kernel(const double* __restrict__ lu, int n, const double* __restrict__ in, double* __restrict__ out,
                      int nbuf) {
    extern __shared__ __align__(16) unsigned char raw[];
    double* tiles = reinterpret_cast<double*>(raw);              // [nbuf][2][kTile]: diagonal, next off-diagonal
    double* y = tiles + (size_t)nbuf * 2 * kTile;                // this CTA's rows, block by block
    __shared__ Shared S;
    cg::cluster_group cl = cg::this_cluster();
    const int q = (int)cl.block_rank(), nc = (int)cl.num_blocks();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = (n + kB - 1) / kB, steps = 2 * nb;
    auto block_of = [&](int t) { return t < nb ? t : steps - 1 - t; };
    auto owned = [&](int b) { return b % nc == q; };
    if (tid == 0) {
        S.dead = 0;
        for (int i = 0; i < kRing; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.full[i])) : "memory");
        for (int i = 0; i < nbuf; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&S.tiles[i])), "n"(kUpdateThreads)
                         : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&S.ready)), "n"(kUpdateWarps) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int b = q; b < nb; b += nc)
        for (int i = tid; i < kB; i += kThreads)
            y[b / nc * kB + i] = b * kB + i < n ? in[b * kB + i] : 0.0;
    cl.sync();  // every CTA runs, its barriers ready, and has read its part of the right-hand side

    // The steps this CTA owns, in order: k-th owned step.
    if (warp == 0) {
        int k = 0;
        for (int t = 0; t < steps; ++t) {
            const int b = block_of(t);
            if (!owned(b)) continue;
            const bool lower = t < nb;
            const bool unit = lower != kTrans;  // L is unit lower, U^T is not; U is not, L^T is unit upper
            const double* tile = tiles + (size_t)(k % nbuf) * 2 * kTile;
            wait(S, S.tiles[k % nbuf], k / nbuf);
            bool divide = false;
            if (!unit) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = lane + 32 * h;
                    const double d = b * kB + r < n ? tile[r * kPitch + r] : 1.0;
                    S.diag[r] = 1.0 / d;
                    divide = divide || !has_reciprocal(d);
                }
                divide = __any_sync(0xffffffffu, divide);
            }
            __syncwarp();
            wait(S, S.ready, k);
            double* yb = y + b / nc * kB;
            double v0 = yb[lane], v1 = yb[lane + 32];
            const bool dead = *(volatile int*)&S.dead;
            if (unit) {  // (lower where not transposed, as U is the other way round)
                solve_block<kTrans, !kTrans, kOnes>(tile, S.diag, v0, v1, lane);
            } else if (divide) {
                const double2 v = divide_block<kTrans>(tile, S.diag, make_double2(v0, v1), lane, n - b * kB);
                v0 = v.x;
                v1 = v.y;
            } else {
                solve_block<kTrans, kTrans, kReciprocals>(tile, S.diag, v0, v1, lane);
            }
            if (dead) v0 = v1 = NAN;
            yb[lane] = v0;
            yb[lane + 32] = v1;
            __threadfence_block();  // the update warps meet these rows again in the second substitution
            __syncwarp();
            const uint4 w = reinterpret_cast<const uint4*>(yb)[lane];
            const int slot = t % kRing;
            const uint32_t dst = smem_addr(&S.x[slot][2 * lane]), bar = smem_addr(&S.full[slot]);
            for (int c = 0; c < nc && t + 1 < steps; ++c) {
                uint32_t d, rb;
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(dst), "r"(c));
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(bar), "r"(c));
                asm volatile(
                    "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(d),
                    "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w), "r"(rb)
                    : "memory");
            }
            if (!lower) {
                if (b * kB + lane < n) out[b * kB + lane] = v0;
                if (b * kB + lane + 32 < n) out[b * kB + lane + 32] = v1;
            }
            ++k;
        }
    } else {
        const int u = tid - 32, uw = warp - 1;
        const bool vec = (n & 1) == 0 && ((uintptr_t)lu & 15) == 0;  // rows begin 16-byte aligned
        int ahead = 0, ahead_t = 0;  // owned steps whose tiles are under way, and where the next may be
        auto prefetch = [&]() {
            while (ahead_t < steps && !owned(block_of(ahead_t))) ++ahead_t;
            if (ahead_t >= steps) return;
            const int b = block_of(ahead_t);
            double* tile = tiles + (size_t)(ahead % nbuf) * 2 * kTile;
            const uint32_t bar = smem_addr(&S.tiles[ahead % nbuf]);
            load_tile(lu, n, b * kB, b * kB, tile, vec, u);
            const int prev = ahead_t < nb ? b - 1 : b + 1;  // the block solved before it
            if (prev >= 0 && prev < nb)  // as it lies in memory
                load_tile(lu, n, (kTrans ? prev : b) * kB, (kTrans ? b : prev) * kB, tile + kTile, vec, u);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
            ++ahead;
            ++ahead_t;
        };
        int k = 0;  // owned steps made ready
        for (int i = 0; i < nbuf - 1; ++i) prefetch();
        auto arrive = [&]() {
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&S.ready)) : "memory");
            ++k;
            prefetch();  // into the buffer of the owned block solved before the last
        };
        if (owned(0)) arrive();
        bool current = true;  // every phase so far complete: the next may be begun
        for (int t = 0; t + 1 < steps; ++t) {
            const int b = block_of(t), next = block_of(t + 1), slot = t % kRing;
            const bool lower = t < nb;
            if (u == 0 && current)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&S.full[slot])),
                             "n"(kB * 8)
                             : "memory");
            current = wait(S, S.full[slot], t / kRing) && current;
            double x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = S.x[slot][(lane & 7) * 2 + 16 * (i / 2) + (i & 1)];
            // A warp always takes the same rows: groups of 8 (kTrans: 32) rows of this CTA's blocks
            // dealt out in turn, so no two warps meet in one.
            constexpr int kPer = kTrans ? 2 : 8;  // groups per block
            if (owned(next)) {
                if (t + 1 != nb) {  // (at the turn the same block follows, with nothing to apply)
                    const double* tile = tiles + ((size_t)(k % nbuf) * 2 + 1) * kTile;
                    wait(S, S.tiles[k % nbuf], k / nbuf);
                    const int first = next / nc * kPer;
                    for (int g = first + ((uw - first) % kUpdateWarps + kUpdateWarps) % kUpdateWarps; g < first + kPer;
                         g += kUpdateWarps) {
                        if (kTrans) {
                            const int r = (g - first) * 32 + lane;
                            apply_column(tile + r, kPitch, kB, S.x[slot], y + g * 32 + lane);
                        } else {
                            const double* m = tile + ((g - first) * 8 + lane / 8) * kPitch;
                            apply8<true>(m, m + 4 * kPitch, x, lane, y + g * 8);
                        }
                    }
                }
                arrive();
            }
            if (t == nb - 1) continue;  // the first substitution's last block meets no rows
            // the other rows of this CTA: its blocks [l0, l1) lie after `next`
            const int mine = (nb - q + nc - 1) / nc;
            const int l0 = lower ? (next + 1 > q ? (next + 1 - q + nc - 1) / nc : 0) : 0;
            const int l1 = lower ? mine : (next > q ? (next - q + nc - 1) / nc : 0);
            const int len = min(kB, n - b * kB);
            const int first = l0 * kPer;
            for (int g = first + ((uw - first) % kUpdateWarps + kUpdateWarps) % kUpdateWarps; g < l1 * kPer;
                 g += kUpdateWarps) {
                const int row0 = (q + g / kPer * nc) * kB + g % kPer * (kB / kPer);  // the group's first row
                if (kTrans) {
                    if (row0 + lane < n)
                        apply_column(lu + (int64_t)b * kB * n + row0 + lane, n, len, S.x[slot], y + g * 32 + lane);
                    continue;
                }
                const int r = row0 + lane / 8;
                const double* m = lu + (int64_t)r * n + (int64_t)b * kB;
                const double *m0 = r < n ? m : nullptr, *m1 = r + 4 < n ? m + (int64_t)4 * n : nullptr;
                if (len == kB) {
                    if (vec) apply8<true>(m0, m1, x, lane, y + g * 8);
                    else apply8<false>(m0, m1, x, lane, y + g * 8);
                } else {  // the matrix ends inside the block's columns
                    double s0 = 0.0, s1 = 0.0;
                    for (int c = lane & 7; c < len; c += 8) {
                        const double xc = S.x[slot][c];
                        if (m0 != nullptr) s0 = fma(m0[c], xc, s0);
                        if (m1 != nullptr) s1 = fma(m1[c], xc, s1);
                    }
#pragma unroll
                    for (int off = 4; off > 0; off >>= 1) {
                        s0 += __shfl_xor_sync(0xffffffffu, s0, off);
                        s1 += __shfl_xor_sync(0xffffffffu, s1, off);
                    }
                    if ((lane & 7) == 0) {
                        y[g * 8 + lane / 8] -= s0;
                        y[g * 8 + 4 + lane / 8] -= s1;
                    }
                }
            }
        }
    }
    if (*(volatile int*)&S.dead) {  // the CTA's own copies and sends arrive first
        asm volatile("cp.async.wait_all;" ::: "memory");
        const long long t0 = clock64();
        while (clock64() - t0 < kSettleCycles) {
        }
    }
    cl.sync();  // no CTA leaves while another may still send to it
}

template <int kChunk>
__global__ void __launch_bounds__(1024) permute_kernel(const int32_t* __restrict__ piv, int n,
                                                       const double* __restrict__ b, double* __restrict__ x,
                                                       int scatter) {
    extern __shared__ int perm[];
    __shared__ PermScratch<kChunk> S;
    build_perm(piv, n, perm, S);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        if (scatter) x[perm[i]] = b[i];
        else x[i] = b[perm[i]];
    }
}

}  // namespace

int lu_substitute64(const double* lu, int n, const int32_t* piv, double* b, double* work, bool transposed,
                    cudaStream_t s) {
    const size_t psm = (size_t)n * sizeof(int);
    if (n > kPermRows<kPermChunkSmall>) return fail(FJ_ERR_UNSUPPORTED, "lu_solve: n=%d too large", n);
    auto* permute = n <= kPermRows<kPermChunk> ? permute_kernel<kPermChunk> : permute_kernel<kPermChunkSmall>;
    FJ_TRY(allow_dynamic_smem((const void*)permute, psm));
    const int nb = (n + kB - 1) / kB;
    // one CTA per four blocks: below, the exchange costs more than the reading it shares
    const int nc = std::max(1, std::min(kMaxCtas, nb / 4));
    const size_t rows = (size_t)((nb + nc - 1) / nc) * kB * sizeof(double);
    auto bytes = [&](int nbuf) { return (size_t)nbuf * 2 * kTile * sizeof(double) + rows; };
    constexpr size_t kRoom = 232448 - sizeof(Shared) - 1024;  // shared memory of a CTA
    const int nbuf = bytes(kMaxBuf) <= kRoom ? kMaxBuf : 2;
    if (bytes(nbuf) > kRoom) return fail(FJ_ERR_UNSUPPORTED, "lu_solve: n=%d too large", n);
    const void* fn = transposed ? (const void*)substitute_kernel<true> : (const void*)substitute_kernel<false>;
    FJ_TRY(allow_dynamic_smem(fn, bytes(nbuf)));
    if (!transposed) {
        permute<<<1, 1024, psm, s>>>(piv, n, b, work, 0);
        note_launch();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nc);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = bytes(nbuf);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim = {(unsigned)nc, 1, 1};
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (!transposed) {
        FJ_CUDA(cudaLaunchKernelEx(&cfg, substitute_kernel<false>, lu, n, (const double*)work, b, nbuf));
    } else {
        FJ_CUDA(cudaLaunchKernelEx(&cfg, substitute_kernel<true>, lu, n, (const double*)b, work, nbuf));
        permute<<<1, 1024, psm, s>>>(piv, n, work, b, 1);
        note_launch();
    }
    note_launch();
    FJ_LAUNCH_CHECK("lu_substitute64");
    return FJ_OK;
}

}  // namespace fj
