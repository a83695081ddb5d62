// Sparse triangular solves and ILU(0) on CSR matrices (the analysis, the
// solve and the factorization kernels, and their C ABI).  The design is
// described at the top of hpb_tri.cuh.
//
// Arithmetic.  Every operation goes through the round-to-nearest intrinsics
// (a - l*u as one FMA per real product, complex products and quotients by
// the textbook formulas spelled out below), so a row's result does not
// depend on compiler contraction and equals the CPU restatement
// (oracle/oro.c, oro_csr_trsv_* / oro_csr_ilu0_*) bit for bit: each row is
// computed by one thread, over its entries in index order, whatever the
// schedule.
#include <algorithm>
#include <atomic>
#include <climits>
#include <mutex>
#include <vector>

#include "hpb_fused.cuh"
#include "hpb_tri.cuh"

namespace hpb {
namespace tri {
namespace {

constexpr int kSortThreads = 1024;
constexpr int kPre = 4;                          // dependencies per row prefetched into registers
constexpr int kMore = 10;                        // solve: those of rows with more than kPre, at most
constexpr int kMerge = 8;                        // ILU(0): update pairs per batch of loads
// Every wait ends after kWaitNs of GPU time (%globaltimer) at the latest.
// A legitimate wait lasts at most as long as the launch itself (a tile waits
// for rows of tiles that started earlier), so a launch whose waits run out
// is either broken or a factorization / solve whose dependency chain takes
// seconds; both report HPB_ERROR_TIMEOUT.
constexpr unsigned long long kWaitNs = 4000000000ull;

// ---- arithmetic -----------------------------------------------------------
__device__ __forceinline__ float fms(float a, float l, float u) { return __fmaf_rn(-l, u, a); }
__device__ __forceinline__ double fms(double a, double l, double u) { return __fma_rn(-l, u, a); }
// a - l*u with l*u = (lr ur - li ui) + i (lr ui + li ur)
__device__ __forceinline__ cf fms(cf a, cf l, cf u) {
    return cf{__fmaf_rn(-l.re, u.re, __fmaf_rn(l.im, u.im, a.re)), __fmaf_rn(-l.re, u.im, __fmaf_rn(-l.im, u.re, a.im))};
}
__device__ __forceinline__ cd fms(cd a, cd l, cd u) {
    return cd{__fma_rn(-l.re, u.re, __fma_rn(l.im, u.im, a.re)), __fma_rn(-l.re, u.im, __fma_rn(-l.im, u.re, a.im))};
}
__device__ __forceinline__ float scale(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double scale(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ cf scale(cf a, cf b) {
    return cf{__fmaf_rn(a.re, b.re, -__fmul_rn(a.im, b.im)), __fmaf_rn(a.re, b.im, __fmul_rn(a.im, b.re))};
}
__device__ __forceinline__ cd scale(cd a, cd b) {
    return cd{__fma_rn(a.re, b.re, -__dmul_rn(a.im, b.im)), __fma_rn(a.re, b.im, __dmul_rn(a.im, b.re))};
}
__device__ __forceinline__ float quot(float a, float d) { return __fdiv_rn(a, d); }
__device__ __forceinline__ double quot(double a, double d) { return __ddiv_rn(a, d); }
// a / d = (a conj(d)) / |d|^2
__device__ __forceinline__ cf quot(cf a, cf d) {
    const float den = __fmaf_rn(d.re, d.re, __fmul_rn(d.im, d.im));
    return cf{__fdiv_rn(__fmaf_rn(a.re, d.re, __fmul_rn(a.im, d.im)), den),
              __fdiv_rn(__fmaf_rn(a.im, d.re, -__fmul_rn(a.re, d.im)), den)};
}
__device__ __forceinline__ cd quot(cd a, cd d) {
    const double den = __fma_rn(d.re, d.re, __dmul_rn(d.im, d.im));
    return cd{__ddiv_rn(__fma_rn(a.re, d.re, __dmul_rn(a.im, d.im)), den),
              __ddiv_rn(__fma_rn(a.im, d.re, -__dmul_rn(a.re, d.im)), den)};
}
__device__ __forceinline__ bool zero_of(float a) { return a == 0.0f; }
__device__ __forceinline__ bool zero_of(double a) { return a == 0.0; }
__device__ __forceinline__ bool zero_of(cf a) { return a.re == 0.0f && a.im == 0.0f; }
__device__ __forceinline__ bool zero_of(cd a) { return a.re == 0.0 && a.im == 0.0; }

// L2 loads (values another block or warp wrote during this kernel)
__device__ __forceinline__ float ldcgE(const float* p, int64_t i) { return __ldcg(p + i); }
__device__ __forceinline__ double ldcgE(const double* p, int64_t i) { return __ldcg(p + i); }
__device__ __forceinline__ cf ldcgE(const cf* p, int64_t i) {
    const float* q = reinterpret_cast<const float*>(p + i);
    return cf{__ldcg(q), __ldcg(q + 1)};
}
__device__ __forceinline__ cd ldcgE(const cd* p, int64_t i) {
    const double* q = reinterpret_cast<const double*>(p + i);
    return cd{__ldcg(q), __ldcg(q + 1)};
}

__device__ __forceinline__ void stcgE(float* p, int64_t i, float v) { __stcg(p + i, v); }
__device__ __forceinline__ void stcgE(double* p, int64_t i, double v) { __stcg(p + i, v); }
__device__ __forceinline__ void stcgE(cf* p, int64_t i, cf v) {
    float* q = reinterpret_cast<float*>(p + i);
    __stcg(q, v.re);
    __stcg(q + 1, v.im);
}
__device__ __forceinline__ void stcgE(cd* p, int64_t i, cd v) {
    double* q = reinterpret_cast<double*>(p + i);
    __stcg(q, v.re);
    __stcg(q + 1, v.im);
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned long long ld_relaxed64(const void* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_relaxed32(const void* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(void* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed32(void* p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A timeout is sticky: once one wait has given up, every later wait of the
// launch returns at its next check of the error word, so a failed launch
// ends within about one wait limit instead of one limit per waiting row.
__device__ __forceinline__ bool timed_out(const int* err) {
    return (*reinterpret_cast<const volatile int*>(err) & kErrTimeout) != 0;
}

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Deadline bookkeeping for one wait: check() every `every` polls; true when
// the wait must stop (limit reached, recorded; or another wait timed out).
struct Waiter {
    unsigned long long t0 = 0;
    long long it = 0;
    unsigned long long limit = kWaitNs;
    Waiter() = default;
    __device__ __forceinline__ explicit Waiter(unsigned long long lim) : limit(lim) {}
    __device__ __forceinline__ bool check(int* err, int every_mask) {
        if ((++it & every_mask) != 0) return false;
        if (timed_out(err)) return true;
        const unsigned long long now = gtimer();
        if (t0 == 0) {
            t0 = now;
            return false;
        }
        if (now - t0 > limit) {
            atomicOr(err, kErrTimeout);
            return true;
        }
        return false;
    }
};

// Wait (bounded) until row j of another tile is published.
__device__ __forceinline__ void wait_row(const unsigned* flags, int32_t j, int* err) {
    Waiter w;
    while (ld_acquire(flags + j) == 0u)
        if (w.check(err, 63)) return;
}

// Lane 0 waits (bounded) until the tile's levels [0, l) are complete; then
// the warp may read what those levels wrote.
__device__ __forceinline__ void wait_levels(volatile int* done, int l, int lane, int* err) {
    if (lane == 0) {
        Waiter w;
        while (*done < l)
            if (w.check(err, 1023)) break;
    }
    __syncwarp();
    __threadfence_block();
}

// ---- analysis -------------------------------------------------------------
// Per row: validate the structure (row pointers monotone and within nnz,
// columns in range and strictly increasing), locate the diagonal, and the
// dependency range: strictly lower part [rp[i], first column >= i) or
// strictly upper part (first column > i, rp[i+1]).
__global__ void k_tri_rows(int32_t n, int64_t nnz, int upper, const int32_t* __restrict__ rp,
                           const int32_t* __restrict__ ci, int32_t* __restrict__ beg, int32_t* __restrict__ cnt,
                           int32_t* __restrict__ dpos, int* err, int* missing) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t b = rp[i], e = rp[i + 1];
    int bad = 0;
    if (b < 0 || e < b || int64_t(e) > nnz) {
        bad |= kErrColumn;
        b = e = 0;
    }
    int32_t prev = -1, dp = -1, ge = e, gt = e;
    for (int32_t k = b; k < e; ++k) {
        const int32_t c = ci[k];
        if (c < 0 || c >= n) bad |= kErrColumn;
        if (c <= prev) bad |= kErrUnsorted;
        prev = c;
        if (c == i) dp = k;
        if (c >= i && ge == e) ge = k;
        if (c > i && gt == e) gt = k;
    }
    if (bad) atomicOr(err, bad);
    if (dp < 0) atomicAdd(missing, 1);
    beg[i] = upper ? gt : b;
    cnt[i] = upper ? e - gt : ge - b;
    dpos[i] = dp;
}

// Levels: the level of a row is the length of the longest chain of
// dependencies ending at it over the whole triangle.  One block per tile,
// tiles taken by ticket in the solve's order (ascending for a lower,
// descending for an upper triangle), all of them at work at once.  A block
// first lists, for each of its rows, the rows of the tile that depend on it
// (counts, a scan and a fill in shared memory) and how many dependencies each
// row waits for.  Then one warp takes the rows whose dependencies are all
// known from a queue, 32 at a time, publishes their levels to glev and
// hands them on to their dependents, whose last dependency puts them on the
// queue; the other warps poll the levels of other tiles' rows (glev holds -1
// until a level is published) and hand them on the same way.  Each edge is
// touched once, in whatever order the levels become known, so the time is
// the chain's and no tile waits for another to finish.
// Measured on B200: 1.0 ms a triangle for the 1024^2 5-point operator (2047
// levels, 128 tiles), against 23.4 ms for relaxation sweeps over the tiles
// one after another; about 0.3 us a level and 5 us a tile boundary.  The
// polling lanes hold all of a 7-point tile's dependencies on other tiles at
// once (10 each): with 4 or 8 a lane waits for one that comes late while
// others are there already (96^3: 6 and 2 ms instead of 0.6).
// A tile with more than kMaxEdges dependencies inside it takes the sweeps,
// once all levels from outside are known.
constexpr int kGlThreads = 1024;
constexpr int kMaxEdges = 7 * kTriTile;  // in-tile dependencies of a tile
constexpr int kGlSlots = 10;             // other-tile levels in flight per polling lane
struct LevelTile {
    int lev[kTriTile + 1];       // the largest level + 1 of the dependencies met so far (last: no row)
    int left[kTriTile + 1];      // dependencies not met yet
    uint16_t queue[kTriTile];    // rows in the order they became ready (kNoRow: not yet)
    int off[kTriTile];           // dependents met while listing; general list: end of each row's part of `to`
    union {
        uint16_t to4[kTriTile][4];  // up to four dependents of each row (kTriTile: none)
        uint16_t to[kMaxEdges];     // general list of dependents
    };
    int tail, edges, more, scan[kGlThreads / 32];
};
constexpr uint16_t kNoRow = 0xFFFFu;

// Dependency j of row i of the tile [base, base + m): does it count at all
// (within range and in the solve's direction, so the graph has no cycle even
// before the structure checks are read)?
template <bool UPPER>
__device__ __forceinline__ bool is_dep(int32_t n, int32_t i, int32_t j) {
    return j >= 0 && j < n && (UPPER ? j > i : j < i);
}

// Row d has met a dependency of level lv - 1; its last one puts it on the
// queue.  The maximum is released with the count and acquired by whoever takes
// the count to zero, the row released with its place in the queue, so whoever
// takes it off (next_row) finds its final level.
__device__ __forceinline__ void meet(LevelTile& T, int d, int lv) {
    asm volatile("red.relaxed.cta.shared::cta.max.s32 [%0], %1;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(&T.lev[d]))),
                 "r"(lv)
                 : "memory");
    int left;
    asm volatile("atom.acq_rel.cta.shared::cta.add.s32 %0, [%1], -1;"
                 : "=r"(left)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&T.left[d])))
                 : "memory");
    if (left == 1) {
        int at;
        asm volatile("atom.relaxed.cta.shared::cta.add.s32 %0, [%1], 1;"
                     : "=r"(at)
                     : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&T.tail)))
                     : "memory");
        asm volatile("st.release.cta.shared::cta.u16 [%0], %1;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&T.queue[at]))),
                     "h"(uint16_t(d))
                     : "memory");
    }
}
// The queue's entry at `at` (kNoRow: not there yet).
__device__ __forceinline__ int next_row(const LevelTile& T, int at) {
    uint16_t v;
    asm volatile("ld.acquire.cta.shared::cta.u16 %0, [%1];"
                 : "=h"(v)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&T.queue[at])))
                 : "memory");
    return int(v);
}

template <bool UPPER>
__global__ void __launch_bounds__(kGlThreads, 1)
k_tri_levels(int32_t n, int32_t ntiles, const int32_t* __restrict__ ci, const int32_t* __restrict__ beg,
             const int32_t* __restrict__ cnt, int32_t* glev, unsigned* ticket, int* err) {
    extern __shared__ __align__(16) unsigned char shraw[];
    LevelTile& T = *reinterpret_cast<LevelTile*>(shraw);
    __shared__ int s_tile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        const int tk = int(atomicAdd(ticket, 1u));
        s_tile = UPPER ? ntiles - 1 - tk : tk;
        T.tail = 0;
    }
    __syncthreads();
    const int t = s_tile;
    if (t < 0 || t >= ntiles) return;
    const int32_t base = int32_t(t) * kTriTile;
    const int32_t m = min(kTriTile, n - base);
    if (tid == 0) {
        T.more = 0;
        T.lev[kTriTile] = 0;
        T.left[kTriTile] = INT_MAX;  // "no dependent" never becomes ready
    }
    for (int r = tid; r < kTriTile; r += kGlThreads) {
        T.lev[r] = 0;
        T.off[r] = 0;
        T.queue[r] = kNoRow;
        *reinterpret_cast<uint2*>(T.to4[r]) = make_uint2(kTriTile * 0x10001u, kTriTile * 0x10001u);
    }
    __syncthreads();
    // ---- who depends on each row: up to four dependents in one go
    bool more = false;
    for (int r = tid; r < m; r += kGlThreads) {
        const int32_t i = base + r, b = __ldg(beg + i), c = __ldg(cnt + i);
        int left = 0;
        for (int32_t k = b; k < b + c; ++k) {
            const int32_t j = __ldg(ci + k), jl = j - base;
            if (!is_dep<UPPER>(n, i, j)) continue;
            ++left;
            if (jl >= 0 && jl < m) {
                const int at = atomicAdd(&T.off[jl], 1);
                if (at < 4) T.to4[jl][at] = uint16_t(r);
                more |= at >= 4;
            }
        }
        T.left[r] = left;
        if (left == 0) T.queue[atomicAdd(&T.tail, 1)] = uint16_t(r);
    }
    more = __syncthreads_or(more);
    if (more) {  // ---- rows with more dependents: a list by offsets
        // exclusive scan of off: kTriTile / kGlThreads entries per thread
        {
            constexpr int P = kTriTile / kGlThreads;
            int v[P], s = 0;
#pragma unroll
            for (int k = 0; k < P; ++k) {
                v[k] = T.off[tid * P + k];
                s += v[k];
            }
            int x = s;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += y;
            }
            if (lane == 31) T.scan[warp] = x;
            __syncthreads();
            if (warp == 0) {
                const int ws = T.scan[lane];
                int y = ws;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int z = __shfl_up_sync(0xffffffffu, y, d);
                    if (lane >= d) y += z;
                }
                T.scan[lane] = y - ws;
                if (lane == 31) T.edges = y;
            }
            __syncthreads();
            int acc = T.scan[warp] + x - s;
#pragma unroll
            for (int k = 0; k < P; ++k) {
                T.off[tid * P + k] = acc;
                acc += v[k];
            }
        }
        __syncthreads();
        if (T.edges > kMaxEdges) {  // ---- relaxation sweeps
            volatile int* lev = T.lev;
            int* ext = T.left;
            for (int r = tid; r < m; r += kGlThreads) {  // 1 + the largest level from outside the tile
                const int32_t i = base + r, b = __ldg(beg + i), c = __ldg(cnt + i);
                int e = 0;
                for (int32_t k = b; k < b + c; ++k) {
                    const int32_t j = __ldg(ci + k), jl = j - base;
                    if (!is_dep<UPPER>(n, i, j) || (jl >= 0 && jl < m)) continue;
                    Waiter w;
                    int v;
                    while ((v = int(ld_relaxed32(glev + j))) < 0)
                        if (w.check(err, 63)) break;
                    e = max(e, v + 1);
                }
                ext[r] = e;
                lev[r] = e;
            }
            __syncthreads();
            // contiguous segments walked in dependency order until a sweep
            // changes nothing (a sweep that changes something brings one more row
            // of the longest in-tile chain to its final value)
            const int seg = (m + kGlThreads - 1) / kGlThreads;
            const int s0 = min(m, tid * seg), s1 = min(m, s0 + seg);
            int changed, sweeps = 0;
            do {
                changed = 0;
                for (int k = 0; k < s1 - s0; ++k) {
                    const int r = UPPER ? s1 - 1 - k : s0 + k;
                    const int32_t i = base + r, b = __ldg(beg + i), c = __ldg(cnt + i);
                    int lv = ext[r];
                    for (int32_t e = b; e < b + c; ++e) {
                        const int32_t j = __ldg(ci + e), jl = j - base;
                        if (is_dep<UPPER>(n, i, j) && jl >= 0 && jl < m) lv = max(lv, lev[jl] + 1);
                    }
                    if (lv > lev[r]) {
                        lev[r] = lv;
                        changed = 1;
                    }
                }
            } while (__syncthreads_or(changed) && ++sweeps <= m);
            for (int r = tid; r < m; r += kGlThreads) st_relaxed32(glev + base + r, unsigned(lev[r]));
            return;
        }
        for (int r = tid; r < m; r += kGlThreads) {
            const int32_t i = base + r, b = __ldg(beg + i), c = __ldg(cnt + i);
            for (int32_t k = b; k < b + c; ++k) {
                const int32_t j = __ldg(ci + k), jl = j - base;
                if (is_dep<UPPER>(n, i, j) && jl >= 0 && jl < m) T.to[atomicAdd(&T.off[jl], 1)] = uint16_t(r);
            }
        }
        __syncthreads();  // off[r] is now the end of row r's part, its start the end of row r - 1's
    }

    if (warp == 0) {  // ---- the queue
        // Up to eight ready rows: four lanes each, a dependent per lane; more
        // of them: a lane each, its dependents one after another.  This chain
        // of shared loads and atomics is what a level costs, so it is kept
        // short (one warp issues it; every instruction counts).
        int head = 0, spins = 0;
        const int grp = lane >> 2, sub = lane & 3;
        unsigned long long t0 = 0;
        while (head < m) {
            const int wide = head + lane < m ? next_row(T, head + lane) : int(kNoRow);
            int row = __shfl_sync(0xffffffffu, wide, grp);
            const unsigned none = __ballot_sync(0xffffffffu, wide == int(kNoRow));
            const int k = none ? __ffs(int(none)) - 1 : 32;  // rows ready without a gap
            if (k == 0) {
                if ((++spins & 255) != 0) continue;
                const unsigned long long now = gtimer();
                if (t0 == 0) t0 = now;
                if (now - t0 > 2 * kWaitNs) {  // the polls below give up earlier: never expected
                    if (lane == 0) atomicOr(err, kErrTimeout);
                    return;
                }
                continue;
            }
            t0 = 0;
            head += k;
            const bool few = k <= 8;
            if (!few) row = wide;
            if ((few ? grp : lane) < k) {
                const int lv = *reinterpret_cast<volatile int*>(&T.lev[row]);
                if (!more && few) {
                    const int d = T.to4[row][sub];
                    if (d < kTriTile) meet(T, d, lv + 1);
                } else if (!more) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int d = T.to4[row][q];
                        if (d < kTriTile) meet(T, d, lv + 1);
                    }
                } else {
                    const int e1 = T.off[row];
                    for (int e = (row > 0 ? T.off[row - 1] : 0) + (few ? sub : 0); e < e1; e += few ? 4 : 1)
                        meet(T, T.to[e], lv + 1);
                }
                if (!few || sub == 0) st_relaxed32(glev + base + row, unsigned(lv));
            }
            __syncwarp();
        }
        return;
    }
    // ---- levels from other tiles: each lane walks its rows' dependencies,
    // kGlSlots of them in flight
    constexpr int kStride = kGlThreads - 32;
    int r = UPPER ? m - 1 - (tid - 32) : tid - 32;  // in the order the solve needs them
    int32_t b = 0, c = 0, k = 0;
    auto open_row = [&]() {
        k = 0;
        c = 0;
        if (r >= 0 && r < m) {
            b = __ldg(beg + base + r);
            c = __ldg(cnt + base + r);
        }
    };
    open_row();
    int sr[kGlSlots];
    int32_t sj[kGlSlots];
    auto refill = [&](int& row, int32_t& from) {  // the lane's next other-tile dependency, -1: none left
        row = -1;
        from = 0;
        while (r >= 0 && r < m) {
            if (k >= c) {
                r += UPPER ? -kStride : kStride;
                open_row();
                continue;
            }
            const int32_t j = __ldg(ci + b + k), jl = j - base;
            ++k;
            if (is_dep<UPPER>(n, base + r, j) && !(jl >= 0 && jl < m)) {
                row = r;
                from = j;
                return;
            }
        }
    };
#pragma unroll
    for (int q = 0; q < kGlSlots; ++q) refill(sr[q], sj[q]);
    Waiter w;
    int pause = 20;
    for (;;) {
        int v[kGlSlots];
        bool any = false, got = false;
#pragma unroll
        for (int q = 0; q < kGlSlots; ++q)
            if (sr[q] >= 0) {
                v[q] = int(ld_relaxed32(glev + sj[q]));
                any = true;
            }
        if (!any) break;
        const bool stop = w.check(err, 63);
        unsigned met = 0;
#pragma unroll
        for (int q = 0; q < kGlSlots; ++q)
            if (sr[q] >= 0 && (v[q] >= 0 || stop)) {
                meet(T, sr[q], max(v[q], 0) + 1);
                met |= 1u << q;
                got = true;
            }
        if (met != 0u)
#pragma unroll
            for (int q = 0; q < kGlSlots; ++q)
                if ((met >> q) & 1u) refill(sr[q], sj[q]);
        if (got) {
            w = Waiter();
            pause = 20;
        } else {  // a tile far behind the front polls less often
            __nanosleep(pause);
            pause = min(2 * pause, 320);
        }
    }
}

// Bitonic sort of get(0..m-1) (distinct keys) into key[0, m) by the block.
template <class K, class F>
__device__ __forceinline__ void sort_tile(K* key, int m, F get) {
    int size = 32;  // the power of two the sort runs over
    while (size < m) size <<= 1;
    for (int r = threadIdx.x; r < size; r += blockDim.x) key[r] = r < m ? get(r) : ~K(0);
    __syncthreads();
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int q = threadIdx.x; q < size / 2; q += blockDim.x) {
                const int i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), ixj = i | j;
                const K a = key[i], b = key[ixj];
                if ((a > b) == ((i & k) == 0)) {
                    key[i] = b;
                    key[ixj] = a;
                }
            }
            __syncthreads();
        }
}

// Per tile (one block): the tile's rows in (level, row) order -- the order in
// which the solve takes them -- by a bitonic sort in shared memory.  For
// position p of the tile: desc (row, first dependency, dependency count,
// diagonal position) and dsrc, where the first four dependencies are found:
// >= 0 the tile's own position of that row, <= -2 row -(c + 2) of another
// tile, -1 none.  pos is the inverse (position of each row in its tile),
// lvlptr / nlev hold the level starts, and chunks the runs of at most 32
// positions that a warp of the solve takes at a time: chunks[0].x is their
// number, chunks[1 + c] the positions in chunk c that start a level (bits) and
// its first position | length << 16.  Chunks end with a level where that takes
// at most a sixteenth more of them than runs of 32: a level cut in two
// costs a step of the chain twice.  Levels are global, so rows of the
// tile never wait on an other-tile row that is late in its own tile merely
// because of where the tile boundary falls.
__global__ void __launch_bounds__(kSortThreads)
k_tri_sort(int32_t n, const int32_t* __restrict__ ci, const int32_t* __restrict__ beg,
           const int32_t* __restrict__ cnt, const int32_t* __restrict__ dpos, const int32_t* __restrict__ glev,
           int4* __restrict__ desc, int4* __restrict__ dsrc, uint16_t* __restrict__ pos, uint2* __restrict__ chunks,
           int32_t* __restrict__ lvlptr, int32_t* __restrict__ nlev) {
    extern __shared__ __align__(16) unsigned char shraw[];
    unsigned long long* key = reinterpret_cast<unsigned long long*>(shraw);  // kTriTile
    uint16_t* inv = reinterpret_cast<uint16_t*>(key + kTriTile);             // kTriTile
    uint16_t* lst = inv + kTriTile;                                          // kTriTile + 1: level starts
    __shared__ uint16_t cut[kTriChunkCap + 1];  // chunk starts
    __shared__ int ncut;
    __shared__ int first[kTriChunks + 1];  // level starts before each chunk of 32 positions
    __shared__ int s_lo, s_hi;
    const int t = blockIdx.x;
    const int32_t base = int32_t(t) * kTriTile;
    const int32_t m = min(kTriTile, n - base);
    if (threadIdx.x == 0) {
        s_lo = INT_MAX;
        s_hi = 0;
    }
    __syncthreads();
    {
        int lo = INT_MAX, hi = 0;
        for (int r = threadIdx.x; r < m; r += blockDim.x) {
            const int v = glev[base + r];
            lo = min(lo, v);
            hi = max(hi, v);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&s_lo, lo);
            atomicMax(&s_hi, hi);
        }
    }
    __syncthreads();
    // the tile's levels span less than 2^18 unless its chains are very long
    // elsewhere: 32-bit keys then, half the shared-memory traffic
    const int lo = s_lo;
    if (s_hi - lo < (1 << 18)) {
        unsigned* k32 = reinterpret_cast<unsigned*>(key);
        sort_tile(k32, m, [&](int r) { return (unsigned(glev[base + r] - lo) << 13) | unsigned(r); });
        // widened in place
        unsigned v[kTriTile / kSortThreads];
#pragma unroll
        for (int k = 0; k < kTriTile / kSortThreads; ++k) {
            const int p = threadIdx.x + k * kSortThreads;
            v[k] = p < m ? k32[p] : 0u;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTriTile / kSortThreads; ++k) {
            const int p = threadIdx.x + k * kSortThreads;
            if (p < m) key[p] = v[k];
        }
        __syncthreads();
    } else {
        sort_tile(key, m, [&](int r) {
            return (static_cast<unsigned long long>(glev[base + r] - lo) << 13) | static_cast<unsigned long long>(r);
        });
    }
    for (int p = threadIdx.x; p < m; p += blockDim.x) {
        const int r = int(key[p] & 8191ull);
        inv[r] = uint16_t(p);
        pos[base + r] = uint16_t(p);
    }
    // level starts: one ballot per chunk, then a scan of their counts
    const int nc = (m + 31) >> 5, lane = threadIdx.x & 31;
    for (int c = threadIdx.x >> 5; c < kTriChunks; c += blockDim.x >> 5) {
        const int p = 32 * c + lane;
        const bool st = p < m && (p == 0 || (key[p] >> 13) != (key[p - 1] >> 13));
        const uint32_t w = __ballot_sync(0xffffffffu, st);
        if (lane == 0) first[c] = __popc(w);
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan of the kTriChunks counts, kTriChunks / 32 per lane
        int v[kTriChunks / 32], s = 0;
#pragma unroll
        for (int k = 0; k < kTriChunks / 32; ++k) {
            v[k] = first[lane * (kTriChunks / 32) + k];
            s += v[k];
        }
        int x = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        int acc = x - s;
#pragma unroll
        for (int k = 0; k < kTriChunks / 32; ++k) {
            first[lane * (kTriChunks / 32) + k] = acc;
            acc += v[k];
        }
        if (lane == 31) first[kTriChunks] = acc;
    }
    __syncthreads();
    int32_t* lp = lvlptr + size_t(t) * (kTriTile + 1);
    if (threadIdx.x == 0) {
        nlev[t] = first[kTriChunks];
        lp[first[kTriChunks]] = m;
        lst[first[kTriChunks]] = uint16_t(m);
    }
    for (int c = threadIdx.x >> 5; c < nc; c += blockDim.x >> 5) {
        const int p = 32 * c + lane;
        const bool st = p < m && (p == 0 || (key[p] >> 13) != (key[p - 1] >> 13));
        const uint32_t w = __ballot_sync(0xffffffffu, st);
        if (p >= m) continue;
        if (st) {
            const int l = first[c] + __popc(w & ((1u << lane) - 1u));
            lp[l] = p;
            lst[l] = uint16_t(p);
        }
        const int32_t row = base + int32_t(key[p] & 8191ull);
        const int32_t b = __ldg(beg + row), d = __ldg(cnt + row);
        desc[base + p] = make_int4(row, b, d, __ldg(dpos + row));
        int sc[kPre];
#pragma unroll
        for (int k = 0; k < kPre; ++k) {
            sc[k] = -1;
            if (k < d) {
                const int32_t j = __ldg(ci + b + k), jl = j - base;
                // (columns outside [0, n) are reported by k_tri_rows)
                if (j >= 0 && j < n) sc[k] = (jl >= 0 && jl < m) ? int(inv[jl]) : -(j + 2);
            }
        }
        dsrc[base + p] = make_int4(sc[0], sc[1], sc[2], sc[3]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int levels = first[kTriChunks], most = min(nc + nc / 16, kTriChunkCap);
        int k = 0, from = 0;  // the chunk being filled starts at `from`
        cut[0] = 0;
        for (int l = 0; l < levels && k < most; ++l) {
            const int end = lst[l + 1];
            if (end - from <= 32) continue;
            if (lst[l] > from) cut[++k] = uint16_t(from = lst[l]);
            while (end - from > 32 && k < most) cut[++k] = uint16_t(from += 32);
        }
        ncut = k < most ? k + 1 : 0;  // 0: runs of 32
    }
    __syncthreads();
    const int nk = ncut ? ncut : nc;
    chunks += size_t(t) * (kTriChunkCap + 1);
    if (threadIdx.x == 0) chunks[0] = make_uint2(unsigned(nk), 0u);
    for (int c = threadIdx.x >> 5; c < nk; c += blockDim.x >> 5) {
        const int from = ncut ? cut[c] : 32 * c, to = ncut ? (c + 1 < nk ? int(cut[c + 1]) : m) : min(32 * c + 32, m);
        const int p = from + lane;
        const bool st = p < to && (p == 0 || (key[p] >> 13) != (key[p - 1] >> 13));
        const uint32_t w = __ballot_sync(0xffffffffu, st);
        if (lane == 0) chunks[1 + c] = make_uint2(w, unsigned(from) | unsigned(to - from) << 16);
    }
}

// ---- solve ----------------------------------------------------------------
// Rows of other tiles are read from x itself: the solve first fills x with
// a signalling-NaN sentinel, which no arithmetic operation returns (IEEE
// 754 operations deliver quiet NaNs), and every row's value is stored once
// with a relaxed store of the whole (8- or 4-byte) word.  A reader that
// loads anything but the sentinel therefore holds the final value: one L2
// round trip per dependency, issued with the row's other loads before the
// warp waits for its level, instead of a flag acquire followed by the load.
constexpr unsigned long long kSent64 = 0x7FF0DEAD0000BEEFull;  // exponent all ones, quiet bit 0
constexpr unsigned kSent32 = 0x7F80BEEFu;

// Published values: load / store / fill / "still the sentinel" per element
// type (complex: per component; a component is final once it is not the
// sentinel).
template <class E> struct Pub;
template <> struct Pub<double> {
    static __device__ __forceinline__ double load(const double* x, int64_t j) {
        return __longlong_as_double(static_cast<long long>(ld_relaxed64(x + j)));
    }
    static __device__ __forceinline__ void store(double* x, int64_t i, double v) {
        st_relaxed64(x + i, static_cast<unsigned long long>(__double_as_longlong(v)));
    }
    static __device__ __forceinline__ bool pending(double v) {
        return static_cast<unsigned long long>(__double_as_longlong(v)) == kSent64;
    }
    static __device__ __forceinline__ void fill(double* x, int64_t i) {
        x[i] = __longlong_as_double(static_cast<long long>(kSent64));
    }
};
template <> struct Pub<float> {
    static __device__ __forceinline__ float load(const float* x, int64_t j) {
        return __uint_as_float(ld_relaxed32(x + j));
    }
    static __device__ __forceinline__ void store(float* x, int64_t i, float v) {
        st_relaxed32(x + i, __float_as_uint(v));
    }
    static __device__ __forceinline__ bool pending(float v) { return __float_as_uint(v) == kSent32; }
    static __device__ __forceinline__ void fill(float* x, int64_t i) { x[i] = __uint_as_float(kSent32); }
};
template <> struct Pub<cd> {
    static __device__ __forceinline__ cd load(const cd* x, int64_t j) {
        const double* q = reinterpret_cast<const double*>(x + j);
        return cd{Pub<double>::load(q, 0), Pub<double>::load(q, 1)};
    }
    static __device__ __forceinline__ void store(cd* x, int64_t i, cd v) {
        double* q = reinterpret_cast<double*>(x + i);
        Pub<double>::store(q, 0, v.re);
        Pub<double>::store(q, 1, v.im);
    }
    static __device__ __forceinline__ bool pending(cd v) { return Pub<double>::pending(v.re) || Pub<double>::pending(v.im); }
    static __device__ __forceinline__ void fill(cd* x, int64_t i) {
        double* q = reinterpret_cast<double*>(x + i);
        Pub<double>::fill(q, 0);
        Pub<double>::fill(q, 1);
    }
};
template <> struct Pub<cf> {
    static __device__ __forceinline__ cf load(const cf* x, int64_t j) {
        const float* q = reinterpret_cast<const float*>(x + j);
        return cf{Pub<float>::load(q, 0), Pub<float>::load(q, 1)};
    }
    static __device__ __forceinline__ void store(cf* x, int64_t i, cf v) {
        float* q = reinterpret_cast<float*>(x + i);
        Pub<float>::store(q, 0, v.re);
        Pub<float>::store(q, 1, v.im);
    }
    static __device__ __forceinline__ bool pending(cf v) { return Pub<float>::pending(v.re) || Pub<float>::pending(v.im); }
    static __device__ __forceinline__ void fill(cf* x, int64_t i) {
        float* q = reinterpret_cast<float*>(x + i);
        Pub<float>::fill(q, 0);
        Pub<float>::fill(q, 1);
    }
};

// Wait (bounded) until x[j], as last loaded into v, is published.
template <class E>
__device__ __forceinline__ E await_value(const E* x, int32_t j, E v, int* err, unsigned long long lim) {
    Waiter w(lim);
    while (Pub<E>::pending(v)) {
        if (w.check(err, 63)) break;
        v = Pub<E>::load(x, j);
    }
    return v;
}

template <class E>
__global__ void k_tri_fill(int32_t n, E* __restrict__ x, unsigned* ticket) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0u;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        Pub<E>::fill(x, i);
}

// One tile.  What bounds a solve is the chain of levels, so a tile's rows are
// taken in level order, up to 32 positions (a chunk) at a time with one row per
// lane: a warp steps through the levels its chunk spans and passes every
// value to the next level through shared memory with a __syncwarp.  The
// block's warps take the chunks round-robin and hand the chain on from chunk
// to chunk through a named barrier (bar.arrive / bar.sync of the two warps: it
// orders the shared-memory accesses, with no fence).  All that does not
// depend on the chain a warp has done before its turn: descriptors and values
// loaded one and two turns ahead, the values of other tiles' rows polled from
// x, the division by the diagonal prepared.  A level costs a shared load, the
// row's FMAs and a shared store (and, at a non-unit diagonal, a division),
// whatever the number of rows up to 32; wider levels take several chunks.
// Measured on B200 (f64, ILU(0) factors of the 1024^2 5-point operator, 2047
// levels in 128 tiles): lower + upper solve 826 us; with fifteen warps instead
// of seven 902 us, and with these 972 us with chunks of 32 that cut levels in
// two and 2460 us for levels handed round the warps one by one with a receiver
// warp for the other tiles' values.  One tile of 1024 x 8 points, 1031 levels,
// takes 66 / 129 us and each further one 2.0 / 3.0 us: the eight levels it
// starts later, a chunk's worth of waiting and a value's way to L2 and back.
// (Polling the other tiles' values in the shared memory of a cluster's blocks
// instead of L2 took 0.3 us off a tile and was not worth its code.)
// (A solver warp fed through a shared-memory ring by the others was slower,
// 480 / 719 us: about 500 cycles a chunk went into taking over the records.)
// A division by the diagonal sits on the chain, so the loader prepares it:
// the reciprocal of d to twice the working precision, y + z.  With it the
// correctly rounded quotient takes four dependent operations: q = a y + a z,
// which is a / d but for its last rounding, and one correction
// q += (a - d q) y with the residual exact in an FMA, which from a q within
// one ulp gives the rounded a / d (Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, 1990) as long as nothing
// over- or underflows on the way: the diagonal's exponent within +-DivRange::d
// (checked by the loader) and the numerator's within +-DivRange::n; otherwise the
// plain division is taken.
template <class R> struct DivRange;
template <> struct DivRange<double> { static constexpr int d = 100, n = 880; };
template <> struct DivRange<float> { static constexpr int d = 30, n = 80; };
__device__ __forceinline__ int exponent(double v) { return ((__double2hiint(v) >> 20) & 0x7ff) - 1023; }
__device__ __forceinline__ int exponent(float v) { return int((__float_as_uint(v) >> 23) & 0xffu) - 127; }
template <class R>
__device__ __forceinline__ bool within(R v, int e) { return unsigned(exponent(v) + e) <= unsigned(2 * e); }
__device__ __forceinline__ double rcp_rn(double d) { return __drcp_rn(d); }
__device__ __forceinline__ float rcp_rn(float d) { return __frcp_rn(d); }
// A row's prepared diagonal: the divisor (complex: |d|^2) and its reciprocal
// (y = 0 when the plain division has to be taken).
template <class E> struct Prep { typename real_of<E>::type den, y, z; };
template <class E, class R>
__device__ __forceinline__ R div_prepared(R a, const Prep<E>& p) {
    const R q = fma_rn(a, p.y, mul_rn(a, p.z));
    return fma_rn(fma_rn(-p.den, q, a), p.y, q);
}
__device__ __forceinline__ double divisor(double d) { return d; }
__device__ __forceinline__ float divisor(float d) { return d; }
__device__ __forceinline__ float divisor(cf d) { return __fmaf_rn(d.re, d.re, __fmul_rn(d.im, d.im)); }
__device__ __forceinline__ double divisor(cd d) { return __fma_rn(d.re, d.re, __dmul_rn(d.im, d.im)); }
template <class E>
__device__ __forceinline__ Prep<E> prepare_div(E d) {
    using R = typename real_of<E>::type;
    const R den = divisor(d);
    if (!within(den, DivRange<R>::d)) return Prep<E>{den, R(0), R(0)};
    const R y = rcp_rn(den);
    return Prep<E>{den, y, mul_rn(fma_rn(-den, y, R(1)), y)};  // 1/d - y = (1 - d y) / d
}
// a / d = quot(a, d); `on`: the lane's result is used (others skip the plain division)
template <class R>
__device__ __forceinline__ R quot_prepared(R a, R, const Prep<R>& p, bool on) {
    R q = div_prepared(a, p);
    if (on && (p.y == R(0) || !within(a, DivRange<R>::n))) q = quot(a, p.den);
    return q;
}
__device__ __forceinline__ cf quot_prepared(cf a, cf d, const Prep<cf>& p, bool on) {
    const float re = __fmaf_rn(a.re, d.re, __fmul_rn(a.im, d.im)), im = __fmaf_rn(a.im, d.re, -__fmul_rn(a.re, d.im));
    cf q{div_prepared(re, p), div_prepared(im, p)};
    if (on && (p.y == 0.f || !within(re, DivRange<float>::n) || !within(im, DivRange<float>::n))) q = quot(a, d);
    return q;
}
__device__ __forceinline__ cd quot_prepared(cd a, cd d, const Prep<cd>& p, bool on) {
    const double re = __fma_rn(a.re, d.re, __dmul_rn(a.im, d.im)), im = __fma_rn(a.im, d.re, -__dmul_rn(a.re, d.im));
    cd q{div_prepared(re, p), div_prepared(im, p)};
    if (on && (p.y == 0.0 || !within(re, DivRange<double>::n) || !within(im, DivRange<double>::n))) q = quot(a, d);
    return q;
}

// One named barrier (1..15) behind each warp.  Seven warps are far enough ahead
// of the chain with their loads and poll L2 half as much as fifteen (lower /
// upper solve, ILU(0) on B200, fifteen -> seven: f64 1024^2 370 / 545, 1296 ->
// 334 / 511, 1228 us; f64 96^3 356 / 349, 814 -> 312 / 340, 772; c128 700^2
// 309 / 560, 2957 -> 275 / 469, 2344; c64 300 x 1000 234 / 408, 1603 -> 254 /
// 387, 1565); eleven 346 / 538 in the first, and five 338 / 373 in the second.
constexpr int kSolveWarps = 7;
constexpr int kSolveThreads = 32 * kSolveWarps;

template <class E>
struct TileValues {
    E xs[kTriTile];                        // the tile's solution by position
    E ext[kSolveWarps][kPre][32];          // each warp's current other-tile values
};

__device__ __forceinline__ void chunk_arrive(int w) {
    asm volatile("bar.arrive %0, 64;" ::"r"(1 + w) : "memory");
}
__device__ __forceinline__ void chunk_sync(int w) {
    asm volatile("bar.sync %0, 64;" ::"r"(1 + w) : "memory");
}

__device__ __forceinline__ int at4(const int4& s, int k) { return k == 0 ? s.x : k == 1 ? s.y : k == 2 ? s.z : s.w; }

// A row as its lane holds it before the warp's turn.
template <class E>
struct RowData {
    int4 d;          // row, first dependency entry, dependency count, diagonal entry
    int4 s;          // dependency sources (dsrc)
    uint32_t starts; // the chunk's level starts
    int first;       // its first position
    E rhs, dg, v[kPre];
};
template <class E>
__device__ __forceinline__ void gather_idx(RowData<E>& r, uint2 chunk, int lane, const int4* __restrict__ desc,
                                           const int4* __restrict__ dsrc) {
    r.first = int(chunk.y & 0xffffu);
    r.starts = chunk.x;
    r.d = make_int4(-1, 0, 0, -1);
    r.s = make_int4(-1, -1, -1, -1);
    if (lane < int(chunk.y >> 16)) {
        r.d = __ldg(desc + r.first + lane);
        r.s = __ldg(dsrc + r.first + lane);
    }
}
// Chunk c of the tile's nc; no positions past the last.
__device__ __forceinline__ uint2 chunk_at(const uint2* __restrict__ chunks, int c, int nc) {
    return c < nc ? __ldg(chunks + 1 + c) : make_uint2(0u, 0u);
}
template <class E, bool UNIT>
__device__ __forceinline__ void gather_val(RowData<E>& r, const E* __restrict__ val, const E* __restrict__ b) {
    if (r.d.x < 0) return;
    r.rhs = ldE(b, r.d.x);
    if (!UNIT) r.dg = ldE(val, r.d.w);
#pragma unroll
    for (int k = 0; k < kPre; ++k)
        if (k < r.d.z) r.v[k] = ldE(val, int64_t(r.d.y) + k);
}

// The chain of one chunk whose rows have at most ND dependencies: `steps`
// levels, this lane's row in level `mine` (0: no row).  The turn is taken and
// handed on in here, with nothing but the levels between: with the choice of
// ND after the turn was taken, and the last level's values published before it
// was handed on, a chunk took 100 cycles longer (lower / upper solve of one
// tile of 1024 x 8 points 103 / 192 us, 82 / 160 as it is).  Every lane computes
// in every step and only the level's lanes store, so a step has no divergent
// branch: a lane's term past its own count has a zero value and a source that
// holds a value already (complex: it is left out, since adding +0 to -0 would
// change the sign of a zero).
template <class E, bool UNIT, int ND>
__device__ __forceinline__ void solve_steps(const RowData<E>& r, const Prep<E>& prep, const E* const (&src)[kPre], E* out,
                                            int steps, int mine, bool publish, E* xo, int from, int to) {
    __syncwarp();
    if (from >= 0) chunk_sync(from);  // the chunks before this one are complete
#pragma unroll 1
    for (int l = 1; l <= steps; ++l) {
        const bool on = mine == l;
        E xj[ND > 0 ? ND : 1];
#pragma unroll
        for (int k = 0; k < ND; ++k) xj[k] = *src[k];
        E acc = r.rhs;
#pragma unroll
        for (int k = 0; k < ND; ++k) {
            const E f = fms(acc, r.v[k], xj[k]);
            acc = (!is_cplx<E>::value || k < r.d.z) ? f : acc;
        }
        if (!UNIT) acc = quot_prepared(acc, r.dg, prep, on);
        if (on) *out = acc;
        __syncwarp();
        if (l == steps && to >= 0) chunk_arrive(to);  // the next chunk goes first
        if (on && publish) Pub<E>::store(xo, 0, acc);
    }
}

// The chain of one chunk in which rows have more than kPre dependencies: the
// sources and values of the next kMore, and other tiles' values, are taken in
// before the turn.  (Looked up during it -- column, position, value one after
// another, other tiles' rows one by one from L2 -- they were most of a solve:
// lower / upper, ILU(0) on B200, f64 27-point 64^3 4964 / 5347 -> 932 / 1067 us,
// 13-point 500^2 2022 / 2785 -> 1085 / 1231, f32 27-point 64^3 3500 / 4103 ->
// 705 / 905.)
// A function of its own: inside the kernel it cost the rows of at most kPre
// dependencies 3 % of the lower solve (321 -> 330 us at 1024^2).
template <class E, bool UNIT>
__device__ __noinline__ void long_rows(RowData<E> r, Prep<E> prep, int w, int lane, int steps, int mine, bool publish,
                                       int from, int to, int32_t base, int32_t m, const int32_t* __restrict__ ci,
                                       const uint16_t* __restrict__ pos, const E* __restrict__ val, E* x, int* err,
                                       unsigned long long lim) {
    extern __shared__ __align__(16) unsigned char smraw[];
    TileValues<E>& T = *reinterpret_cast<TileValues<E>*>(smraw);
    const E* src[kPre];
#pragma unroll
    for (int k = 0; k < kPre; ++k) {
        const int sk = at4(r.s, k);
        src[k] = sk >= 0 ? T.xs + sk : &T.ext[w][k][lane];
    }
    int ms[kMore];
    E mv[kMore], mx[kMore];
#pragma unroll
    for (int k = 0; k < kMore; ++k) {
        ms[k] = -1;
        if (kPre + k < r.d.z) {
            const int32_t e = r.d.y + kPre + k, j = __ldg(ci + e), jl = j - base;
            mv[k] = ldE(val, e);
            if (jl >= 0 && jl < m)
                ms[k] = __ldg(pos + j);
            else
                mx[k] = Pub<E>::load(x, j);
        }
    }
#pragma unroll
    for (int k = 0; k < kMore; ++k)
        if (kPre + k < r.d.z && ms[k] < 0 && Pub<E>::pending(mx[k]))
            mx[k] = await_value(x, __ldg(ci + (r.d.y + kPre + k)), mx[k], err, lim);
    __syncwarp();
    if (from >= 0) chunk_sync(from);
    for (int l = 1; l <= steps; ++l) {
        if (mine == l) {
            E acc = r.rhs;
#pragma unroll
            for (int k = 0; k < kPre; ++k)
                if (k < r.d.z) acc = fms(acc, r.v[k], *src[k]);
#pragma unroll
            for (int k = 0; k < kMore; ++k)
                if (kPre + k < r.d.z) acc = fms(acc, mv[k], ms[k] >= 0 ? T.xs[ms[k]] : mx[k]);
            for (int32_t e = r.d.y + kPre + kMore; e < r.d.y + r.d.z; ++e) {
                const int32_t j = __ldg(ci + e), jl = j - base;
                const E xv = (jl >= 0 && jl < m) ? T.xs[__ldg(pos + j)]
                                                 : await_value(x, j, Pub<E>::load(x, j), err, lim);
                acc = fms(acc, ldE(val, e), xv);
            }
            if (!UNIT) acc = quot_prepared(acc, r.dg, prep, true);
            T.xs[r.first + lane] = acc;
            if (publish) Pub<E>::store(x, r.d.x, acc);
        }
        __syncwarp();
    }
    if (to >= 0) chunk_arrive(to);
}

template <class E, bool UPPER, bool UNIT>
__global__ void __launch_bounds__(kSolveThreads, 1)
k_trsv(int32_t n, int32_t ntiles, const int4* __restrict__ desc, const int4* __restrict__ dsrc,
       const uint2* __restrict__ chunks, const uint16_t* __restrict__ pos, const int32_t* __restrict__ ci,
       const E* __restrict__ val, E alpha, const E* __restrict__ b, E* x, unsigned* ticket, int* err,
       unsigned long long lim, int32_t withhold) {
    extern __shared__ __align__(16) unsigned char smraw[];
    TileValues<E>& T = *reinterpret_cast<TileValues<E>*>(smraw);
    __shared__ int s_tile;
    if (threadIdx.x == 0) {
        const int tk = int(atomicAdd(ticket, 1u));
        s_tile = UPPER ? ntiles - 1 - tk : tk;
    }
    __syncthreads();
    const int t = s_tile;
    if (t < 0 || t >= ntiles) return;
    const int32_t base = int32_t(t) * kTriTile;
    const int32_t m = min(kTriTile, n - base);
    chunks += size_t(t) * (kTriChunkCap + 1);
    const int nc = int(__ldg(&chunks->x));
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    desc += base;
    dsrc += base;

    RowData<E> r{}, nx{};
    gather_idx(r, chunk_at(chunks, w, nc), lane, desc, dsrc);
    gather_idx(nx, chunk_at(chunks, w + kSolveWarps, nc), lane, desc, dsrc);
    uint2 ahead = chunk_at(chunks, w + 2 * kSolveWarps, nc);
    gather_val<E, UNIT>(r, val, b);
    for (int c = w; c < nc; c += kSolveWarps) {
        // in flight meanwhile: the next chunk's values, the descriptors of the one after it
        RowData<E> nn{};
        gather_val<E, UNIT>(nx, val, b);
        gather_idx(nn, ahead, lane, desc, dsrc);
        ahead = chunk_at(chunks, c + 3 * kSolveWarps, nc);
        // sources in shared memory: the tile's own positions, or (another
        // tile's value; a zero where there is no dependency) the warp's own places
        const E* src[kPre];
        unsigned pend = 0;
#pragma unroll
        for (int k = 0; k < kPre; ++k) {
            const int sk = at4(r.s, k);
            src[k] = sk >= 0 ? T.xs + sk : &T.ext[w][k][lane];
            if (sk == -1) T.ext[w][k][lane] = E{};
            if (sk <= -2) pend |= 1u << k;
            if (k >= r.d.z) r.v[k] = E{};
        }
        r.rhs = scale(alpha, r.rhs);
        const Prep<E> prep = UNIT ? Prep<E>{} : prepare_div(r.dg);
        const uint32_t starts = r.starts | 1u;
        const int steps = __popc(starts);
        const int mine = r.d.x >= 0 ? __popc(starts & ((2u << lane) - 1u)) : 0;  // this lane's level within the chunk
        const int most = __reduce_max_sync(0xffffffffu, r.d.z);
        const bool publish = r.d.x != withhold;
        E* const out = T.xs + r.first + lane;
        E* const xo = x + (r.d.x >= 0 ? r.d.x : 0);
        // the other tiles' values, last: nothing but the turn comes after their arrival
        if (pend != 0u) {
            Waiter wt(lim);
            for (;;) {
                E xe[kPre];
#pragma unroll
                for (int k = 0; k < kPre; ++k)
                    if ((pend >> k) & 1u) xe[k] = Pub<E>::load(x, -at4(r.s, k) - 2);
                const bool stop = wt.check(err, 63);  // the values go in as they are then
#pragma unroll
                for (int k = 0; k < kPre; ++k)
                    if (((pend >> k) & 1u) && (stop || !Pub<E>::pending(xe[k]))) {
                        T.ext[w][k][lane] = xe[k];
                        pend &= ~(1u << k);
                    }
                if (pend == 0u) break;
            }
        }
        const int from = c > 0 ? (w == 0 ? kSolveWarps - 1 : w - 1) : -1, to = c + 1 < nc ? w : -1;
        switch (most) {
            case 0: solve_steps<E, UNIT, 0>(r, prep, src, out, steps, mine, publish, xo, from, to); break;
            case 1: solve_steps<E, UNIT, 1>(r, prep, src, out, steps, mine, publish, xo, from, to); break;
            case 2: solve_steps<E, UNIT, 2>(r, prep, src, out, steps, mine, publish, xo, from, to); break;
            case 3: solve_steps<E, UNIT, 3>(r, prep, src, out, steps, mine, publish, xo, from, to); break;
            case 4: solve_steps<E, UNIT, 4>(r, prep, src, out, steps, mine, publish, xo, from, to); break;
            default:  // rows with more than kPre dependencies among them
                long_rows<E, UNIT>(r, prep, w, lane, steps, mine, publish, from, to, base, m, ci, pos, val, x, err, lim);
        }
        r = nx;
        nx = nn;
    }
}

// ---- approximate solves: Jacobi sweeps ------------------------------------
// x_{k+1} = D^-1 (alpha b - (T - D) x_k), x_0 = 0 (so the first pass forms
// D^-1 alpha b; D = I for a unit diagonal): one pass per kernel, one thread
// per row over the row's triangle in index order.  Bandwidth-bound passes
// instead of the exact solve's chain of levels; the result approaches
// T^-1 alpha b as the sweeps grow (exact after as many sweeps as the
// triangle's depth).
template <class E, bool UPPER, bool UNIT, bool FIRST>
__global__ void __launch_bounds__(256)
k_tri_sweep(int32_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
            const int32_t* __restrict__ dpos, const E* __restrict__ val, E alpha, const E* __restrict__ b,
            const E* __restrict__ xin, E* __restrict__ xout) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        E acc = scale(alpha, ldE(b, i));
        const int32_t dp = __ldg(dpos + i);
        if (!FIRST) {
            const int32_t b0 = __ldg(rp + i), b1 = __ldg(rp + i + 1);
            int32_t e0, e1;
            if (dp >= 0) {
                e0 = UPPER ? dp + 1 : b0;
                e1 = UPPER ? b1 : dp;
            } else {  // no stored diagonal (unit solves only): locate the triangle by column
                e0 = b0;
                while (e0 < b1 && __ldg(ci + e0) < i) ++e0;
                if (UPPER) {
                    e1 = b1;
                } else {
                    e1 = e0;
                    e0 = b0;
                }
            }
            for (int32_t e = e0; e < e1; ++e) acc = fms(acc, ldE(val, e), ldE(xin, __ldg(ci + e)));
        }
        if (!UNIT) acc = quot(acc, ldE(val, dp));
        stE(xout, i, acc);
    }
}

// ---- ILU(0), diagonal updates only ----------------------------------------
// Where no entry of row i beside its diagonal lies in the pattern of a row k
// it eliminates (a graph without triangles, as that of every 5- and 7-point
// stencil), eliminating k from row i changes a_ii alone:
//     l_ik = a_ik / d_k,   d_i = a_ii - sum_k l_ik a_ki  (k ascending),
// with a_ik, a_ki still the matrix' own values.  The factorization is then a
// recurrence in one value per row, run like a triangular solve: the same
// chunks of the level order, d by position in shared memory and published
// once to a sentinel-filled array for the other tiles.  The operations are
// those of the general kernel (k_ilu0) in the same order, so the same bits.
// Measured on B200 (f64, 1024^2 5-point operator): 1.22 ms with its pattern
// check, against 15.6 ms for the general kernel, whose every level (7.6 us) is a chain of
// dependent loads from L2 and fences.
// k_ilu0_pattern finds for each of a row's first kPre dependencies where row
// k holds column i (wpos, in level order; -1: nowhere) and sets *general if
// the matrix is not of that kind or a row has more dependencies.
__global__ void k_ilu0_pattern(int32_t n, const int4* __restrict__ desc, const int32_t* __restrict__ rp,
                               const int32_t* __restrict__ ci, const int32_t* __restrict__ dpos,
                               int4* __restrict__ wpos, int* general) {
    const int32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int4 d = desc[p];
    int w[kPre] = {-1, -1, -1, -1};
    bool gen = d.z > kPre;
    const int32_t end = __ldg(rp + d.x + 1);
#pragma unroll
    for (int q = 0; q < kPre; ++q) {
        if (q >= d.z || gen) continue;
        const int32_t k = __ldg(ci + d.y + q);
        int32_t a = d.y + q + 1, b = __ldg(dpos + k) + 1;
        const int32_t bend = __ldg(rp + k + 1);
        while (a < end && b < bend) {  // the common columns past k
            const int32_t ca = __ldg(ci + a), cb = __ldg(ci + b);
            if (ca == cb) {
                if (ca == d.x)
                    w[q] = b;
                else
                    gen = true;
                ++a;
                ++b;
            } else if (ca < cb) {
                ++a;
            } else {
                ++b;
            }
        }
    }
    wpos[p] = make_int4(w[0], w[1], w[2], w[3]);
    if (gen) *general = 1;
}

// A diagonal value that happens to be the sentinel (only a signalling NaN in
// the input can be) is published as a quiet one.
__device__ __forceinline__ double publishable(double v) {
    return Pub<double>::pending(v) ? __longlong_as_double(0x7FF8000000000000ll) : v;
}
__device__ __forceinline__ float publishable(float v) { return Pub<float>::pending(v) ? __int_as_float(0x7FC00000) : v; }
template <class C>
__device__ __forceinline__ C publishable(C v) { return C{publishable(v.re), publishable(v.im)}; }
template <class E> __device__ __forceinline__ E one_of();
template <> __device__ __forceinline__ float one_of<float>() { return 1.f; }
template <> __device__ __forceinline__ double one_of<double>() { return 1.0; }
template <> __device__ __forceinline__ cf one_of<cf>() { return cf{1.f, 0.f}; }
template <> __device__ __forceinline__ cd one_of<cd>() { return cd{1.0, 0.0}; }

template <class E>
struct PivotRow {
    int4 d, s, w;
    uint32_t starts;
    int first;
    E diag, v[kPre], u[kPre];  // a_ii, a_ik, a_ki
};

template <class E>
__global__ void __launch_bounds__(kSolveThreads, 1)
k_ilu0_diag(int32_t n, int32_t ntiles, const int4* __restrict__ desc, const int4* __restrict__ dsrc,
            const uint2* __restrict__ chunks, const int4* __restrict__ wpos, E* val, E* piv, unsigned* ticket,
            const int* __restrict__ general, int* err, int* err_row) {
    if (*general) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    TileValues<E>& T = *reinterpret_cast<TileValues<E>*>(smraw);
    __shared__ int s_tile;
    if (threadIdx.x == 0) s_tile = int(atomicAdd(ticket, 1u));
    __syncthreads();
    const int t = s_tile;
    if (t >= ntiles) return;
    const int32_t base = int32_t(t) * kTriTile;
    chunks += size_t(t) * (kTriChunkCap + 1);
    const int nc = int(__ldg(&chunks->x));
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    desc += base;
    dsrc += base;
    wpos += base;

    auto idx = [&](PivotRow<E>& r, uint2 chunk) {
        const int32_t p = int32_t(chunk.y & 0xffffu) + lane;
        r.first = p - lane;
        r.d = make_int4(-1, 0, 0, -1);
        r.s = make_int4(-1, -1, -1, -1);
        r.w = r.s;
        r.starts = chunk.x;
        if (lane < int(chunk.y >> 16)) {
            r.d = __ldg(desc + p);
            r.s = __ldg(dsrc + p);
            r.w = __ldg(wpos + p);
        }
    };
    // (the entries read here are written by their own row's lane alone, later)
    auto values = [&](PivotRow<E>& r) {
        if (r.d.x < 0) return;
        r.diag = ldE(val, r.d.w);
#pragma unroll
        for (int k = 0; k < kPre; ++k)
            if (k < r.d.z) {
                r.v[k] = ldE(val, int64_t(r.d.y) + k);
                if (at4(r.w, k) >= 0) r.u[k] = ldE(val, at4(r.w, k));
            }
    };
    PivotRow<E> r{}, nx{};
    idx(r, chunk_at(chunks, w, nc));
    idx(nx, chunk_at(chunks, w + kSolveWarps, nc));
    uint2 ahead = chunk_at(chunks, w + 2 * kSolveWarps, nc);
    values(r);
    for (int c = w; c < nc; c += kSolveWarps) {
        // in flight meanwhile (complex<double> rows fill the registers as they are: its next values come after the turn)
        constexpr bool kAhead = sizeof(E) < 16;
        PivotRow<E> nn{};
        if (kAhead) values(nx);
        idx(nn, ahead);
        ahead = chunk_at(chunks, c + 3 * kSolveWarps, nc);
        const E* src[kPre];
        unsigned pend = 0;
#pragma unroll
        for (int k = 0; k < kPre; ++k) {
            const int sk = at4(r.s, k);
            src[k] = sk >= 0 ? T.xs + sk : &T.ext[w][k][lane];
            if (sk == -1) T.ext[w][k][lane] = one_of<E>();
            if (sk <= -2) pend |= 1u << k;
        }
        const uint32_t starts = r.starts | 1u;
        const int steps = __popc(starts);
        const int mine = r.d.x >= 0 ? __popc(starts & ((2u << lane) - 1u)) : 0;
        const int most = __reduce_max_sync(0xffffffffu, r.d.z);
        if (pend != 0u) {
            Waiter wt;
            for (;;) {
                E xe[kPre];
#pragma unroll
                for (int k = 0; k < kPre; ++k)
                    if ((pend >> k) & 1u) xe[k] = Pub<E>::load(piv, -at4(r.s, k) - 2);
                const bool stop = wt.check(err, 63);
#pragma unroll
                for (int k = 0; k < kPre; ++k)
                    if (((pend >> k) & 1u) && (stop || !Pub<E>::pending(xe[k]))) {
                        T.ext[w][k][lane] = xe[k];
                        pend &= ~(1u << k);
                    }
                if (pend == 0u) break;
            }
        }
        __syncwarp();
        if (c > 0) chunk_sync(w == 0 ? kSolveWarps - 1 : w - 1);
        E piv_i{}, l[kPre];
#pragma unroll 1
        for (int s = 1; s <= steps; ++s) {
            const bool on = mine == s;
            E acc = r.diag, q[kPre];
#pragma unroll
            for (int k = 0; k < kPre; ++k)
                if (k < most) {  // the same for the whole warp
                    // lanes that are not at this level divide 1 by 1: no slow path for what they hold
                    const bool has = on && k < r.d.z;
                    q[k] = quot(has ? r.v[k] : one_of<E>(), has ? *src[k] : one_of<E>());
                }
#pragma unroll
            for (int k = 0; k < kPre; ++k)
                if (k < most) {
                    const E f = fms(acc, q[k], r.u[k]);
                    acc = (k < r.d.z && at4(r.w, k) >= 0) ? f : acc;
                }
            if (on) {
                T.xs[r.first + lane] = acc;
                piv_i = acc;
#pragma unroll
                for (int k = 0; k < kPre; ++k) l[k] = q[k];
            }
            __syncwarp();
            if (on) Pub<E>::store(piv, r.d.x, publishable(acc));
        }
        __syncwarp();
        if (c + 1 < nc) chunk_arrive(w);
        if (r.d.x >= 0) {
            stE(val, r.d.w, piv_i);
#pragma unroll
            for (int k = 0; k < kPre; ++k)
                if (k < r.d.z) stE(val, int64_t(r.d.y) + k, l[k]);
            if (zero_of(piv_i)) {
                atomicOr(err, kErrZeroPivot);
                atomicMin(err_row, r.d.x);
            }
        }
        if (!kAhead) values(nx);
        r = nx;
        nx = nn;
    }
}

// ---- ILU(0), general ------------------------------------------------------
// Row i, for each strictly lower entry k (ascending): l_ik = a_ik / u_kk,
// then a_ij -= l_ik u_kj for every j > k present in both rows (the IKJ
// variant of ILU(0), Saad, Iterative Methods for Sparse Linear Systems,
// 2nd ed., Algorithm 10.4).  Rows k are complete when read: earlier levels
// of the tile (level counter) or other tiles (row flags).  All accesses to
// val go to L2 (ld.cg / st.cg): rows finished by other warps and blocks are
// read there, and no L1 line of a neighbouring row can go stale.
template <class E>
__global__ void __launch_bounds__(kTriThreads)
k_ilu0(int32_t n, int32_t ntiles, const int4* __restrict__ desc, const int32_t* __restrict__ lvlptr,
       const int32_t* __restrict__ nlev, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
       const int32_t* __restrict__ dpos, E* val, unsigned* flags, const int* __restrict__ general, int* err,
       int* err_row) {
    if (general != nullptr && !*general) return;  // k_ilu0_diag has done it
    __shared__ int s_tile;
    __shared__ int s_done;
    if (threadIdx.x == 0) {
        s_tile = int(atomicAdd(flags + n, 1u));
        s_done = 0;
    }
    __syncthreads();
    const int t = s_tile;
    if (t < 0 || t >= ntiles) return;
    const int32_t base = int32_t(t) * kTriTile;
    const int32_t m = min(kTriTile, n - base);
    const int L = nlev[t];
    const int32_t* lp = lvlptr + size_t(t) * (kTriTile + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int W = kTriThreads / 32;
    volatile int* done = &s_done;
    for (int l = warp; l < L; l += W) {
        const int32_t p0 = lp[l], p1 = lp[l + 1];
        wait_levels(done, l, lane, err);
        for (int32_t q = p0; q < p1; q += 32) {
            const int32_t p = q + lane;
            if (p >= p1) continue;
            const int4 d = desc[base + p];
            const int32_t i = d.x, e_end = __ldg(rp + i + 1);
            for (int32_t e = d.y; e < d.y + d.z; ++e) {
                const int32_t k = __ldg(ci + e);
                const int32_t kl = k - base;
                if (!(kl >= 0 && kl < m)) wait_row(flags, k, err);
                const int32_t dk = __ldg(dpos + k);
                const E lik = quot(ldcgE(val, e), ldcgE(val, dk));
                stcgE(val, e, lik);
                // Merge the columns after e in row i with those after the
                // diagonal in row k; the matching pairs are collected first
                // (columns only, read-only path) and their values then loaded
                // as one batch, so a batch costs one L2 round trip.
                int32_t pi = e + 1, pk = dk + 1;
                const int32_t pk_end = __ldg(rp + k + 1);
                for (;;) {
                    int32_t P[kMerge], Q[kMerge];
                    int np = 0;
                    while (np < kMerge && pi < e_end && pk < pk_end) {
                        const int32_t ca = __ldg(ci + pi), cb = __ldg(ci + pk);
                        if (ca == cb) {
                            P[np] = pi++;
                            Q[np++] = pk++;
                        } else if (ca < cb) {
                            ++pi;
                        } else {
                            ++pk;
                        }
                    }
                    E a[kMerge], u[kMerge];
#pragma unroll
                    for (int j = 0; j < kMerge; ++j)
                        if (j < np) {
                            a[j] = ldcgE(val, P[j]);
                            u[j] = ldcgE(val, Q[j]);
                        }
#pragma unroll
                    for (int j = 0; j < kMerge; ++j)
                        if (j < np) stcgE(val, P[j], fms(a[j], lik, u[j]));
                    if (np < kMerge) break;
                }
            }
            if (zero_of(ldcgE(val, d.w))) {
                atomicOr(err, kErrZeroPivot);
                atomicMin(err_row, i);
            }
            __threadfence();
            st_release(flags + i, 1u);
        }
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            *done = l + 1;
        }
    }
}

template <class K>
void allow_smem(K kernel, size_t bytes) {
    if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
}

}  // namespace

int analyse(hpb_context* ctx, int upper, int32_t n, int64_t nnz, const int32_t* rp, const int32_t* ci, Plan* P) {
    *P = Plan{};
    P->upper = upper ? 1 : 0;
    P->n = n;
    P->nnz = nnz;
    P->rp = rp;
    P->ci = ci;
    P->ntiles = int32_t((int64_t(n) + kTriTile - 1) / kTriTile);
    cudaGetDevice(&P->device);
    cudaStream_t s = ctx->stream;
    // Two allocations from the analyses' pool: what the plan keeps, and the
    // analysis' own work arrays.  The stream is synchronised before they are
    // used or given back elsewhere.
    size_t keep = 0, tmp = 0;
    auto part = [](size_t& total, size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) & ~size_t(255);
        return at;
    };
    const size_t nn = size_t(n), nt = size_t(P->ntiles);
    const size_t o_desc = part(keep, nn * sizeof(int4)), o_dsrc = part(keep, nn * sizeof(int4));
    const size_t o_pos = part(keep, nn * sizeof(uint16_t)), o_chunks = part(keep, nt * (kTriChunkCap + 1) * sizeof(uint2));
    const size_t o_lvl = part(keep, nt * (kTriTile + 1) * sizeof(int32_t)), o_dpos = part(keep, nn * sizeof(int32_t));
    const size_t o_flags = part(keep, (nn + 1) * sizeof(unsigned));
    const size_t o_err = part(keep, (4 + nt) * sizeof(int));  // err, err_row, rows without a diagonal, -, nlev
    const size_t o_beg = part(tmp, nn * sizeof(int32_t)), o_cnt = part(tmp, nn * sizeof(int32_t));
    const size_t o_glev = part(tmp, nn * sizeof(int32_t)), o_tick = part(tmp, sizeof(unsigned));
    char* work = nullptr;
    auto fail = [&](int status, const char* what) {
        cudaStreamSynchronize(s);
        fused::analysis_free(work, s);
        release(P);
        return set_error(ctx, status, "hpb_csr_tri_create: %s", what);
    };
    P->block = fused::analysis_alloc(keep, s);
    work = static_cast<char*>(fused::analysis_alloc(tmp, s));
    if (P->block == nullptr || work == nullptr) return fail(HPB_ERROR_OUT_OF_MEMORY, "device allocation failed");
    char* blk = static_cast<char*>(P->block);
    P->desc = reinterpret_cast<int4*>(blk + o_desc);
    P->dsrc = reinterpret_cast<int4*>(blk + o_dsrc);
    P->pos = reinterpret_cast<uint16_t*>(blk + o_pos);
    P->chunks = reinterpret_cast<uint2*>(blk + o_chunks);
    P->lvlptr = reinterpret_cast<int32_t*>(blk + o_lvl);
    P->dpos = reinterpret_cast<int32_t*>(blk + o_dpos);
    P->flags = reinterpret_cast<unsigned*>(blk + o_flags);
    P->err = reinterpret_cast<int*>(blk + o_err);
    P->err_row = P->err + 1;
    P->nlev = P->err + 4;
    int* missing = P->err + 2;
    int32_t* beg = reinterpret_cast<int32_t*>(work + o_beg);
    int32_t* cnt = reinterpret_cast<int32_t*>(work + o_cnt);
    int32_t* glev = reinterpret_cast<int32_t*>(work + o_glev);
    unsigned* ticket = reinterpret_cast<unsigned*>(work + o_tick);
    const int init[4] = {0, INT_MAX, 0, 0};
    cudaMemcpyAsync(P->err, init, sizeof(init), cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(glev, 0xFF, nn * sizeof(int32_t), s);
    cudaMemsetAsync(ticket, 0, sizeof(unsigned), s);
    k_tri_rows<<<(n + 255) / 256, 256, 0, s>>>(n, nnz, P->upper, rp, ci, beg, cnt, P->dpos, P->err, missing);
    auto levels = P->upper ? k_tri_levels<true> : k_tri_levels<false>;
    allow_smem(levels, sizeof(LevelTile));
    levels<<<P->ntiles, kGlThreads, sizeof(LevelTile), s>>>(n, P->ntiles, ci, beg, cnt, glev, ticket, P->err);
    const size_t sort_smem = size_t(kTriTile) * (sizeof(unsigned long long) + 2 * sizeof(uint16_t)) + 16;
    allow_smem(k_tri_sort, sort_smem);
    k_tri_sort<<<P->ntiles, kSortThreads, sort_smem, s>>>(n, ci, beg, cnt, P->dpos, glev, P->desc, P->dsrc, P->pos,
                                                          P->chunks, P->lvlptr, P->nlev);
    count_launch(3);
    if (cudaGetLastError() != cudaSuccess) return fail(HPB_ERROR_CUDA, "analysis launch failed");
    std::vector<int32_t> got(4 + nt);  // err, err_row, missing, -, nlev
    if (cudaMemcpyAsync(got.data(), P->err, got.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return fail(HPB_ERROR_CUDA, "analysis failed");
    if (got[0] & kErrColumn) return fail(HPB_ERROR_INVALID_VALUE, "row pointer or column index out of range");
    if (got[0] & kErrUnsorted)
        return fail(HPB_ERROR_INVALID_VALUE, "column indices of a row are not strictly increasing");
    if (got[0] & kErrTimeout) return fail(HPB_ERROR_TIMEOUT, "a bounded device-side wait gave up");
    fused::analysis_free(work, s);
    P->all_diag = got[2] == 0;
    for (size_t t = 0; t < nt; ++t) {
        P->max_levels = std::max(P->max_levels, got[4 + t]);
        P->sum_levels += got[4 + t];
    }
    return HPB_SUCCESS;
}

// As cudaFree would, this waits for the device: solves with the analysis may
// still be running on any stream.
void release(Plan* P) {
    int dev = 0;
    const bool other = cudaGetDevice(&dev) == cudaSuccess && dev != P->device;
    if (other) cudaSetDevice(P->device);
    if (P->block != nullptr || P->scratch != nullptr) cudaDeviceSynchronize();
    fused::analysis_free(P->block, nullptr);
    cudaFree(P->scratch);
    if (other) cudaSetDevice(dev);
    P->block = P->scratch = nullptr;
    P->desc = P->dsrc = nullptr;
    P->pos = nullptr;
    P->chunks = nullptr;
    P->lvlptr = P->nlev = P->dpos = nullptr;
    P->flags = nullptr;
    P->err = P->err_row = nullptr;
}

template <class E>
cudaError_t launch_trsv(const Plan& P, int unit, const E* val, E alpha, const E* b, E* x, cudaStream_t s) {
    if (P.n == 0) return cudaSuccess;
    const int fill_grid = int(std::min<int64_t>((int64_t(P.n) + 255) / 256, 148 * 8));
    k_tri_fill<E><<<fill_grid, 256, 0, s>>>(P.n, x, P.flags + P.n);
    constexpr size_t sm = sizeof(TileValues<E>);
    static_assert(sm <= 226 * 1024, "shared memory of a tile");
    // the shared-memory limit is a per-device function attribute: raise it
    // once for every device this process launches on
    static std::atomic<uint64_t> done_mask{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return cudaErrorInvalidDevice;
    const uint64_t bit = dev < 64 ? (uint64_t(1) << dev) : 0;
    if (bit == 0 || !(done_mask.load(std::memory_order_acquire) & bit)) {
        allow_smem(k_trsv<E, false, false>, sm);
        allow_smem(k_trsv<E, false, true>, sm);
        allow_smem(k_trsv<E, true, false>, sm);
        allow_smem(k_trsv<E, true, true>, sm);
        done_mask.fetch_or(bit, std::memory_order_release);
    }
    auto k = P.upper ? (unit ? k_trsv<E, true, true> : k_trsv<E, true, false>)
                     : (unit ? k_trsv<E, false, true> : k_trsv<E, false, false>);
    k<<<P.ntiles, kSolveThreads, sm, s>>>(P.n, P.ntiles, P.desc, P.dsrc, P.chunks, P.pos, P.ci, val, alpha, b, x,
                                        P.flags + P.n, P.err, P.wait_ns ? P.wait_ns : kWaitNs, P.withhold_row);
    count_launch(2);
    return cudaGetLastError();
}

template <class E, bool UPPER, bool UNIT>
cudaError_t sweeps_t(const Plan& P, const E* val, E alpha, const E* b, E* x, E* tmp, int sweeps, cudaStream_t s) {
    const int grid = int(std::min<int64_t>((int64_t(P.n) + 255) / 256, 148 * 8));
    const int K = sweeps + 1;  // kernels; the last one writes x
    auto dst = [&](int t) { return ((K - 1 - t) % 2 == 0) ? x : tmp; };
    k_tri_sweep<E, UPPER, UNIT, true><<<grid, 256, 0, s>>>(P.n, P.rp, P.ci, P.dpos, val, alpha, b, nullptr, dst(0));
    for (int t = 1; t < K; ++t)
        k_tri_sweep<E, UPPER, UNIT, false><<<grid, 256, 0, s>>>(P.n, P.rp, P.ci, P.dpos, val, alpha, b, dst(t - 1),
                                                                dst(t));
    count_launch(uint64_t(K));
    return cudaGetLastError();
}

template <class E>
cudaError_t launch_trsv_sweeps(const Plan& P, int unit, const E* val, E alpha, const E* b, E* x, E* tmp, int sweeps,
                               cudaStream_t s) {
    if (P.n == 0) return cudaSuccess;
    if (P.upper) return unit ? sweeps_t<E, true, true>(P, val, alpha, b, x, tmp, sweeps, s)
                             : sweeps_t<E, true, false>(P, val, alpha, b, x, tmp, sweeps, s);
    return unit ? sweeps_t<E, false, true>(P, val, alpha, b, x, tmp, sweeps, s)
                : sweeps_t<E, false, false>(P, val, alpha, b, x, tmp, sweeps, s);
}

template <class E>
cudaError_t launch_ilu0(const Plan& P, E* val, cudaStream_t s) {
    if (P.n == 0) return cudaSuccess;
    // scratch: the published diagonal, the positions of a_ki, the tile ticket and the
    // kind of matrix.  Without memory for it the general kernel, which needs none.
    const size_t o_piv = (size_t(P.n) * sizeof(int4) + 255) & ~size_t(255);
    const size_t o_word = (o_piv + size_t(P.n) * sizeof(E) + 255) & ~size_t(255);
    char* work = static_cast<char*>(fused::analysis_alloc(o_word + 8, s));
    int* general = work ? reinterpret_cast<int*>(work + o_word + 4) : nullptr;
    cudaError_t e = cudaMemsetAsync(P.flags, 0, (size_t(P.n) + 1) * sizeof(unsigned), s);
    if (e == cudaSuccess && work != nullptr) {
        int4* wpos = reinterpret_cast<int4*>(work);
        E* piv = reinterpret_cast<E*>(work + o_piv);
        unsigned* ticket = reinterpret_cast<unsigned*>(work + o_word);
        e = cudaMemsetAsync(general, 0, sizeof(int), s);
        if (e == cudaSuccess) {
            k_ilu0_pattern<<<(P.n + 255) / 256, 256, 0, s>>>(P.n, P.desc, P.rp, P.ci, P.dpos, wpos, general);
            k_tri_fill<E><<<int(std::min<int64_t>((int64_t(P.n) + 255) / 256, 148 * 8)), 256, 0, s>>>(P.n, piv, ticket);
            allow_smem(k_ilu0_diag<E>, sizeof(TileValues<E>));
            k_ilu0_diag<E><<<P.ntiles, kSolveThreads, sizeof(TileValues<E>), s>>>(
                P.n, P.ntiles, P.desc, P.dsrc, P.chunks, wpos, val, piv, ticket, general, P.err, P.err_row);
            count_launch(3);
        }
    }
    if (e == cudaSuccess) {
        k_ilu0<E><<<P.ntiles, kTriThreads, 0, s>>>(P.n, P.ntiles, P.desc, P.lvlptr, P.nlev, P.rp, P.ci, P.dpos, val,
                                                   P.flags, general, P.err, P.err_row);
        count_launch();
        e = cudaGetLastError();
    }
    fused::analysis_free(work, s);
    return e;
}

template cudaError_t launch_trsv<float>(const Plan&, int, const float*, float, const float*, float*, cudaStream_t);
template cudaError_t launch_trsv<double>(const Plan&, int, const double*, double, const double*, double*,
                                         cudaStream_t);
template cudaError_t launch_trsv<cf>(const Plan&, int, const cf*, cf, const cf*, cf*, cudaStream_t);
template cudaError_t launch_trsv<cd>(const Plan&, int, const cd*, cd, const cd*, cd*, cudaStream_t);
template cudaError_t launch_trsv_sweeps<float>(const Plan&, int, const float*, float, const float*, float*, float*,
                                               int, cudaStream_t);
template cudaError_t launch_trsv_sweeps<double>(const Plan&, int, const double*, double, const double*, double*,
                                                double*, int, cudaStream_t);
template cudaError_t launch_trsv_sweeps<cf>(const Plan&, int, const cf*, cf, const cf*, cf*, cf*, int, cudaStream_t);
template cudaError_t launch_trsv_sweeps<cd>(const Plan&, int, const cd*, cd, const cd*, cd*, cd*, int, cudaStream_t);
template cudaError_t launch_ilu0<float>(const Plan&, float*, cudaStream_t);
template cudaError_t launch_ilu0<double>(const Plan&, double*, cudaStream_t);
template cudaError_t launch_ilu0<cf>(const Plan&, cf*, cudaStream_t);
template cudaError_t launch_ilu0<cd>(const Plan&, cd*, cudaStream_t);

}  // namespace tri

namespace {

bool aligned(const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; }

template <class E>
int trsv_impl(hpb_context* ctx, const hpb_csr_tri* tri, int unit, const E* val, E alpha, const E* b, E* x,
              const char* name) {
    HPB_CHECK_CTX(ctx);
    if (tri == nullptr) return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: null analysis", name);
    const tri::Plan& P = tri->plan;
    if (P.n == 0) return HPB_SUCCESS;
    if (val == nullptr || b == nullptr || x == nullptr)
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: null pointer", name);
    constexpr size_t kA = sizeof(typename real_of<E>::type);
    if (!aligned(val, kA) || !aligned(b, kA) || !aligned(x, kA))
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: pointer not aligned to its element type", name);
    if (!unit && !P.all_diag)
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: a row stores no diagonal entry (structural zero)", name);
    const size_t bytes = size_t(P.n) * sizeof(E);
    const char* bb = reinterpret_cast<const char*>(b);
    const char* xb = reinterpret_cast<const char*>(x);
    if (b != x && bb < xb + bytes && xb < bb + bytes)
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: b and x overlap without being equal", name);
    if (b == x) {  // in place: solve into the analysis' scratch, then copy back
        tri::Plan& Pm = const_cast<tri::Plan&>(P);
        if (Pm.scratch == nullptr && cudaMalloc(&Pm.scratch, size_t(P.n) * 16) != cudaSuccess) {
            cudaGetLastError();
            Pm.scratch = nullptr;
            return set_error(ctx, HPB_ERROR_OUT_OF_MEMORY, "%s: in-place scratch allocation failed", name);
        }
        E* tmp = static_cast<E*>(Pm.scratch);
        HPB_CUDA_TRY(ctx, tri::launch_trsv<E>(P, unit, val, alpha, b, tmp, ctx->stream));
        HPB_CUDA_TRY(ctx, cudaMemcpyAsync(x, tmp, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        return HPB_SUCCESS;
    }
    HPB_CUDA_TRY(ctx, tri::launch_trsv<E>(P, unit, val, alpha, b, x, ctx->stream));
    return HPB_SUCCESS;
}

template <class E>
int sweeps_impl(hpb_context* ctx, const hpb_csr_tri* tri, int unit, const E* val, E alpha, const E* b, E* x,
                int sweeps, const char* name) {
    HPB_CHECK_CTX(ctx);
    if (tri == nullptr) return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: null analysis", name);
    const tri::Plan& P = tri->plan;
    if (sweeps < 0) return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: negative sweep count", name);
    if (P.n == 0) return HPB_SUCCESS;
    if (val == nullptr || b == nullptr || x == nullptr)
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: null pointer", name);
    constexpr size_t kA = sizeof(typename real_of<E>::type);
    if (!aligned(val, kA) || !aligned(b, kA) || !aligned(x, kA))
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: pointer not aligned to its element type", name);
    if (!unit && !P.all_diag)
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: a row stores no diagonal entry (structural zero)", name);
    const size_t bytes = size_t(P.n) * sizeof(E);
    const char* bb = reinterpret_cast<const char*>(b);
    const char* xb = reinterpret_cast<const char*>(x);
    if (bb < xb + bytes && xb < bb + bytes)
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: b and x must not overlap", name);
    tri::Plan& Pm = const_cast<tri::Plan&>(P);
    if (Pm.scratch == nullptr && cudaMalloc(&Pm.scratch, size_t(P.n) * 16) != cudaSuccess) {
        cudaGetLastError();
        Pm.scratch = nullptr;
        return set_error(ctx, HPB_ERROR_OUT_OF_MEMORY, "%s: scratch allocation failed", name);
    }
    HPB_CUDA_TRY(ctx, tri::launch_trsv_sweeps<E>(P, unit, val, alpha, b, x, static_cast<E*>(Pm.scratch), sweeps,
                                                 ctx->stream));
    return HPB_SUCCESS;
}

template <class E>
int ilu0_impl(hpb_context* ctx, const hpb_csr_tri* tri, E* val, const char* name) {
    HPB_CHECK_CTX(ctx);
    if (tri == nullptr) return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: null analysis", name);
    const tri::Plan& P = tri->plan;
    if (P.upper) return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: needs the analysis of the lower triangle", name);
    if (P.n == 0) return HPB_SUCCESS;
    if (val == nullptr) return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: null pointer", name);
    if (!aligned(val, sizeof(typename real_of<E>::type)))
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: pointer not aligned to its element type", name);
    if (!P.all_diag)
        return set_error(ctx, HPB_ERROR_INVALID_VALUE, "%s: a row stores no diagonal entry (structural zero)", name);
    const int init[2] = {0, INT_MAX};
    HPB_CUDA_TRY(ctx, cudaMemcpyAsync(P.err, init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
    HPB_CUDA_TRY(ctx, tri::launch_ilu0<E>(P, val, ctx->stream));
    int h[2] = {0, 0};
    HPB_CUDA_TRY(ctx, cudaMemcpyAsync(h, P.err, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    HPB_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    if (h[0] & tri::kErrTimeout)
        return set_error(ctx, HPB_ERROR_TIMEOUT, "%s: a bounded device-side wait gave up", name);
    if (h[0] & tri::kErrZeroPivot) return set_error(ctx, HPB_ERROR_BREAKDOWN, "%s: zero pivot in row %d", name, h[1]);
    return HPB_SUCCESS;
}

}  // namespace
}  // namespace hpb

using hpb::cd;
using hpb::cf;

extern "C" {

int hpb_csr_tri_create(hpb_context* ctx, int upper, int32_t rows, int64_t nnz, const int32_t* row_ptr,
                       const int32_t* col_ind, hpb_csr_tri** tri) {
    HPB_CHECK_CTX(ctx);
    if (tri == nullptr) return hpb::set_error(ctx, HPB_ERROR_INVALID_VALUE, "hpb_csr_tri_create: null output");
    *tri = nullptr;
    if (rows < 0 || nnz < 0 || nnz > INT32_MAX)
        return hpb::set_error(ctx, HPB_ERROR_INVALID_VALUE, "hpb_csr_tri_create: invalid dimensions");
    if (rows > 0 && (row_ptr == nullptr || (nnz > 0 && col_ind == nullptr)))
        return hpb::set_error(ctx, HPB_ERROR_INVALID_VALUE, "hpb_csr_tri_create: null pointer");
    auto* h = new (std::nothrow) hpb_csr_tri;
    if (h == nullptr) return hpb::set_error(ctx, HPB_ERROR_OUT_OF_MEMORY, "hpb_csr_tri_create: host allocation");
    if (rows == 0) {
        h->plan = hpb::tri::Plan{};
        h->plan.upper = upper ? 1 : 0;
        h->plan.all_diag = 1;
        *tri = h;
        return HPB_SUCCESS;
    }
    const int st = hpb::tri::analyse(ctx, upper, rows, nnz, row_ptr, col_ind, &h->plan);
    if (st != HPB_SUCCESS) {
        delete h;
        return st;
    }
    *tri = h;
    return HPB_SUCCESS;
}

int hpb_csr_tri_destroy(hpb_csr_tri* tri) {
    if (tri == nullptr) return HPB_SUCCESS;
    hpb::tri::release(&tri->plan);
    delete tri;
    return HPB_SUCCESS;
}

int hpb_csr_tri_info(const hpb_csr_tri* tri, int32_t* tiles, int32_t* max_levels, int64_t* sum_levels,
                     int* has_diagonal) {
    if (tri == nullptr) return HPB_ERROR_INVALID_VALUE;
    if (tiles) *tiles = tri->plan.ntiles;
    if (max_levels) *max_levels = tri->plan.max_levels;
    if (sum_levels) *sum_levels = tri->plan.sum_levels;
    if (has_diagonal) *has_diagonal = tri->plan.all_diag;
    return HPB_SUCCESS;
}

int hpb_csr_tri_check(hpb_context* ctx, const hpb_csr_tri* tri) {
    HPB_CHECK_CTX(ctx);
    if (tri == nullptr) return hpb::set_error(ctx, HPB_ERROR_INVALID_VALUE, "hpb_csr_tri_check: null analysis");
    if (tri->plan.err == nullptr) return HPB_SUCCESS;
    int h = 0;
    HPB_CUDA_TRY(ctx, cudaMemcpyAsync(&h, tri->plan.err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    HPB_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    if (h & hpb::tri::kErrTimeout) {
        // reported once: the word is cleared for the solves that follow
        HPB_CUDA_TRY(ctx, cudaMemsetAsync(tri->plan.err, 0, sizeof(int), ctx->stream));
        HPB_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        return hpb::set_error(ctx, HPB_ERROR_TIMEOUT, "hpb_csr_tri_check: a bounded device-side wait gave up");
    }
    return HPB_SUCCESS;
}

int hpb_csr_tri_set_wait_limit(hpb_csr_tri* tri, uint64_t ns) {
    if (tri == nullptr) return HPB_ERROR_INVALID_VALUE;
    tri->plan.wait_ns = ns;
    return HPB_SUCCESS;
}

int hpb_csr_tri_test_withhold_row(hpb_csr_tri* tri, int32_t row) {
    if (tri == nullptr || row < -1 || row >= tri->plan.n) return HPB_ERROR_INVALID_VALUE;
    tri->plan.withhold_row = row;
    return HPB_SUCCESS;
}

int hpb_csr_trsv_f32(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const float* val, float alpha,
                     const float* b, float* x) {
    return hpb::trsv_impl<float>(ctx, tri, unit_diag, val, alpha, b, x, "hpb_csr_trsv_f32");
}
int hpb_csr_trsv_f64(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const double* val, double alpha,
                     const double* b, double* x) {
    return hpb::trsv_impl<double>(ctx, tri, unit_diag, val, alpha, b, x, "hpb_csr_trsv_f64");
}
int hpb_csr_trsv_c64(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const void* val, hpb_c64 alpha,
                     const void* b, void* x) {
    return hpb::trsv_impl<cf>(ctx, tri, unit_diag, static_cast<const cf*>(val), cf{alpha.re, alpha.im},
                              static_cast<const cf*>(b), static_cast<cf*>(x), "hpb_csr_trsv_c64");
}
int hpb_csr_trsv_c128(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const void* val, hpb_c128 alpha,
                      const void* b, void* x) {
    return hpb::trsv_impl<cd>(ctx, tri, unit_diag, static_cast<const cd*>(val), cd{alpha.re, alpha.im},
                              static_cast<const cd*>(b), static_cast<cd*>(x), "hpb_csr_trsv_c128");
}

int hpb_csr_trsv_sweeps_f32(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const float* val, float alpha,
                            const float* b, float* x, int sweeps) {
    return hpb::sweeps_impl<float>(ctx, tri, unit_diag, val, alpha, b, x, sweeps, "hpb_csr_trsv_sweeps_f32");
}
int hpb_csr_trsv_sweeps_f64(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const double* val,
                            double alpha, const double* b, double* x, int sweeps) {
    return hpb::sweeps_impl<double>(ctx, tri, unit_diag, val, alpha, b, x, sweeps, "hpb_csr_trsv_sweeps_f64");
}
int hpb_csr_trsv_sweeps_c64(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const void* val, hpb_c64 alpha,
                            const void* b, void* x, int sweeps) {
    return hpb::sweeps_impl<cf>(ctx, tri, unit_diag, static_cast<const cf*>(val), cf{alpha.re, alpha.im},
                                static_cast<const cf*>(b), static_cast<cf*>(x), sweeps, "hpb_csr_trsv_sweeps_c64");
}
int hpb_csr_trsv_sweeps_c128(hpb_context* ctx, const hpb_csr_tri* tri, int unit_diag, const void* val,
                             hpb_c128 alpha, const void* b, void* x, int sweeps) {
    return hpb::sweeps_impl<cd>(ctx, tri, unit_diag, static_cast<const cd*>(val), cd{alpha.re, alpha.im},
                                static_cast<const cd*>(b), static_cast<cd*>(x), sweeps, "hpb_csr_trsv_sweeps_c128");
}

int hpb_csr_ilu0_f32(hpb_context* ctx, const hpb_csr_tri* lower, float* val) {
    return hpb::ilu0_impl<float>(ctx, lower, val, "hpb_csr_ilu0_f32");
}
int hpb_csr_ilu0_f64(hpb_context* ctx, const hpb_csr_tri* lower, double* val) {
    return hpb::ilu0_impl<double>(ctx, lower, val, "hpb_csr_ilu0_f64");
}
int hpb_csr_ilu0_c64(hpb_context* ctx, const hpb_csr_tri* lower, void* val) {
    return hpb::ilu0_impl<cf>(ctx, lower, static_cast<cf*>(val), "hpb_csr_ilu0_c64");
}
int hpb_csr_ilu0_c128(hpb_context* ctx, const hpb_csr_tri* lower, void* val) {
    return hpb::ilu0_impl<cd>(ctx, lower, static_cast<cd*>(val), "hpb_csr_ilu0_c128");
}

}  // extern "C"
