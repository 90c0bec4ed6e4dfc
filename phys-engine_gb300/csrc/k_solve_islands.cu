// Island-parallel sweeps of the multi-kernel solver (more manifolds than the
// cluster solver holds).  The colouring is the global one (k_color); the
// sweeps then run island by island instead of colour by colour across the
// whole grid: manifolds joined by a dynamic body form an island (static bodies
// join nothing, sequential_impulse_solver.cpp:366-442), no two islands share a
// body, so each island can be solved on its own in the global (colour, index)
// order restricted to it — bit for bit the grid-wide sweeps, without a grid
// barrier per colour.
//
//   k_isl_init  : every dynamic endpoint its own island
//   k_isl_unite : union of the bodies of every solved manifold with two dynamic
//                 bodies (lock-free; roots are the smallest body index)
//   k_isl_count : each solved manifold's island and slot in it; islands listed
//   k_isl_fill  : manifolds into their islands' lists (offsets from a scan);
//                 islands of 32 manifolds or more queued before the others
//   k_isl_solve : islands of kIslBlock to kIslBlockMax manifolds one thread
//                 block each (a pyramid of boxes), sorted by (colour, index) in
//                 shared memory and swept colour by colour with __syncthreads;
//                 then one warp per smaller island (those of 32 manifolds or
//                 more first, from a queue), swept with __syncwarp; islands of
//                 fewer than kIslThread manifolds one per thread, manifold
//                 after manifold in that order (a stack of two boxes would
//                 leave 30 lanes idle); manifolds without a dynamic body
//                 (nothing to share) are solved alone
//   k_isl_sweep : when some island has more than kIslBlockMax manifolds (a
//                 settled pile), all islands together over the whole grid: a
//                 manifold's update starts as soon as the updates before it at
//                 its two bodies are done (each body's velocities carry the
//                 number of updates they have seen), with no barrier between
//                 colours.  Every body sees its manifolds in (colour, index)
//                 order, as in colour-by-colour sweeps, so the result is theirs.
//                 A world whose last steps were piles runs this kernel alone for
//                 every manifold, without the island kernels (launchSolveSweep).
#include <stdexcept>

#include "pe_block.cuh"
#include "pe_kernels.cuh"
#include "pe_prims.cuh"
#include "pe_solve.cuh"
#include "pe_stages.h"

namespace pe {

namespace {

constexpr int kIslThreads = 128;           // four warps per block
constexpr uint32_t kIslWarpSort = 1024;    // island keys sorted in shared memory up to this size
constexpr uint32_t kIslNone = 0xFFFFFFFFu;
// Islands of kIslBlock manifolds or more are swept by a whole thread block
// (one warp would take them colour by colour 32 manifolds at a time), up to
// kIslBlockMax manifolds (the block's shared key buffer).  An island above
// that (a settled pile of thousands of bodies) sends every island of the step
// to the grid-wide sweeps: measured on piles of 5,000 and 10,000 bodies,
// keeping the smaller islands apart only adds their sweep time to the grid's.
constexpr uint32_t kIslBlock = 512;
constexpr uint32_t kIslBlockMax = 4 * kIslWarpSort;
constexpr uint32_t kIslThread = 8;         // islands of fewer manifolds: one thread each
// islCounters: [0] islands, [1] lone manifolds (solved, no dynamic body), [2]
// work queue of the warp items, [3] listed manifolds, [4] / [5] islands of 32
// manifolds or more / kIslThread to 31 queued, [6] smaller islands, [7] set
// when an island exceeds kIslBlockMax manifolds, [8] block islands queued,
// [9] work queue of the block islands; [kIslColorCount + c] manifolds of
// colour c in the grid-wide sweeps, [kIslColorFill + c] their fill cursors
constexpr uint32_t kIslColorCount = 10;
constexpr uint32_t kIslColorFill = 10 + kMaxColors;
static_assert(kIslColorFill + kMaxColors == kIslCounterWords, "island counter layout");

inline uint32_t islGrid(uint32_t n) {
    const uint32_t b = (n + kIslThreads - 1) / kIslThreads;
    const uint32_t maxGrid = 16u * (uint32_t)smCount();
    return b ? (b < maxGrid ? b : maxGrid) : 1u;
}

// Root of i's island, halving the path on the way (par[i] = grandparent).
// Safe beside concurrent unions: only non-roots are written, a non-root
// never becomes a root again, and a grandparent stays an ancestor.
__device__ __forceinline__ uint32_t islFind(uint32_t *par, uint32_t i, uint32_t nb) {
    for (uint32_t n = 0; n <= nb; ++n) {
        const uint32_t p = ldvol(&par[i]);
        if (p == i) return i;
        const uint32_t gp = ldvol(&par[p]);
        if (gp == p) return p;
        par[i] = gp;
        i = gp;
    }
    return i;
}

__device__ __forceinline__ void islUnite(uint32_t *par, uint32_t a, uint32_t b, uint32_t nb, uint32_t *err) {
    for (uint32_t spins = 0; spins < spinLimit(); ++spins) {
        a = islFind(par, a, nb);
        b = islFind(par, b, nb);
        if (a == b) return;
        const uint32_t hi = a > b ? a : b, lo = a > b ? b : a;
        const uint32_t old = atomicCAS(&par[hi], hi, lo);
        if (old == hi) return;
        a = old;
        b = lo;
    }
    atomicOr(err, kErrTimeout);
}

// More colours than the per-colour counters hold (colour windows): every
// island goes to the grid-wide sweeps, with its per-colour counts and fill
// cursors in sb.colorStart.
__device__ __forceinline__ uint32_t islWideColors(const SolveArgs &a, uint32_t M) {
    const uint32_t C = __ldcg(&a.st->colors);
    return C > (uint32_t)kMaxColors ? (C < M ? C : M) : 0u;
}

__device__ __forceinline__ uint32_t *islPar(const SolveArgs &a) { return a.sb.islPar; }
__device__ __forceinline__ uint32_t *islCnt(const SolveArgs &a) { return a.sb.islPar + a.w.nb; }

} // namespace

// Per-body counts all zero (they are scanned into list offsets), every dynamic
// endpoint its own island and without colours.
__global__ void k_isl_init(SolveArgs a) {
    const uint32_t M = min(*a.count, a.mcap);
    uint32_t *par = islPar(a), *cnt = islCnt(a);
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t i = t; i < kIslCounterWords; i += stride) a.sb.islCounters[i] = 0u;
    for (uint32_t i = t; i < a.w.nb; i += stride) cnt[i] = 0u;
    const uint32_t wideC = islWideColors(a, M);
    for (uint32_t i = t; i < wideC; i += stride) a.sb.colorStart[i] = 0u;
    for (uint32_t m = t; m < M; m += stride) {
        const uint32_t fl = a.sb.dyn[m];
        for (int e = 0; e < 2; ++e) {
            if (!(fl & (e ? kFlagDynB : kFlagDynA))) continue;
            const uint32_t b = e ? a.mv.bodyB[m] : a.mv.bodyA[m];
            par[b] = b;
            a.sb.bodyUsed[2 * b] = a.sb.bodyUsed[2 * b + 1] = 0ull;  // colours of the sweeps, set by k_isl_fill
        }
    }
}

__global__ void k_isl_unite(SolveArgs a) {
    const uint32_t M = min(*a.count, a.mcap);
    uint32_t *par = islPar(a);
    for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        const uint32_t fl = a.sb.dyn[m];
        if ((fl & (kFlagValid | kFlagDynA | kFlagDynB)) == (kFlagValid | kFlagDynA | kFlagDynB))
            islUnite(par, a.mv.bodyA[m], a.mv.bodyB[m], a.w.nb, &a.st->err);
    }
}

__global__ void k_isl_count(SolveArgs a) {
    const uint32_t M = min(*a.count, a.mcap);
    uint32_t *par = islPar(a), *cnt = islCnt(a);
    for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        const uint32_t fl = a.sb.dyn[m];
        uint32_t root = kIslNone;
        if ((fl & kFlagValid) && (fl & (kFlagDynA | kFlagDynB))) {
            root = islFind(par, (fl & kFlagDynA) ? a.mv.bodyA[m] : a.mv.bodyB[m], a.w.nb);
            const uint32_t pos = aggregatedAppendKeyed(cnt, root);
            a.sb.islSlot[m] = pos;
            if (pos == kIslBlockMax) a.sb.islCounters[7] = 1u;
            if (pos == 0) a.sb.islRoots[aggregatedAppend(&a.sb.islCounters[0])] = root;
        } else if (fl & kFlagValid) {
            a.sb.islLone[aggregatedAppend(&a.sb.islCounters[1])] = m;
        }
        a.sb.islRoot[m] = root;
    }
}

// Islands of at least this many manifolds go to the grid-wide sweeps: all
// once some island is large or the colours exceed kMaxColors, none otherwise.
__device__ __forceinline__ uint32_t islSweepFrom(const SolveArgs &a, uint32_t M) {
    return (a.sb.islCounters[7] || islWideColors(a, M)) ? 1u : kIslNone;
}

__global__ void k_isl_fill(SolveArgs a) {
    const uint32_t M = min(*a.count, a.mcap);
    const uint32_t *cnt = islCnt(a);
    const uint32_t sweepFrom = islSweepFrom(a, M), wideC = islWideColors(a, M);
    uint32_t *colorCounts = wideC ? a.sb.colorStart : a.sb.islCounters + kIslColorCount;
    const uint32_t colorLimit = wideC ? wideC : (uint32_t)kMaxColors;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t m = t; m < M; m += stride) {
        const uint32_t r = a.sb.islRoot[m];
        if (r == kIslNone) continue;
        a.sb.islList[a.sb.islOff[r] + a.sb.islSlot[m]] = m;
        const uint32_t c = a.sb.color[m];
        if (cnt[r] >= sweepFrom && c < colorLimit) {
            aggregatedAppendKeyed(colorCounts, c);
            if (!wideC) {
                const uint32_t fl = a.sb.dyn[m], word = c >> 6;
                const unsigned long long bit = 1ull << (c & 63);
                if (fl & kFlagDynA) atomicOr(&a.sb.bodyUsed[2 * a.mv.bodyA[m] + word], bit);
                if (fl & kFlagDynB) atomicOr(&a.sb.bodyUsed[2 * a.mv.bodyB[m] + word], bit);
            }
        }
    }
    // the warp queue: islands of 32 manifolds or more at the front (a warp's
    // lanes all busy; they bound the sweep), those of kIslThread to 31 from
    // the back; smaller ones to the per-thread list, islands of kIslBlock or
    // more to the block list (the per-thread list's area, from its end)
    uint32_t *queue = reinterpret_cast<uint32_t *>(a.sb.islKeys), *tiny = queue + a.mcap;
    const uint32_t nIsl = a.sb.islCounters[0];
    for (uint32_t i = t; i < nIsl; i += stride) {
        const uint32_t r = a.sb.islRoots[i];
        if (cnt[r] >= sweepFrom) continue;
        if (cnt[r] >= kIslBlock) tiny[a.mcap - 1 - aggregatedAppend(&a.sb.islCounters[8])] = r;
        else if (cnt[r] >= 32) queue[aggregatedAppend(&a.sb.islCounters[4])] = r;
        else if (cnt[r] >= kIslThread) queue[nIsl - 1 - aggregatedAppend(&a.sb.islCounters[5])] = r;
        else {
            tiny[aggregatedAppend(&a.sb.islCounters[6])] = r;
            aggregatedAdd32(&a.st->loose, cnt[r]);
        }
    }
}

namespace {
// Sorts keys[0, n) (n a power of two) ascending with one warp.
__device__ __forceinline__ void warpBitonicSort(unsigned long long *keys, uint32_t n, uint32_t lane) {
    for (uint32_t k = 2; k <= n; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = lane; i < n; i += 32) {
                const uint32_t ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long x = keys[i], y = keys[ixj];
                    if ((x > y) == ((i & k) == 0)) {
                        keys[i] = y;
                        keys[ixj] = x;
                    }
                }
            }
            __syncwarp();
        }
}
} // namespace

__global__ void __launch_bounds__(kIslThreads) k_isl_solve(SolveArgs a) {
    __shared__ unsigned long long s_keys[kIslThreads / 32][kIslWarpSort];
    __shared__ uint32_t s_start[kIslThreads / 32][kMaxColors + 1];
    __shared__ uint32_t s_item;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // islands of kIslBlock manifolds or more: one block each
    {
        const uint32_t nBlock = a.sb.islCounters[8];
        const uint32_t *blockList = reinterpret_cast<const uint32_t *>(a.sb.islKeys) + a.mcap;
        unsigned long long *keys = &s_keys[0][0];  // kIslBlockMax keys
        uint32_t *start = s_start[0];
        for (;;) {
            if (threadIdx.x == 0) s_item = atomicAdd(&a.sb.islCounters[9], 1u);
            __syncthreads();
            const uint32_t item = s_item;
            if (item >= nBlock) break;
            const uint32_t r = blockList[a.mcap - 1 - item];
            const uint32_t n = islCnt(a)[r], base = a.sb.islOff[r];
            const uint32_t n2 = nextPow2(n);
            for (uint32_t j = threadIdx.x; j < n2; j += blockDim.x) {
                unsigned long long key = ~0ull;
                if (j < n) {
                    const uint32_t m = a.sb.islList[base + j];
                    key = ((unsigned long long)a.sb.color[m] << 32) | m;
                }
                keys[j] = key;
            }
            __syncthreads();
            blockBitonicSort(keys, n2);
            // colour ranges [start[c], start[c + 1])
            const uint32_t lastColor = (uint32_t)(keys[n - 1] >> 32);
            const uint32_t C = lastColor < (uint32_t)kMaxColors ? lastColor + 1 : (uint32_t)kMaxColors;
            for (uint32_t c = threadIdx.x; c <= C; c += blockDim.x) {
                uint32_t lo = 0, hi = n;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if ((uint32_t)(keys[mid] >> 32) < c) lo = mid + 1;
                    else hi = mid;
                }
                start[c] = lo;
            }
            __syncthreads();
            for (int pass = 0; pass <= a.iterations; ++pass)
                for (uint32_t c = 0; c < C; ++c) {
                    for (uint32_t j = start[c] + threadIdx.x; j < start[c + 1]; j += blockDim.x) {
                        const uint32_t m = (uint32_t)(keys[j] & 0xFFFFFFFFull);
                        if (pass == 0) warmStartOne(a, j, m);
                        else solveOneChained(a, j, m);
                    }
                    __syncthreads();
                }
        }
    }
    const uint32_t nIsl = a.sb.islCounters[0];
    const uint32_t nFront = a.sb.islCounters[4], nWarp = nFront + a.sb.islCounters[5], nTiny = a.sb.islCounters[6];
    const uint32_t nItems = nWarp + (nTiny + 31) / 32;
    const uint32_t *queue = reinterpret_cast<const uint32_t *>(a.sb.islKeys), *tiny = queue + a.mcap;
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(&a.sb.islCounters[2], 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= nItems) break;
        if (i >= nWarp) {
            // 32 small islands, one per lane, each swept manifold after
            // manifold in (colour, index) order
            const uint32_t t = (i - nWarp) * 32 + lane;
            if (t < nTiny) {
                const uint32_t r = tiny[t];
                const uint32_t n = islCnt(a)[r], base = a.sb.islOff[r];
                unsigned long long *keys = &s_keys[warp][lane * kIslThread];
                for (uint32_t j = 0; j < n; ++j) {
                    const uint32_t m = a.sb.islList[base + j];
                    const unsigned long long key = ((unsigned long long)a.sb.color[m] << 32) | m;
                    uint32_t p = j;
                    for (; p > 0 && keys[p - 1] > key; --p) keys[p] = keys[p - 1];
                    keys[p] = key;
                }
                for (int pass = 0; pass <= a.iterations; ++pass)
                    for (uint32_t j = 0; j < n; ++j) {
                        const uint32_t m = (uint32_t)(keys[j] & 0xFFFFFFFFull);
                        if (pass == 0) warmStartOne(a, j, m);
                        else solveOneChained(a, j, m);
                    }
            }
            __syncwarp();
            continue;
        }
        const uint32_t r = i < nFront ? queue[i] : queue[nIsl - 1 - (i - nFront)];
        const uint32_t n = islCnt(a)[r], base = a.sb.islOff[r];
        // the island's manifolds in (colour, index) order
        const uint32_t n2 = nextPow2(n);
        // large islands sort in global scratch: [2 base, 2 base + n2) lies
        // inside the island's own range [2 base, 2 (base + n)) of 2 mcap keys
        unsigned long long *keys = n2 <= kIslWarpSort ? s_keys[warp] : a.sb.islSort + (size_t)2 * base;
        for (uint32_t j = lane; j < n2; j += 32) {
            unsigned long long key = ~0ull;
            if (j < n) {
                const uint32_t m = a.sb.islList[base + j];
                key = ((unsigned long long)a.sb.color[m] << 32) | m;
            }
            keys[j] = key;
        }
        __syncwarp();
        warpBitonicSort(keys, n2, lane);
        // colour ranges [s_start[c], s_start[c + 1])
        const uint32_t lastColor = (uint32_t)(keys[n - 1] >> 32);
        const uint32_t C = lastColor < (uint32_t)kMaxColors ? lastColor + 1 : (uint32_t)kMaxColors;
        for (uint32_t c = lane; c <= C; c += 32) {
            uint32_t lo = 0, hi = n;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if ((uint32_t)(keys[mid] >> 32) < c) lo = mid + 1;
                else hi = mid;
            }
            s_start[warp][c] = lo;
        }
        __syncwarp();
        for (int pass = 0; pass <= a.iterations; ++pass)
            for (uint32_t c = 0; c < C; ++c) {
                for (uint32_t j = s_start[warp][c] + lane; j < s_start[warp][c + 1]; j += 32) {
                    const uint32_t m = (uint32_t)(keys[j] & 0xFFFFFFFFull);
                    if (pass == 0) warmStartOne(a, j, m);
                    else solveOneChained(a, j, m);
                }
                __syncwarp();
            }
        __syncwarp();
    }
    // manifolds with no dynamic body: nothing is shared, each alone
    const uint32_t nLone = a.sb.islCounters[1];
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nLone; j += gridDim.x * blockDim.x) {
        const uint32_t m = a.sb.islLone[j];
        warmStartOne(a, j, m);
        for (int it = 0; it < a.iterations; ++it) solveOne(a, j, m);
    }
}

// More than kMaxColors colours: every island in grid-wide sweeps, the
// per-colour counts in sb.colorStart scanned into starts by block 0, then used
// as fill cursors (after the fill, colorStart[c] is the end of colour c).
__device__ void islSolveWide(const SolveArgs &a, uint32_t M, uint32_t C) {
    __shared__ uint32_t s_scan[9], s_carry;
    uint32_t *cur = a.sb.colorStart;
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) s_carry = 0;
        __syncthreads();
        for (uint32_t c0 = 0; c0 < C; c0 += blockDim.x) {
            const uint32_t c = c0 + threadIdx.x;
            const uint32_t v = c < C ? __ldcg(&cur[c]) : 0u;
            uint32_t total;
            const uint32_t ex = blockExclusiveScan(v, total, s_scan);
            if (c < C) __stcg(&cur[c], s_carry + ex);
            __syncthreads();
            if (threadIdx.x == 0) s_carry += total;
            __syncthreads();
        }
    }
    if (!gridBarrier(a.sb.bar + 1, &a.st->err)) return;
    const uint32_t *cnt = islCnt(a);
    uint32_t *list = reinterpret_cast<uint32_t *>(a.sb.islKeysTmp);
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, gstride = gridDim.x * blockDim.x;
    for (uint32_t m = gtid; m < M; m += gstride) {
        const uint32_t r = a.sb.islRoot[m];
        const uint32_t c = a.sb.color[m];
        if (r == kIslNone || cnt[r] == 0 || c >= C) continue;
        list[aggregatedAppendKeyed(cur, c)] = m;
    }
    if (!gridBarrier(a.sb.bar + 1, &a.st->err)) return;
    for (int pass = 0; pass <= a.iterations; ++pass)
        for (uint32_t c = 0; c < C; ++c) {
            const uint32_t lo = c ? __ldcg(&cur[c - 1]) : 0u, hi = __ldcg(&cur[c]);
            for (uint32_t k = lo + gtid; k < hi; k += gstride) {
                if (pass == 0) warmStartOne(a, k, list[k]);
                else solveOne(a, k, list[k]);
            }
            if (!gridBarrier(a.sb.bar + 1, &a.st->err)) return;
        }
}

// ----------------------------------------------------------------- sweeps ---
// A body's velocity vectors carry in .w how many updates the body has seen this
// solve (0 as the integrate kernel leaves them; the body's last update writes 0
// again).  The update of pass p at a manifold whose colour has r lower colours
// among the body's d waits for p d + r and leaves p d + r + 1: data and flag are
// one 16-byte word, read and written whole, so no fence or barrier goes with it.
//
// A warp takes eight manifolds of one colour, four lanes each, one lane a
// contact point: the point's constants and impulses stay in the lane's registers
// for the whole solve, the velocities move from lane to lane as the points follow
// one another, and lane r loads and stores vector r (linear and angular velocity
// of body A, then of B).  All eight start together once their sixteen bodies are
// ready; what they wait for has an earlier (pass, colour), so with every warp
// resident (cooperative launch) and each taking its items in that order some warp
// can always go on.  With more items than warps a warp reloads the constants.
//
// What bounds it is the chain of updates at the busiest bodies: 9 or 21 passes x
// 8 colours in the piles below, an update about 0.45 us a point and 0.5 us from
// a store to the load that sees it.  Measured against a grid barrier after each
// colour (4.0 us a colour step), us a whole step: field of 10,000 bodies (18,000
// manifolds) 568 -> 428, of 50,000 (84,000, several items a warp) 840 -> 700; 16
// pyramids with hulls (7,000) 1,056 -> 692, 256 of them (110,000) 1,829 -> 1,373.
constexpr uint32_t kWarp = 0xffffffffu;
constexpr uint32_t kItemManifolds = 8;
// List entries: manifold index | solved points << 29.
constexpr uint32_t kEntryShift = 29;
constexpr uint32_t kEntryMask = (1u << kEntryShift) - 1u;
constexpr uint32_t kNoEntry = 0xFFFFFFFFu;  // (a manifold has at most four points)

// 16 bytes read or written in one access at device scope.
__device__ __forceinline__ float4 loadWord(const float4 *p) {
    unsigned __int128 v;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(v) : "l"(p) : "memory");
    return make_float4(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)),
                       __uint_as_float((uint32_t)(v >> 64)), __uint_as_float((uint32_t)(v >> 96)));
}
__device__ __forceinline__ void storeWord(float4 *p, const V3 &v, uint32_t tag) {
    const unsigned long long lo = ((unsigned long long)__float_as_uint(v.y) << 32) | __float_as_uint(v.x),
                             hi = ((unsigned long long)tag << 32) | __float_as_uint(v.z);
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(((unsigned __int128)hi << 64) | lo) : "memory");
}

// One lane's share of a manifold.
struct SweepLane {
    float4 o[kPreparedVec4], imp;  // the lane's point
    V3 n;
    float friction, imA, imB;
    uint32_t m, npts;
    bool act, sA, sB;  // the group has a manifold; its bodies are static
    // the lane's velocity vector: where it is, whether its updates are counted
    // (a moving body), whether it is written, lower colours and colours there
    float4 *addr;
    bool counted, writes;
    uint32_t rank, degree;
};

__device__ __forceinline__ void loadSweepLane(const SolveArgs &a, uint32_t entry, uint32_t p, SweepLane &f) {
    f.act = entry != kNoEntry;
    f.m = f.act ? entry & kEntryMask : 0u;
    f.npts = f.act ? entry >> kEntryShift : 0u;
    const SolverBuffers &sb = a.sb;
    const float4 pm = sb.pm[f.m], pn = sb.pn[f.m];
    const uint2 b = sb.pbody[f.m];
    const uint32_t fl = sb.dyn[f.m], c = sb.color[f.m];
    f.n = f4xyz(pn);
    f.friction = pn.w;
    f.imA = pm.x;
    f.imB = pm.z;
    f.sA = pm.y != 0.0f;
    f.sB = pm.w != 0.0f;
    if (p < f.npts) {
#pragma unroll
        for (uint32_t v = 0; v < (uint32_t)kPreparedVec4; ++v) f.o[v] = sb.pp[(size_t)(v * 4 + p) * a.mcap + f.m];
        f.imp = sb.pimp[(size_t)p * a.mcap + f.m];
    }
    const uint32_t body = p < 2 ? b.x : b.y;
    f.addr = (p & 1u ? a.w.nxt.ang : a.w.nxt.lin) + body;
    f.counted = f.act && (fl & (p < 2 ? kFlagDynA : kFlagDynB)) != 0;
    f.writes = f.act && !(p < 2 ? f.sA : f.sB);
    f.rank = f.degree = 0;
    if (f.counted) {
        const unsigned long long u0 = __ldcg(&sb.bodyUsed[2 * body]), u1 = __ldcg(&sb.bodyUsed[2 * body + 1]);
        f.degree = (uint32_t)(__popcll(u0) + __popcll(u1));
        const unsigned long long below = (1ull << (c & 63)) - 1ull;
        f.rank = c < 64 ? (uint32_t)__popcll(u0 & below) : (uint32_t)(__popcll(u0) + __popcll(u1 & below));
    }
}

__device__ __forceinline__ V3 shfl3(const V3 &v, uint32_t from) {
    return {__shfl_sync(kWarp, v.x, from), __shfl_sync(kWarp, v.y, from), __shfl_sync(kWarp, v.z, from)};
}

// The update of pass `pass` (0: the warm start) of the warp's eight manifolds.
// False when the wait for their bodies ran out.
__device__ __forceinline__ bool sweepVisit(const SolveArgs &a, SweepLane &f, uint32_t pass, uint32_t passes) {
    const uint32_t lane = threadIdx.x & 31, p = lane & 3, first = lane & ~3u;
    const uint32_t want = pass * f.degree + f.rank;
    float4 own = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    bool ready = !f.act;
    for (uint32_t spins = 0;;) {
        if (!ready) {
            own = loadWord(f.addr);
            ready = !f.counted || __float_as_uint(own.w) == want;
        }
        if (__all_sync(kWarp, ready)) break;
        if (++spins > spinLimit() || ((spins & 1023u) == 0 && (ldvol(&a.st->err) & kErrTimeout))) {
            if (lane == 0) atomicOr(&a.st->err, kErrTimeout);
            return false;
        }
    }
    const V3 v = f4xyz(own);
    V3 linA = shfl3(v, first), angA = shfl3(v, first + 1), linB = shfl3(v, first + 2), angB = shfl3(v, first + 3);
    const bool movesA = __any_sync(kWarp, f.act && !f.sA);  // some group's body A (often the floor) moves
    const uint32_t turns = __reduce_max_sync(kWarp, f.npts);
    M3 IA, IB;
    if (pass == 0 && p < f.npts && f.imp.w != 0.0f) {
        float4 r[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) r[j] = a.sb.pmInertia[(size_t)j * a.mcap + f.m];
        IA = M3{r[0].x, r[0].y, r[0].z, r[1].x, r[1].y, r[1].z, r[2].x, r[2].y, r[2].z};
        IB = M3{r[3].x, r[3].y, r[3].z, r[4].x, r[4].y, r[4].z, r[5].x, r[5].y, r[5].z};
    }
    for (uint32_t q = 0; q < turns; ++q) {
        if (p == q && q < f.npts) {
            const float4(&o)[kPreparedVec4] = f.o;
            const V3 offA = f4xyz(o[0]), offB = f4xyz(o[1]), t1 = f4xyz(o[2]), t2 = f4xyz(o[3]);
            if (pass == 0) {
                // warmStartOne's application
                if (f.imp.w != 0.0f) {
                    const V3 wi = f.n * f.imp.x + t1 * f.imp.y + t2 * f.imp.z;
                    const V3 nw = -wi;
                    if (!f.sA) {
                        linA += nw * f.imA;
                        angA += mul(IA, cross(offA, nw));
                    }
                    if (!f.sB) {
                        linB += wi * f.imB;
                        angB += mul(IB, cross(offB, wi));
                    }
                }
            } else if (!(o[0].w <= 0.0f)) {
                // solveOne's update, operation for operation
                const float iem = o[0].w, bias = o[1].w, rv = o[2].w, itm00 = o[3].w, itm01 = o[4].w, itm11 = o[5].w;
                const V3 vA = linA + cross(angA, offA);
                const V3 vB = linB + cross(angB, offB);
                const V3 rel = vB - vA;
                const float vn = dot(rel, f.n);
                const float delta = -(vn + rv - bias) / iem;
                const float prev = f.imp.x;
                f.imp.x = smax(prev + delta, 0.0f);
                const float applied = f.imp.x - prev;
                const V3 impulse = f.n * applied;
                if (!f.sA) {
                    linA += (-impulse) * f.imA;
                    angA += f4xyz(o[4]) * (-applied);
                }
                if (!f.sB) {
                    linB += impulse * f.imB;
                    angB += f4xyz(o[5]) * applied;
                }
                if (!(itm00 <= 0.0f || itm11 <= 0.0f)) {
                    const float limit = smax(f.friction, 0.0f) * f.imp.x;
                    const float tv1 = dot(rel, t1) + o[6].w * applied;
                    const float tv2 = dot(rel, t2) + o[7].w * applied;
                    const float d1 = -(itm00 * tv1 + itm01 * tv2);
                    const float d2 = -(itm01 * tv1 + itm11 * tv2);
                    const float p1 = f.imp.y, p2 = f.imp.z;
                    f.imp.y += d1;
                    f.imp.z += d2;
                    const float lsq = f.imp.y * f.imp.y + f.imp.z * f.imp.z;
                    if (lsq > limit * limit) {
                        const float sc = limit / sqrtf(lsq);
                        f.imp.y *= sc;
                        f.imp.z *= sc;
                    }
                    const float a1 = f.imp.y - p1, a2 = f.imp.z - p2;
                    const V3 ti = t1 * a1 + t2 * a2;
                    const V3 rA = f4xyz(o[6]) * a1 + f4xyz(o[8]) * a2;
                    const V3 rB = f4xyz(o[7]) * a1 + f4xyz(o[9]) * a2;
                    if (!f.sA) {
                        linA += (-ti) * f.imA;
                        angA += -rA;
                    }
                    if (!f.sB) {
                        linB += ti * f.imB;
                        angB += rB;
                    }
                }
            }
        }
        // on to the next point's lane, and after the last to all four
        if (movesA) {
            linA = shfl3(linA, first + q);
            angA = shfl3(angA, first + q);
        }
        linB = shfl3(linB, first + q);
        angB = shfl3(angB, first + q);
    }
    const V3 out = p == 0 ? linA : p == 1 ? angA : p == 2 ? linB : angB;
    if (f.counted) {
        const bool end = pass + 1 == passes && f.rank + 1 == f.degree;
        storeWord(f.addr, out, end ? 0u : want + 1u);
    } else if (f.writes) {
        st4(f.addr, make4(out, 0.0f));
    }
    return true;
}

// The solved point's impulse and its warm-start cache entry (cache in manifold
// order: offsets from k_cache_offsets).
__device__ __forceinline__ void writePoint(const SolveArgs &a, const CacheView &nc, uint32_t cacheCap, uint32_t m,
                                           uint32_t p, float4 imp) {
    imp.w = 0.0f;
    a.mv.impulse[4 * m + p] = imp;
    const uint32_t e = a.sb.cacheOff[m] + p;
    if (e >= cacheCap) return;
    const float4 aa = a.mv.anchorA[4 * m + p], ab = a.mv.anchorB[4 * m + p];
    nc.key[e] = ((unsigned long long)a.mv.bodyA[m] << 32) | a.mv.bodyB[m];
    nc.gens[e] = ((unsigned long long)a.mv.genA[m] << 32) | a.mv.genB[m];
    nc.anchorA[e] = make_float4(aa.x, aa.y, aa.z, imp.x);
    nc.anchorB[e] = make_float4(ab.x, ab.y, ab.z, imp.y);
    nc.tangent2[e] = imp.z;
}

// ALL: every manifold of the step (colour counts and body masks from k_color,
// results written here); otherwise those that k_isl_fill left to the sweeps.
// ALL takes manifolds whose body handles are both live, or whose bodies both do not
// move (sleeping).  A stale handle beside a moving body would count in that body's mask
// without an update, and the body's later updates would wait for it until their limit.
// The host takes this path only where collider i is on live body i (launchSolver).
template <bool ALL>
__global__ void __launch_bounds__(kSolveThreads, 2) k_isl_sweep(SolveArgs a, CacheView nc, uint32_t cacheCap) {
    __shared__ uint32_t s_start[kMaxColors + 1];  // first item of each colour
    const uint32_t M = min(*a.count, a.mcap);
    {
        const uint32_t wideC = islWideColors(a, M);
        if (wideC) {  // every block sees the same colour count
            if (!ALL) islSolveWide(a, M, wideC);
            else if (threadIdx.x == 0) atomicOr(&a.st->err, kErrSmallPath);  // re-run on the island path
            return;
        }
    }
    const uint32_t *count = ALL ? a.sb.colorCount : a.sb.islCounters + kIslColorCount;
    uint32_t *fill = a.sb.islCounters + kIslColorFill;
    if (threadIdx.x == 0) {
        uint32_t acc = 0;
        for (int c = 0; c < kMaxColors; ++c) {
            s_start[c] = acc;
            acc += (count[c] + kItemManifolds - 1) / kItemManifolds;
        }
        s_start[kMaxColors] = acc;
    }
    __syncthreads();
    const uint32_t items = s_start[kMaxColors];
    if (items == 0) return;
    // the manifolds colour by colour, each colour from a whole item
    const uint32_t *cnt = islCnt(a);
    const uint32_t sweepFrom = ALL ? 0u : islSweepFrom(a, M);
    uint32_t *list = reinterpret_cast<uint32_t *>(a.sb.islKeysTmp);
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, gstride = gridDim.x * blockDim.x;
    for (uint32_t m = gtid; m < M; m += gstride) {
        const uint32_t c = a.sb.color[m];
        if (c >= (uint32_t)kMaxColors) continue;
        if (!ALL) {
            const uint32_t r = a.sb.islRoot[m];
            if (r == kIslNone || cnt[r] < sweepFrom) continue;
        }
        list[kItemManifolds * s_start[c] + aggregatedAppendKeyed(fill, c)] =
            m | min(a.sb.pcount[m], 4u) << kEntryShift;
    }
    for (uint32_t c = gtid; c < (uint32_t)kMaxColors; c += gstride)
        for (uint32_t i = kItemManifolds * s_start[c] + count[c]; i < kItemManifolds * s_start[c + 1]; ++i)
            list[i] = kNoEntry;
    if (!gridBarrier(a.sb.bar + 1, &a.st->err)) return;
    const uint32_t lane = threadIdx.x & 31, p = lane & 3, passes = (uint32_t)a.iterations + 1u;
    // items go round the blocks, so that a colour's are spread over every SM
    const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps = gridDim.x * (blockDim.x >> 5);
    auto keepImpulse = [&](const SweepLane &f, bool end) {
        if (p >= f.npts) return;
        if (ALL && end) writePoint(a, nc, cacheCap, f.m, p, f.imp);
        else a.sb.pimp[(size_t)p * a.mcap + f.m] = f.imp;
    };
    // manifolds at bodies with few others (the host's choice of the next step's path)
    auto countLoose = [&](const SweepLane &f) {
        uint32_t g = __ballot_sync(kWarp, f.act && f.degree <= 2);
        g &= g >> 1;
        g &= g >> 2;
        if (lane == 0 && (g & 0x11111111u)) atomicAdd(&a.st->loose, (uint32_t)__popc(g & 0x11111111u));
    };
    if (items <= warps) {
        if (warp >= items) return;
        SweepLane f;
        loadSweepLane(a, __ldcg(&list[kItemManifolds * warp + (lane >> 2)]), p, f);
        if (ALL) countLoose(f);
        for (uint32_t pass = 0; pass < passes; ++pass)
            if (!sweepVisit(a, f, pass, passes)) return;
        keepImpulse(f, true);
        return;
    }
    for (uint32_t pass = 0; pass < passes; ++pass)
        for (uint32_t item = warp; item < items; item += warps) {
            SweepLane f;
            loadSweepLane(a, __ldcg(&list[kItemManifolds * item + (lane >> 2)]), p, f);
            if (ALL && pass == 0) countLoose(f);
            if (!sweepVisit(a, f, pass, passes)) return;
            keepImpulse(f, pass + 1 == passes);
        }
}

// A cooperative launch of k_isl_sweep on every block that the device holds.
template <bool ALL> static void launchSweep(const SolveArgs &a, const CacheView &nc, uint32_t cacheCap, cudaStream_t s) {
    // list entries carry the manifold index in kEntryShift bits
    if (a.mcap > kEntryMask) throw std::length_error("manifold capacity beyond the grid-wide sweeps' index range");
    const void *kernel = (const void *)k_isl_sweep<ALL>;
    static PerDevice resident;
    const int perSm = resident([&] {
        int b = 0;
        PE_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kSolveThreads, 0));
        return b < 1 ? 1 : b;
    });
    SolveArgs args = a;
    CacheView cache = nc;
    void *params[] = {&args, &cache, &cacheCap};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(perSm * smCount());
    cfg.blockDim = dim3(kSolveThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PE_CHECK(cudaLaunchKernelExC(&cfg, kernel, params));
    PE_LAUNCHED();
}

void launchSolveSweep(const SolveArgs &a, const CacheView &newCache, uint32_t cacheCap, cudaStream_t s) {
    launchSweep<true>(a, newCache, cacheCap, s);
}

void launchSolveIslands(const SolveArgs &a, Scratch &ws, cudaStream_t s) {
    const uint32_t mcap = a.mcap;
    k_isl_init<<<islGrid(mcap), kIslThreads, 0, s>>>(a);
    PE_LAUNCHED();
    k_isl_unite<<<islGrid(mcap), kIslThreads, 0, s>>>(a);
    PE_LAUNCHED();
    k_isl_count<<<islGrid(mcap), kIslThreads, 0, s>>>(a);
    PE_LAUNCHED();
    // offsets of the islands' lists: exclusive scan of the per-body counts
    // (zero for bodies that are not an island root)
    launchScanExclusive(a.sb.islPar + a.w.nb, a.sb.islOff, nullptr, a.w.nb, &a.sb.islCounters[3], ws, &a.st->err, s);
    k_isl_fill<<<islGrid(mcap), kIslThreads, 0, s>>>(a);
    PE_LAUNCHED();
    k_isl_solve<<<4 * smCount(), kIslThreads, 0, s>>>(a);
    PE_LAUNCHED();
    launchSweep<false>(a, CacheView{}, 0u, s);
}

void setSpinLimitIslands(uint32_t limit) { setSpinLimitOfUnit(limit); }

} // namespace pe
