// Narrowphase: eight lanes or one thread per candidate pair; manifolds are compacted
// in pair order in the same pass (a tile's hit flags + decoupled look-back), so
// manifold order equals the reference's (src/world/physics_world.cpp:692-736).
// Per pair this is the world's generateContact lambda
// (physics_world.cpp:645-691): collider world transforms, shape dispatch with
// the box-sphere swap (src/collision/narrowphase.cpp:353-365), anchors moved
// from collider space to body space, restitution = max, friction =
// sqrt(max(fa,0) * max(fb,0)).
#include "pe_kernels.cuh"
#include "pe_narrow.cuh"
#include "pe_stages.h"

namespace pe {

// A pair is a chain of dependent arithmetic (two boxes: some 7,000 cycles on one
// thread), so what bounds a step is latency until the chip is full: eight lanes a
// pair (pe_narrow.cuh), and tiles of 32 pairs, whose hit flags one ballot ranks, so
// that the few pairs of a small step are on many SMs.  The lanes repeat what a
// pair's axes and vertices share, though, and hold an eighth of the pairs at a time:
// from kLaneRounds rounds of the grid's tiles on, a thread takes a pair.  Measured,
// us a step, a thread a pair in tiles of 64 before: 10 boxes 77 -> 68, field of
// 1,501 bodies 399 -> 380, 100,000 mixed bodies 143 -> 135, 16 pyramids with hulls
// 599 -> 574; 65,536 boxes in stacks (65,536 pairs, seven rounds) 320, with lanes 336.
// A round is 9 us and a thread a pair 22 to 23 whatever there is: 25,070 pairs, three
// rounds, 27.2 with lanes and 21.8 without.  There a warp takes its pairs by itself: in
// tiles of a block's 256 pairs, which wait for their slowest and leave SMs without one,
// 23,082 pairs of hulls took 288 us and 92,476 of boxes 49 (255 and 44 in the blocks of
// 64 before the lanes), now 200 and 45.
constexpr int kNarrowThreads = 256;
constexpr int kNarrowBlocks = 2;  // resident blocks an SM
constexpr uint32_t kNarrowPairs = kNarrowThreads / kPairLanes;
constexpr uint32_t kLaneRounds = 2;
static_assert(kNarrowPairs == 32, "one warp ranks a tile's pairs");
static_assert(kNarrowPairs >= kMinLookbackTile, "look-back scratch is sized for kMinLookbackTile");

struct NarrowShared {
    uint32_t tile, abort;
    uint32_t hits[kNarrowPairs], rank[kNarrowPairs];
};

// Counters of a tested pair (the first lane of its lanes).
__device__ __forceinline__ void countPair(DevStats *st, uint32_t category, bool epaFailed, bool hit, uint32_t points) {
    if (epaFailed) atomicAdd(&st->epaFailures, 1ull);
    aggregatedCount(st->npCandidates, category);
    if (hit) {
        aggregatedCount(st->npContacts, category);
        aggregatedAdd32(&st->points, points);
    }
}

// One tile, eight lanes a pair.  False when the look-back's wait ran out (then
// nothing of the tile is written).
__device__ __forceinline__ bool laneTile(const WorldView &w, const uint32_t *pairA, const uint32_t *pairB, uint32_t P,
                                         uint32_t ntiles, const ManifoldView &out, uint32_t mcap, DevStats *st,
                                         unsigned long long *state, NarrowShared &sh) {
    const uint32_t lane = threadIdx.x & (kPairLanes - 1), pair = threadIdx.x / kPairLanes;
    const uint32_t p = sh.tile * kNarrowPairs + pair;
    const bool act = p < P;
    // (lanes without a pair run the last pair's arithmetic along)
    const uint32_t ca = pairA[act ? p : P - 1], cb = pairB[act ? p : P - 1];
    const PairSide a = loadPairSide(w, ca), b = loadPairSide(w, cb);
    float restitution = 0.0f, friction = 0.0f;
    LaneManifold lm;
    bool epaFailed;
    narrowphaseLanes(w, act, ca, cb, a, b, lm, restitution, friction, epaFailed);
    if (act && lane == 0) countPair(st, pairCategory(a, b), epaFailed, lm.hit, lm.count);
    if (lane == 0) sh.hits[pair] = lm.hit ? 1u : 0u;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t hits = __ballot_sync(0xffffffffu, sh.hits[threadIdx.x] != 0);
        bool timedOut;
        const uint32_t pre = lookbackExclusiveWarp(state, sh.tile, __popc(hits), &st->err, &timedOut);
        sh.rank[threadIdx.x] = pre + __popc(hits & ((1u << threadIdx.x) - 1u));
        if (threadIdx.x == 0) {
            sh.abort = timedOut ? 1u : 0u;
            if (sh.tile + 1 == ntiles && !timedOut) {
                st->manifolds = pre + __popc(hits);
                st->stamp[3] = globalNs();
            }
        }
    }
    // contacts go out by their lanes, empty ones by the lane of their index
    const uint32_t contacts = (__ballot_sync(0xffffffffu, lm.mine) >> (threadIdx.x & 24u)) & 0xFFu;
    __syncthreads();
    if (sh.abort) return false;
    const uint32_t m = sh.rank[pair];
    if (act && sh.hits[pair] != 0 && m < mcap) {
        if (lane == 0) {
            out.bodyA[m] = a.body;
            out.genA[m] = a.gen;
            out.bodyB[m] = b.body;
            out.genB[m] = b.gen;
            out.normalFriction[m] = make4(lm.normal, friction);
            out.restitution[m] = restitution;
            out.pointCount[m] = lm.count;
        }
        if (lm.mine) {
            out.anchorA[4 * m + lm.slot] = make4(lm.anchorA, lm.depth);
            out.anchorB[4 * m + lm.slot] = make4(lm.anchorB, 0.0f);
            out.feature[4 * m + lm.slot] = lm.feature;
        }
        if (lane < 4) {
            if (lane >= (uint32_t)__popc(contacts)) {
                out.anchorA[4 * m + lane] = make_float4(0, 0, 0, 0);
                out.anchorB[4 * m + lane] = make_float4(0, 0, 0, 0);
                out.feature[4 * m + lane] = 0u;
            }
            out.impulse[4 * m + lane] = make_float4(0, 0, 0, 0);
        }
    }
    return true;
}

// A thread a pair: each warp takes tiles of 32 pairs by itself, so that it waits for
// the slowest of 32 pairs and not of a block's 256.
__device__ __forceinline__ void threadTiles(const WorldView &w, const uint32_t *pairA, const uint32_t *pairB,
                                            uint32_t P, const ManifoldView &out, uint32_t mcap, DevStats *st,
                                            unsigned long long *state, uint32_t *counter, NarrowShared &sh) {
    const uint32_t lane = threadIdx.x & 31, ntiles = (P + 31) / 32;
    // a block's share of the first round by one atomic (one a warp is 2 us of them), the
    // tiles spread over all blocks
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t first = min(kNarrowThreads / 32u, (ntiles + gridDim.x - 1) / gridDim.x);
    if (threadIdx.x == 0) sh.tile = atomicAdd(counter, first);
    __syncthreads();
    auto next = [&] {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(counter, 1u);
        return __shfl_sync(0xffffffffu, t, 0);
    };
    for (uint32_t tile = warp < first ? sh.tile + warp : next(); tile < ntiles; tile = next()) {
        const uint32_t p = tile * 32 + lane;
        PairSide a, b;
        LocalManifold lm;
        lm.count = 0;
        float restitution = 0.0f, friction = 0.0f;
        bool hit = false, epaFailed;
        if (p < P) {
            const uint32_t ca = pairA[p], cb = pairB[p];
            a = loadPairSide(w, ca);
            b = loadPairSide(w, cb);
            hit = narrowphaseRecords(w, ca, cb, a, b, lm, restitution, friction, epaFailed);
            countPair(st, pairCategory(a, b), epaFailed, hit, lm.count);
        }
        const uint32_t hits = __ballot_sync(0xffffffffu, hit), total = __popc(hits);
        bool timedOut;
        const uint32_t pre = lookbackExclusiveWarp(state, tile, total, &st->err, &timedOut);
        if (timedOut) return;  // nothing of this tile is written
        if (lane == 0 && tile + 1 == ntiles) {
            st->manifolds = pre + total;
            st->stamp[3] = globalNs();
        }
        const uint32_t m = pre + __popc(hits & ((1u << lane) - 1u));
        if (hit && m < mcap) storeManifoldGen(out, m, a.body, a.gen, b.body, b.gen, lm, restitution, friction);
    }
}

__global__ void __launch_bounds__(kNarrowThreads, kNarrowBlocks)
k_narrowphase(WorldView w, const uint32_t *__restrict__ pairA, const uint32_t *__restrict__ pairB,
              const uint32_t *d_pairs, uint32_t laneMax, ManifoldView out, uint32_t mcap, DevStats *st,
              unsigned long long *state, uint32_t *counter) {
    __shared__ NarrowShared sh;
    if (blockIdx.x == 0 && threadIdx.x == 0) st->stamp[2] = globalNs();
    const uint32_t P = min(*d_pairs, mcap);
    if (P == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            st->manifolds = 0;
            st->stamp[3] = globalNs();
        }
        return;
    }
    if (P <= laneMax) {
        const uint32_t ntiles = (P + kNarrowPairs - 1) / kNarrowPairs;
        while (takeTile(counter, &sh.tile) < ntiles) {
            if (!laneTile(w, pairA, pairB, P, ntiles, out, mcap, st, state, sh)) return;
            __syncthreads();
        }
        return;
    }
    threadTiles(w, pairA, pairB, P, out, mcap, st, state, counter, sh);
}

void launchNarrowphase(const WorldView &w, const PairBuffers &pb, const ManifoldView &mv, uint32_t mcap, DevStats *st,
                       Scratch &ws, cudaStream_t s, unsigned long long *state, bool stateCleared) {
    uint32_t tiles = (pb.cap + kNarrowPairs - 1) / kNarrowPairs;
    if (tiles == 0) tiles = 1;
    if (!state) state = ws.scanState;
    if (!stateCleared) PE_CHECK(cudaMemsetAsync(state, 0, sizeof(unsigned long long) * (tiles + 1), s));
    const uint32_t maxGrid = kNarrowBlocks * (uint32_t)smCount();
    const uint32_t grid = tiles < maxGrid ? tiles : maxGrid;
    k_narrowphase<<<grid, kNarrowThreads, 0, s>>>(w, pb.a, pb.b, &st->pairs, kLaneRounds * kNarrowPairs * maxGrid, mv,
                                                  mcap, st, state, (uint32_t *)(state + tiles));
    PE_LAUNCHED();
}

} // namespace pe

namespace pe {

// NarrowPhase::generateContact on explicit transforms (sphere / box only):
// in[6k..6k+5] = dims A (w = shape), pos A, rot A, dims B (w = shape), pos B, rot B;
// out[11k..] = normal (w = hit, point count in bits), 4 x anchorA (w = depth),
// 4 x anchorB, features as uint bits in two float4.
__global__ void k_generate_pairs(const float4 *in, float4 *out, uint32_t n) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 da = in[6 * k], pa = in[6 * k + 1], ra = in[6 * k + 2];
    const float4 db = in[6 * k + 3], pb = in[6 * k + 4], rb = in[6 * k + 5];
    const uint32_t sa = (uint32_t)da.w, sb = (uint32_t)db.w;
    Tf tA{f4xyz(pa), f4q(ra)}, tB{f4xyz(pb), f4q(rb)};
    LocalManifold lm;
    lm.count = 0;
    bool hit;
    if (sa == kShapeSphere && sb == kShapeSphere) hit = sphereSphere(da.x, tA, db.x, tB, lm);
    else if (sa == kShapeSphere) hit = sphereBox(da.x, tA, V3{db.x, db.y, db.z}, tB, lm);
    else if (sb == kShapeSphere) {
        hit = sphereBox(db.x, tB, V3{da.x, da.y, da.z}, tA, lm);
        if (hit) {
            lm.normal = -lm.normal;
            for (uint32_t i = 0; i < lm.count; ++i) {
                V3 t = lm.anchorA[i];
                lm.anchorA[i] = lm.anchorB[i];
                lm.anchorB[i] = t;
            }
        }
    } else hit = boxBox(V3{da.x, da.y, da.z}, tA, V3{db.x, db.y, db.z}, tB, lm);
    float4 *o = out + 11 * k;
    o[0] = make_float4(lm.normal.x, lm.normal.y, lm.normal.z, hit ? (float)lm.count : -1.0f);
    for (uint32_t i = 0; i < 4; ++i) {
        bool live = hit && i < lm.count;
        o[1 + i] = live ? make4(lm.anchorA[i], lm.depth[i]) : make_float4(0, 0, 0, 0);
        o[5 + i] = live ? make4(lm.anchorB[i], 0.0f) : make_float4(0, 0, 0, 0);
    }
    uint32_t f[4];
    for (uint32_t i = 0; i < 4; ++i) f[i] = (hit && i < lm.count) ? lm.feature[i] : 0u;
    o[9] = make_float4(__uint_as_float(f[0]), __uint_as_float(f[1]), __uint_as_float(f[2]), __uint_as_float(f[3]));
    o[10] = make_float4(0, 0, 0, 0);
}

void launchGeneratePairs(const float4 *in, float4 *out, uint32_t n, cudaStream_t s) {
    if (!n) return;
    k_generate_pairs<<<(n + 127) / 128, 128, 0, s>>>(in, out, n);
    PE_LAUNCHED();
}

void setSpinLimitNarrow(uint32_t limit) { setSpinLimitOfUnit(limit); }

} // namespace pe
