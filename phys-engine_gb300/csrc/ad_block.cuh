// The differentiable step (ad_world.cuh) on one thread block.
//
// A step is a chain of short stages, so what bounds it is latency: a stage
// waits for memory, for a barrier or for one thread.  The block therefore
//  * gives a manifold four lanes, one for each contact point: the points'
//    constants, impulses and adjoints stay in the lanes' registers over all
//    iterations, and only the twelve velocity components move from lane to lane
//    (shuffles) as the points follow one another;
//  * keeps the sorts, the colouring and the velocities in shared memory, where
//    a world of up to kStageBodies bodies fits (global memory beyond);
//  * sorts 64 keys at a time in a warp's registers, so that a sort has a
//    barrier only where warps exchange keys;
//  * colours in rounds over all manifolds (a manifold takes its colour once it
//    is the highest-priority one left at both its bodies, which gives the
//    greedy colouring), and writes the warm-start cache from a scan: pair order
//    is the cache's order, one manifold a body pair.
// Prepared data lie field by field (field * 4 maxManifolds + 4 k + p), so that
// neighbouring lanes read neighbouring words.
//
// Measured on 8 worlds of 32 boxes on a plane (20 steps, one block a world), us
// a step, with one thread a manifold, sorts in global memory and the geometry's
// Jacobian in dual numbers before: forward 148, adjoint 748 (of them 153 for
// the recomputed forward step, 222 for the reversed iterations, 360 for the
// geometry); now 44 and 98.
#pragma once
#include "ad_world.cuh"
#include "pe_block.cuh"

namespace pe {
namespace ad {

using F = float;

constexpr uint32_t kSortShared = 2048;   // keys sorted in shared memory
constexpr uint32_t kStageBodies = 1024;  // bodies whose velocities / colour masks are kept there

// Dynamic shared memory of a block that steps worlds of up to n bodies: sort
// keys, colour masks and velocities take turns in it.
__host__ __device__ inline uint32_t sharedSortKeys(uint32_t n) {
    uint32_t k = 256;
    while (k < 4 * n && k < kSortShared) k <<= 1;
    return k;
}
__host__ __device__ inline uint32_t sharedBytes(uint32_t n) {
    const uint32_t sort = 8 * sharedSortKeys(n), stage = 24 * (n < kStageBodies ? n : kStageBodies);
    return sort > stage ? sort : stage;
}

// What the block steps, in shared memory: some sixty pointers and numbers that
// every thread would otherwise hold in registers or reload from its stack
// (by value through the step's calls they cost 1.25x the adjoint's time).
struct BlockWorld {
    WorldParams<F> W;
    StateView<F> in, out;   // the step's start and end
    CacheView<F> cin, cout;
    StepScratch<F> sc;
    AdjointView<F> adj;
    unsigned char *dyn;     // sharedBytes(n) bytes, aligned to 16
    uint32_t scan[33];
    uint32_t pairs, colored, deferred, colors;
};

__device__ __forceinline__ uint32_t blockScan(uint32_t v, uint32_t &total, uint32_t *s) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += n;
    }
    if (lane == 31) s[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t x = lane < nw ? s[lane] : 0u;
        uint32_t xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t n = __shfl_up_sync(0xffffffffu, xi, o);
            if ((int)lane >= o) xi += n;
        }
        if (lane < nw) s[lane] = xi - x;
        if (lane == 31) s[32] = xi;
    }
    __syncthreads();
    const uint32_t r = s[warp] + incl - v;
    total = s[32];
    __syncthreads();
    return r;
}

using Key = unsigned long long;

// ------------------------------------------------------ manifold lane groups --
// Four lanes of a warp work on one manifold; lane p holds point p.  The whole
// warp takes part in every exchange (its eight groups run in step, those without
// a manifold idle): exchanges under one mask a group were issued one group after
// the other, which made a hand-over of the velocities eight times as long.
constexpr uint32_t kWarp = 0xffffffffu;
struct Group {
    uint32_t id, count;  // this group, groups of the block
    uint32_t p, first;   // lane in the group, the group's first lane in the warp
};
__device__ __forceinline__ Group laneGroup() {
    Group g;
    const uint32_t lane = threadIdx.x & 31;
    g.id = threadIdx.x >> 2;
    g.count = blockDim.x >> 2;
    g.p = lane & 3;
    g.first = lane & ~3u;
    return g;
}
__device__ __forceinline__ V3<F> shfl3(const V3<F> &v, uint32_t from) {
    return {__shfl_sync(kWarp, v.x, from), __shfl_sync(kWarp, v.y, from), __shfl_sync(kWarp, v.z, from)};
}
// The velocity part of s from lane `from` of each group.  dynA: some group of
// the warp has a moving body A (a static body's velocities stay as they are).
__device__ __forceinline__ void shareVelocities(const Group &g, PointIn<F> &s, uint32_t from, bool dynA) {
    const uint32_t l = g.first + from;
    if (dynA) {
        s.vA = shfl3(s.vA, l);
        s.wA = shfl3(s.wA, l);
    }
    s.vB = shfl3(s.vB, l);
    s.wB = shfl3(s.wB, l);
}
__device__ __forceinline__ F groupSum(F v) {
    v += __shfl_xor_sync(kWarp, v, 1);
    v += __shfl_xor_sync(kWarp, v, 2);
    return v;
}
__device__ __forceinline__ V3<F> groupSum(const V3<F> &v) {
    return {groupSum(v.x), groupSum(v.y), groupSum(v.z)};
}

// What a manifold's lanes need of it.
struct ManifoldLane {
    uint32_t k, kp, m, a, b, npts;
    bool sA, sB;
    F mu;
    V3<F> n;
};
__device__ __forceinline__ ManifoldLane loadManifold(const BlockWorld &bw, const Group &g, uint32_t k) {
    const StepScratch<F> &sc = bw.sc;
    ManifoldLane l;
    l.k = k;
    l.kp = 4 * k + g.p;
    l.m = sc.order[k];
    l.a = sc.mA[l.m];
    l.b = sc.mB[l.m];
    l.npts = sc.mCount[l.m];
    l.sA = bw.W.isStatic[l.a] != 0;
    l.sB = bw.W.isStatic[l.b] != 0;
    l.mu = sc.mMu[l.m];
    l.n = ld3(sc.mNormal, l.m);
    return l;
}
// Fields that lie apart by `stride` words.
template <int N> __device__ __forceinline__ void loadFields(F (&c)[N], const F *p, size_t stride, size_t i) {
#pragma unroll
    for (int e = 0; e < N; ++e) c[e] = p[e * stride + i];
}
template <int N> __device__ __forceinline__ void storeFields(const F (&c)[N], F *p, size_t stride, size_t i) {
#pragma unroll
    for (int e = 0; e < N; ++e) p[e * stride + i] = c[e];
}

// ------------------------------------------------------------------ prepare --
// One point (lane) of manifold l: its constants, the initial impulses, the
// matched cache entry (or -1) and the manifold's inertias and inverse masses.
struct PreparedLane {
    F c[kPreparedScalars];
    F lam[3];
    int32_t match;
    M3<F> IA, IB;
    F imA, imB;
};
__device__ __forceinline__ void prepareLane(const BlockWorld &bw, const ManifoldLane &l, const Group &g,
                                            PreparedLane &o) {
    const WorldParams<F> &W = bw.W;
    const StateView<F> &in = bw.in, &out = bw.out;
    const CacheView<F> &cin = bw.cin;
    const StepScratch<F> &sc = bw.sc;
    const Q<F> qA = ld4q(in.q, l.a), qB = ld4q(in.q, l.b);
    o.IA = inverseInertiaWorld(qA, W.iinv[3 * l.a], W.iinv[3 * l.a + 1], W.iinv[3 * l.a + 2]);
    o.IB = inverseInertiaWorld(qB, W.iinv[3 * l.b], W.iinv[3 * l.b + 1], W.iinv[3 * l.b + 2]);
    o.imA = inverseMass(l.sA, W.mass[l.a]);
    o.imB = inverseMass(l.sB, W.mass[l.b]);
#pragma unroll
    for (int e = 0; e < kPreparedScalars; ++e) o.c[e] = 0.0f;
    o.lam[0] = o.lam[1] = o.lam[2] = 0.0f;
    o.match = -1;
    if (g.p >= l.npts) return;
    // the cache range of the body pair (sequential_impulse_solver.cpp:448-456)
    const Key key = ((Key)l.a << 32) | l.b;
    const uint32_t cacheN = *cin.count;
    uint32_t lo = 0, hi = cacheN;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (cin.key[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    const V3<F> anA = ld3(sc.mAnchorA, 4 * l.m + g.p), anB = ld3(sc.mAnchorB, 4 * l.m + g.p);
    Prepared<F> pr;
    preparePoint(l.n, anA, anB, sc.mDepth[4 * l.m + g.p], qA, qB, o.IA, o.IB, o.imA, o.imB, ld3(out.v, l.a),
                 ld3(out.w, l.a), ld3(out.v, l.b), ld3(out.w, l.b), sc.mRest[l.m], 1.0f / smax(W.dt, 1e-6f), pr);
    preparedPack(pr, o.c);
    if (!pr.tangentValid || pr.iem <= 0.0f) return;
    const float matchSq = 0.05f * 0.05f;
    for (uint32_t e = lo; e < cacheN && cin.key[e] == key; ++e) {
        const V3<F> da = ld3(cin.anchorA, e) - anA, db = ld3(cin.anchorB, e) - anB;
        if (dot(da, da) > matchSq || dot(db, db) > matchSq) continue;
        warmClamp(l.mu, cin.lam[3 * e], cin.lam[3 * e + 1], cin.lam[3 * e + 2], o.lam[0], o.lam[1], o.lam[2]);
        o.match = (int32_t)e;
        break;
    }
}

// Velocities of a body pair (v, w: three floats a body, shared or global).
__device__ __forceinline__ void loadPair(const ManifoldLane &l, const F *v, const F *w, PointIn<F> &s) {
    s.vA = ld3(v, l.a);
    s.wA = ld3(w, l.a);
    s.vB = ld3(v, l.b);
    s.wB = ld3(w, l.b);
}
__device__ __forceinline__ void storePair(const ManifoldLane &l, F *v, F *w, const PointIn<F> &s) {
    if (!l.sA) {
        st3(v, l.a, s.vA);
        st3(w, l.a, s.wA);
    }
    if (!l.sB) {
        st3(v, l.b, s.vB);
        st3(w, l.b, s.wB);
    }
}

// The number of turns that the warp's points need, over its groups that act.
__device__ __forceinline__ uint32_t warpTurns(bool act, uint32_t npts) {
    return __reduce_max_sync(kWarp, act ? npts : 0u);
}

// Warm start of one manifold a group (warmStartPrepared :453-490): point after
// point.  act: the group has a manifold in this turn (whole warps call).
__device__ __forceinline__ void warmGroup(const Group &g, bool act, const ManifoldLane &l, const F *c, const F *lam,
                                          int32_t match, const M3<F> &IA, const M3<F> &IB, F imA, F imB, F *v, F *w) {
    const uint32_t matched = __ballot_sync(kWarp, act && g.p < l.npts && match >= 0);
    const bool any = ((matched >> g.first) & 0xFu) != 0;  // else the bodies are not written
    const uint32_t turns = warpTurns(any, l.npts);
    if (!turns) return;
    const bool dynA = __any_sync(kWarp, any && !l.sA);
    PointIn<F> s{};
    if (any) loadPair(l, v, w, s);
    for (uint32_t q = 0; q < turns; ++q) {
        if (g.p == q && ((matched >> (g.first + q)) & 1u)) {
            const V3<F> wi = l.n * lam[0] + pv(c, kPT1) * lam[1] + pv(c, kPT2) * lam[2];
            const V3<F> nw = -wi;
            if (!l.sA) {
                s.vA += nw * imA;
                s.wA += mul(IA, cross(pv(c, kPOffA), nw));
            }
            if (!l.sB) {
                s.vB += wi * imB;
                s.wB += mul(IB, cross(pv(c, kPOffB), wi));
            }
        }
        if (q + 1 < turns) shareVelocities(g, s, q, dynA);
    }
    if (any && g.p + 1 == turns) storePair(l, v, w, s);
}

// One velocity update of one manifold a group; tape (nullable): fields `stride`
// apart that take the manifold's velocities and impulses from before it.
__device__ __forceinline__ void solveGroup(const Group &g, bool act, const ManifoldLane &l, const F *c, F *lam, F imA,
                                           F imB, F *v, F *w, F *tape, size_t stride) {
    const uint32_t turns = warpTurns(act, l.npts);
    if (!turns) return;
    const bool dynA = __any_sync(kWarp, act && !l.sA);
    PointIn<F> s{};
    if (act) {
        loadPair(l, v, w, s);
        if (tape) {
            const V3<F> t = g.p == 0 ? s.vA : g.p == 1 ? s.wA : g.p == 2 ? s.vB : s.wB;
            F *o = tape + l.k;
            o[(3 * g.p) * stride] = t.x;
            o[(3 * g.p + 1) * stride] = t.y;
            o[(3 * g.p + 2) * stride] = t.z;
#pragma unroll
            for (uint32_t e = 0; e < 3; ++e) o[(12 + 3 * g.p + e) * stride] = lam[e];
        }
    }
    s.ln = lam[0];
    s.l1 = lam[1];
    s.l2 = lam[2];
    for (uint32_t q = 0; q < turns; ++q) {
        if (act && g.p == q && q < l.npts) pointForward(l.n, l.mu, c, imA, imB, l.sA, l.sB, s);
        if (q + 1 < turns) shareVelocities(g, s, q, dynA);
    }
    if (act) {
        lam[0] = s.ln;
        lam[1] = s.l1;
        lam[2] = s.l2;
        if (g.p + 1 == turns) storePair(l, v, w, s);
    }
}

// ------------------------------------------------------------------ forward --
// The step is two calls, so that the iterations' registers are not shared with
// the narrowphase's.
//
// Bodies to ordered manifolds, cache slots and (in v, w) velocities in front of
// the solve.
__device__ __noinline__ void contactsBlock(BlockWorld &bw) {
    const WorldParams<F> &W = bw.W;
    const StateView<F> &in = bw.in, &out = bw.out;
    const CacheView<F> &cout = bw.cout;
    const StepScratch<F> &sc = bw.sc;
    unsigned char *const dyn = bw.dyn;
    BlockWorld &sh = bw;
    const uint32_t tid = threadIdx.x, nt = blockDim.x, n = W.n;
    const uint32_t lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const uint32_t sortKeys = sharedSortKeys(n);
    Key *const shKeys = reinterpret_cast<Key *>(dyn);

    // 1. velocity integration, AABBs, sweep keys
    const uint32_t n2 = nextPow2u(n > 0 ? n : 1);
    Key *entries = n2 <= sortKeys ? shKeys : sc.bpEntries;
    for (uint32_t i = tid; i < n2; i += nt) {
        Key key = ~0ull;
        if (i < n) {
            st3(out.v, i, integratedVelocity(W, i, ld3(in.v, i)));
            st3(out.w, i, ld3(in.w, i));
            V3<F> mn, mx;
            bodyAabb(W, i, ld3(in.x, i), ld4q(in.q, i), mn, mx);
            st3(sc.aabb, 2 * i, mn);
            st3(sc.aabb, 2 * i + 1, mx);
            key = ((Key)adOrderedKey(mn.x) << 32) | i;
        }
        entries[i] = key;
    }
    if (tid == 0) {
        sh.pairs = 0;
        sc.counts[3] = 0;
    }
    blockChunkSort(entries, n2);

    // 2. sweep: a warp for each body, its lanes along the window (bodies sorted
    // by min.x up to the first whose min.x exceeds this body's max.x)
    for (uint32_t k = warp; k < n; k += nw) {
        const uint32_t i = (uint32_t)entries[k];
        const V3<F> amn = ld3(sc.aabb, 2 * i), amx = ld3(sc.aabb, 2 * i + 1);
        for (uint32_t k0 = k + 1; k0 < n; k0 += 32) {
            const uint32_t kk = k0 + lane;
            uint32_t j = 0;
            bool stop = true, hit = false;
            if (kk < n) {
                j = (uint32_t)entries[kk];
                const V3<F> bmn = ld3(sc.aabb, 2 * j), bmx = ld3(sc.aabb, 2 * j + 1);
                stop = bmn.x > amx.x;
                hit = amn.y <= bmx.y && amx.y >= bmn.y && amn.z <= bmx.z && amx.z >= bmn.z;
            }
            const uint32_t stops = __ballot_sync(0xffffffffu, stop);
            const uint32_t before = stops ? (stops & (0u - stops)) - 1u : 0xffffffffu;  // lanes ahead of the first stop
            const uint32_t hits = __ballot_sync(0xffffffffu, hit) & before;
            if (hits) {
                uint32_t slot = 0;
                if (lane == 0) slot = atomicAdd(&sh.pairs, (uint32_t)__popc(hits));
                slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(hits & ((1u << lane) - 1u));
                if (((hits >> lane) & 1u) && slot < W.maxPairs)
                    sc.bpPairs[slot] = ((Key)(i < j ? i : j) << 32) | (i < j ? j : i);
            }
            if (stops) break;
        }
    }
    __syncthreads();
    uint32_t P = sh.pairs;
    if (P > W.maxPairs) {
        if (tid == 0) sc.counts[3] |= kAdErrPairs;
        P = W.maxPairs;
    }
    const uint32_t P2 = nextPow2u(P > 0 ? P : 1);
    Key *pairs = sc.bpPairs;
    if (P2 <= sortKeys) {
        pairs = shKeys;
        for (uint32_t p = tid; p < P2; p += nt) pairs[p] = p < P ? sc.bpPairs[p] : ~0ull;
    } else {
        for (uint32_t p = P + tid; p < P2; p += nt) pairs[p] = ~0ull;
    }
    blockChunkSort(pairs, P2);

    // 3. narrowphase in pair order, manifolds compacted in that order
    uint32_t M = 0;
    for (uint32_t t0 = 0; t0 < P; t0 += nt) {
        const uint32_t p = t0 + tid;
        Contact<F> c;
        c.count = 0;
        bool hit = false;
        uint32_t a = 0, b = 0;
        if (p < P) {
            a = (uint32_t)(pairs[p] >> 32);
            b = (uint32_t)pairs[p];
            const Tf<F> tA{ld3(in.x, a), ld4q(in.q, a)}, tB{ld3(in.x, b), ld4q(in.q, b)};
            hit = contactPair<F>(W.shape[a], ld3(W.dims, a), tA, W.shape[b], ld3(W.dims, b), tB, c);
        }
        uint32_t cnt;
        const uint32_t m = M + blockScan(hit ? 1u : 0u, cnt, sh.scan);
        if (hit && m < W.maxManifolds) {
            sc.mA[m] = a;
            sc.mB[m] = b;
            sc.mCount[m] = c.count;
            st3(sc.mNormal, m, c.normal);
            sc.mRest[m] = smax(W.rest[a], W.rest[b]);
            sc.mMu[m] = ssqrt(smax(W.mu[a], 0.0f) * smax(W.mu[b], 0.0f));
            for (uint32_t k = 0; k < c.count; ++k) {
                st3(sc.mAnchorA, 4 * m + k, c.anchorA[k]);
                st3(sc.mAnchorB, 4 * m + k, c.anchorB[k]);
                sc.mDepth[4 * m + k] = c.depth[k];
                sc.mFeature[4 * m + k] = c.feature[k] | (c.axis << kAdAxisShift);
            }
        }
        M += cnt;
    }
    if (M > W.maxManifolds) {
        if (tid == 0) sc.counts[3] |= kAdErrManifolds;
        M = W.maxManifolds;
    }

    // 4. colouring: greedy in decreasing priority over manifolds that share a
    // dynamic body (the engine's colouring, in windows of kAdMaxColors colours:
    // a manifold whose neighbours use a whole window waits for the next one, in
    // which only the waiting manifolds take colours), in rounds.  A round
    // colours at least the highest priority left, so M rounds bound it.
    constexpr uint32_t kUncoloredM = 0xFFFFFFFFu, kDeferredM = 0xFFFFFFFEu;
    const bool staged = n <= kStageBodies;
    Key *best = staged ? shKeys : reinterpret_cast<Key *>(sc.aabb);  // the bounds are read no more
    Key *used = staged ? shKeys + n : sc.bodyUsed;
    __syncthreads();
    for (uint32_t i = tid; i < n; i += nt) best[i] = used[2 * i] = used[2 * i + 1] = 0ull;
    for (uint32_t m = tid; m < M; m += nt) sc.color[m] = kUncoloredM;
    if (tid == 0) {
        sh.colored = sh.deferred = sh.colors = 0;
        sc.counts[0] = P;
        sc.counts[1] = M;
    }
    __syncthreads();
    uint32_t base = 0;
    Key round = 0;
    for (uint32_t target = M; target;) {  // one window a turn
        while (sh.colored < target) {
            const Key stamp = ++round << 32;
            __syncthreads();
            for (uint32_t m = tid; m < M; m += nt) {
                if (sc.color[m] != kUncoloredM) continue;
                const Key pr = stamp | adColorPriority(m);
                const uint32_t a = sc.mA[m], b = sc.mB[m];
                if (!W.isStatic[a]) atomicMax(&best[a], pr);
                if (!W.isStatic[b]) atomicMax(&best[b], pr);
            }
            __syncthreads();
            uint32_t done = 0, top = 0, late = 0;
            for (uint32_t m = tid; m < M; m += nt) {
                if (sc.color[m] != kUncoloredM) continue;
                const Key pr = stamp | adColorPriority(m);
                const uint32_t a = sc.mA[m], b = sc.mB[m];
                const bool da = !W.isStatic[a], db = !W.isStatic[b];
                if ((da && *(volatile Key *)&best[a] != pr) || (db && *(volatile Key *)&best[b] != pr)) continue;
                Key u0 = 0, u1 = 0;
                if (da) {
                    u0 |= used[2 * a];
                    u1 |= used[2 * a + 1];
                }
                if (db) {
                    u0 |= used[2 * b];
                    u1 |= used[2 * b + 1];
                }
                ++done;
                if (!~u0 && !~u1) {
                    sc.color[m] = kDeferredM;
                    ++late;
                    continue;
                }
                const uint32_t local = ~u0 ? __ffsll((long long)~u0) - 1 : 64 + __ffsll((long long)~u1) - 1;
                const Key bit = 1ull << (local & 63);
                if (da) used[2 * a + (local >> 6)] |= bit;
                if (db) used[2 * b + (local >> 6)] |= bit;
                sc.color[m] = base + local;
                top = max(top, base + local + 1);
            }
            if (done) atomicAdd(&sh.colored, done);
            if (late) atomicAdd(&sh.deferred, late);
            if (top) atomicMax(&sh.colors, top);
            __syncthreads();
        }
        target = sh.deferred;
        __syncthreads();
        if (target) {
            base += kAdMaxColors;
            for (uint32_t i = tid; i < 2 * n; i += nt) used[i] = 0ull;
            for (uint32_t m = tid; m < M; m += nt)
                if (sc.color[m] == kDeferredM) sc.color[m] = kUncoloredM;
            if (tid == 0) sh.colored = sh.deferred = 0;
            __syncthreads();
        }
    }
    // order = (colour, index)
    const uint32_t C = sh.colors;
    if (tid == 0) {
        sc.counts[2] = C;
        sc.colorStart[C] = M;
    }
    if (C <= 1) {
        for (uint32_t k = tid; k < M; k += nt) sc.order[k] = sc.rank[k] = k;
        if (tid == 0 && C) sc.colorStart[0] = 0;
    } else {
        const uint32_t M2 = nextPow2u(M);
        Key *keys = M2 <= sortKeys ? shKeys : sc.sortKeys;
        __syncthreads();  // the masks are read no more
        for (uint32_t i = tid; i < M2; i += nt) keys[i] = i < M ? ((Key)sc.color[i] << 32) | i : ~0ull;
        blockChunkSort(keys, M2);
        for (uint32_t k = tid; k < M; k += nt) {
            const uint32_t m = (uint32_t)keys[k], ck = (uint32_t)(keys[k] >> 32);
            sc.order[k] = m;
            sc.rank[m] = k;
            if (k == 0 || (uint32_t)(keys[k - 1] >> 32) != ck) sc.colorStart[ck] = k;  // every colour is used
        }
    }
    __syncthreads();
    // cache slots: entries sorted by (body A, body B), which is manifold order
    uint32_t entryTotal = 0;
    for (uint32_t m0 = 0; m0 < M; m0 += nt) {
        const uint32_t m = m0 + tid, cnt = m < M ? sc.mCount[m] : 0u;
        uint32_t add;
        const uint32_t e = entryTotal + blockScan(cnt, add, sh.scan);
        if (m < M) {
            const uint32_t kp = 4 * sc.rank[m];
            for (uint32_t p = 0; p < 4; ++p) sc.cacheSlot[kp + p] = p < cnt && e + p < cout.cap ? e + p : kNoSlot;
        }
        entryTotal += add;
    }
    if (tid == 0) {
        if (entryTotal > cout.cap) sc.counts[3] |= kAdErrCache;
        *cout.count = entryTotal < cout.cap ? entryTotal : cout.cap;
    }
    // velocities into shared memory
    if (staged) {
        F *v = reinterpret_cast<F *>(dyn), *w = v + 3 * n;
        for (uint32_t i = tid; i < 3 * n; i += nt) {
            v[i] = out.v[i];
            w[i] = out.w[i];
        }
    }
    __syncthreads();
}

// Prepare, warm start, velocity iterations, warm-start cache.
__device__ __noinline__ void solveStepBlock(const BlockWorld &bw, bool record, F *v, F *w) {
    const WorldParams<F> &W = bw.W;
    const CacheView<F> &cout = bw.cout;
    const StepScratch<F> &sc = bw.sc;
    const uint32_t M = sc.counts[1], C = sc.counts[2];
    const Group g = laneGroup();
    const size_t K = W.maxManifolds, KP = 4 * K;
    const uint32_t rounds = (uint32_t)W.iterations;
    auto writeCache = [&](const ManifoldLane &l, const F *lam) {
        const uint32_t e = sc.cacheSlot[l.kp];
        if (e == kNoSlot) return;
        cout.key[e] = ((Key)l.a << 32) | l.b;
        st3(cout.anchorA, e, ld3(sc.mAnchorA, 4 * l.m + g.p));
        st3(cout.anchorB, e, ld3(sc.mAnchorB, 4 * l.m + g.p));
        st3(cout.lam, e, V3<F>{lam[0], lam[1], lam[2]});
    };
    auto keep = [&](const ManifoldLane &l, const PreparedLane &o) {
        storeFields(o.c, sc.pp, KP, l.kp);
        storeFields(o.lam, sc.lamInit, KP, l.kp);
        sc.match[l.kp] = o.match;
        const F *ia = &o.IA.m00, *ib = &o.IB.m00;
#pragma unroll
        for (uint32_t e = 0; e < 9; ++e) {  // the group's lanes share the manifold's fields
            if ((e & 3) == g.p) sc.pm[e * K + l.k] = ia[e];
            if (((e + 1) & 3) == g.p) sc.pm[(9 + e) * K + l.k] = ib[e];
        }
        if (g.p == 2) sc.pm[18 * K + l.k] = o.imA;
        if (g.p == 3) sc.pm[19 * K + l.k] = o.imB;
    };
    if (M <= g.count) {
        // a group for every manifold: its data stay in registers
        const bool live = g.id < M;
        ManifoldLane l{};
        PreparedLane o{};
        uint32_t color = 0;
        if (live) {
            l = loadManifold(bw, g, g.id);
            color = sc.color[l.m];
            prepareLane(bw, l, g, o);
            if (record) keep(l, o);
        }
        __syncthreads();  // every manifold has read the velocities
        for (uint32_t c = 0; c < C; ++c) {
            warmGroup(g, live && color == c, l, o.c, o.lam, o.match, o.IA, o.IB, o.imA, o.imB, v, w);
            __syncthreads();
        }
        for (uint32_t it = 0; it < rounds; ++it)
            for (uint32_t c = 0; c < C; ++c) {
                solveGroup(g, live && color == c, l, o.c, o.lam, o.imA, o.imB, v, w,
                           record ? sc.tape + it * (kTapeScalars * K) : nullptr, K);
                __syncthreads();
            }
        if (live) {
            if (record) storeFields(o.lam, sc.lam, KP, l.kp);
            writeCache(l, o.lam);
        }
    } else {
        for (uint32_t k = g.id; k < M; k += g.count) {
            const ManifoldLane l = loadManifold(bw, g, k);
            PreparedLane o;
            prepareLane(bw, l, g, o);
            keep(l, o);
            storeFields(o.lam, sc.lam, KP, l.kp);
        }
        __syncthreads();
        for (uint32_t pass = 0; pass < rounds + 1; ++pass)
            for (uint32_t c = 0; c < C; ++c) {
                const uint32_t end = sc.colorStart[c + 1];
                for (uint32_t k0 = sc.colorStart[c]; k0 < end; k0 += g.count) {
                    const bool act = k0 + g.id < end;  // a group past the end idles on the last manifold
                    const uint32_t k = act ? k0 + g.id : end - 1;
                    const ManifoldLane l = loadManifold(bw, g, k);
                    F cc[kPreparedScalars], lam[3];
                    loadFields(cc, sc.pp, KP, l.kp);
                    loadFields(lam, sc.lam, KP, l.kp);
                    const F imA = sc.pm[18 * K + k], imB = sc.pm[19 * K + k];
                    if (pass == 0) {
                        F ia[9], ib[9];
                        loadFields(ia, sc.pm, K, k);
                        loadFields(ib, sc.pm + 9 * K, K, k);
                        warmGroup(g, act, l, cc, lam, sc.match[l.kp], ldm(ia), ldm(ib), imA, imB, v, w);
                    } else {
                        solveGroup(g, act, l, cc, lam, imA, imB, v, w,
                                   record ? sc.tape + (pass - 1) * (kTapeScalars * K) : nullptr, K);
                        if (act) storeFields(lam, sc.lam, KP, l.kp);
                    }
                }
                __syncthreads();
            }
        for (uint32_t k = g.id; k < M; k += g.count) {
            const ManifoldLane l = loadManifold(bw, g, k);
            F lam[3];
            loadFields(lam, sc.lam, KP, l.kp);
            writeCache(l, lam);
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void forwardStepBlock(BlockWorld &bw, bool record) {
    const WorldParams<F> &W = bw.W;
    const StateView<F> &in = bw.in, &out = bw.out;
    const uint32_t tid = threadIdx.x, nt = blockDim.x, n = W.n;
    contactsBlock(bw);
    const bool staged = n <= kStageBodies;
    F *v = staged ? reinterpret_cast<F *>(bw.dyn) : out.v, *w = staged ? v + 3 * n : out.w;
    solveStepBlock(bw, record, v, w);
    // 8. pose integration
    for (uint32_t i = tid; i < n; i += nt) {
        V3<F> pos = ld3(in.x, i);
        Q<F> rot = ld4q(in.q, i);
        const V3<F> lin = ld3(v, i), ang = ld3(w, i);
        if (!W.isStatic[i]) poseForward(W.dt, lin, ang, pos, rot);
        st3(out.x, i, pos);
        st4q(out.q, i, rot);
        if (staged) {
            st3(out.v, i, lin);
            st3(out.w, i, ang);
        }
    }
    __syncthreads();
}

// ------------------------------------------------------------------ reverse --
// Adjoints that a lane gathers over the iterations.
struct AdjointLane {
    F ac[kPreparedScalars];
    F alam[3];
    V3<F> an;
    F amu, aimA, aimB;
};
constexpr int kAdjointExtra = 6;  // an, amu, aimA, aimB: kept with ac where a group takes several manifolds

// One velocity update of one manifold a group in reverse (act as above).  lam: the impulses before it,
// lamPost: after it; tape: the velocities before it.
__device__ __forceinline__ void reverseGroup(const Group &g, bool act, const ManifoldLane &l, const F *c,
                                             const F (&lam)[3], const F (&lamPost)[3], F imA, F imB, const F *tape,
                                             size_t stride, F *av, F *aw, AdjointLane &r) {
    const uint32_t turns = warpTurns(act, l.npts);
    const bool dynA = __any_sync(kWarp, act && !l.sA);
    // velocities in front of every point: the impulses' differences, applied as
    // the forward pass did
    PointIn<F> cur, in;
    {
        F t[12];
        loadFields(t, tape, stride, l.k);
        cur = PointIn<F>{pv(t, 0), pv(t, 1), pv(t, 2), pv(t, 3), lam[0], lam[1], lam[2]};
    }
    in = cur;
    const bool live = act && g.p < l.npts;
    for (uint32_t q = 0; q + 1 < turns; ++q) {
        if (g.p == q && live && !(c[kPIem] <= 0.0f)) {
            const F applied = lamPost[0] - lam[0];
            const V3<F> impulse = l.n * applied;
            if (!l.sA) {
                cur.vA += (-impulse) * imA;
                cur.wA += pv(c, kPNrA) * (-applied);
            }
            if (!l.sB) {
                cur.vB += impulse * imB;
                cur.wB += pv(c, kPNrB) * applied;
            }
            if (!(c[kPItm00] <= 0.0f || c[kPItm11] <= 0.0f)) {
                const F a1 = lamPost[1] - lam[1], a2 = lamPost[2] - lam[2];
                const V3<F> ti = pv(c, kPT1) * a1 + pv(c, kPT2) * a2;
                if (!l.sA) {
                    cur.vA += (-ti) * imA;
                    cur.wA += -(pv(c, kPTrA1) * a1 + pv(c, kPTrA2) * a2);
                }
                if (!l.sB) {
                    cur.vB += ti * imB;
                    cur.wB += pv(c, kPTrB1) * a1 + pv(c, kPTrB2) * a2;
                }
            }
        }
        shareVelocities(g, cur, q, dynA);
        if (g.p == q + 1) in = cur;
    }
    // the intermediates of all points at once
    PointMid<F> mid;
    mid.live = mid.fric = false;
    if (live) mid = pointMid(l.n, l.mu, c, in);
    // the adjoints, point after point
    PointIn<F> a{};
    if (act && !l.sA) {
        a.vA = ld3(av, l.a);
        a.wA = ld3(aw, l.a);
    }
    if (act && !l.sB) {
        a.vB = ld3(av, l.b);
        a.wB = ld3(aw, l.b);
    }
    a.ln = r.alam[0];
    a.l1 = r.alam[1];
    a.l2 = r.alam[2];
    PointAdj<F> adj{};
    for (int q = (int)turns - 1; q >= 0; --q) {
        if (g.p == (uint32_t)q && live) adj = pointChain(l.n, c, imA, imB, l.sA, l.sB, mid, a);
        if (q > 0) shareVelocities(g, a, (uint32_t)q, dynA);
    }
    if (act && g.p == 0) storePair(l, av, aw, a);
    if (live) {
        r.alam[0] = a.ln;
        r.alam[1] = a.l1;
        r.alam[2] = a.l2;
        pointAccumulate(l.n, l.mu, c, in, l.sA, l.sB, mid, adj, r.ac, r.an, r.amu, r.aimA, r.aimB);
    }
}

// Warm start, matching, preparation, geometry and materials of one manifold in
// reverse; body adjoints are added to with atomics (av, aw: where the
// velocities' adjoints stand; adj.dv, adj.dw: where new ones go, since other
// manifolds still read av, aw).
// A call, with its arguments by value: it needs twice the registers of the
// iterations, and what a call takes by reference leaves the registers.
__device__ __noinline__ void geometryGroup(const BlockWorld &bw, const F *av, const F *aw, const Group g, bool act,
                                           const ManifoldLane l, AdjointLane r) {
    const WorldParams<F> &W = bw.W;
    const StateView<F> &in = bw.in;
    const CacheView<F> &cin = bw.cin;
    const StepScratch<F> &sc = bw.sc;
    const AdjointView<F> &adj = bw.adj;
    const size_t K = W.maxManifolds, KP = 4 * K;
    const bool live = act && g.p < l.npts;
    F pm[kPmScalars], c[kPreparedScalars];
    loadFields(pm, sc.pm, K, l.k);
    loadFields(c, sc.pp, KP, l.kp);
    const M3<F> IA = ldm(pm), IB = ldm(pm + 9);
    const F imA = pm[18], imB = pm[19];
    PrepareGrad<F> gr{};
    Tf<F> gA{}, gB{};
    V3<F> gn{};
    const Tf<F> tA{ld3(in.x, l.a), ld4q(in.q, l.a)}, tB{ld3(in.x, l.b), ld4q(in.q, l.b)};
    const uint32_t shapeA = W.shape[l.a], shapeB = W.shape[l.b];
    if (live) {
        gr.n = r.an;
        gr.imA = r.aimA;
        gr.imB = r.aimB;
        const int32_t e = sc.match[l.kp];
        if (e >= 0) {
            F li[3];
            loadFields(li, sc.lamInit, KP, l.kp);
            V3<F> alam{r.alam[0], r.alam[1], r.alam[2]};
            warmReverse(l.n, c, V3<F>{li[0], li[1], li[2]}, IA, IB, imA, imB, l.sA, l.sB, ld3(av, l.a), ld3(aw, l.a),
                        ld3(av, l.b), ld3(aw, l.b), alam, r.ac, gr.n, gr.IA, gr.IB, gr.imA, gr.imB);
            const V3<F> o = warmClampReverse(l.mu, cin.lam[3 * e], cin.lam[3 * e + 1], cin.lam[3 * e + 2], alam, r.amu);
            atomicAdd(&adj.acache[3 * e], o.x);
            atomicAdd(&adj.acache[3 * e + 1], o.y);
            atomicAdd(&adj.acache[3 * e + 2], o.z);
        }
        const uint32_t mp = 4 * l.m + g.p;
        preparePointReverse(l.n, ld3(sc.mAnchorA, mp), ld3(sc.mAnchorB, mp), sc.mDepth[mp], tA.q, tB.q, IA, IB, imA + imB,
                            integratedVelocity(W, l.a, ld3(in.v, l.a)), ld3(in.w, l.a),
                            integratedVelocity(W, l.b, ld3(in.v, l.b)), ld3(in.w, l.b), sc.mRest[l.m],
                            1.0f / smax(W.dt, 1e-6f), c, r.ac, gr);
        gn = gr.n;
        contactPointReverse(shapeA, ld3(W.dims, l.a), tA, shapeB, ld3(W.dims, l.b), tB, l.n, sc.mFeature[mp],
                            PointGrad<F>{gr.anchorA, gr.anchorB, gr.depth}, gn, gA, gB);
        inverseInertiaAdj(tA.q, ld3(W.iinv, l.a), gr.IA, gr.qA);
        inverseInertiaAdj(tB.q, ld3(W.iinv, l.b), gr.IB, gr.qB);
    }
    gn = groupSum(gn);
    if (act && g.p == 0 && shapeA == 1 && shapeB == 1)
        boxNormalReverse(tA, tB, (sc.mFeature[4 * l.m] & kAdAxisMask) >> kAdAxisShift, l.n, gn, gA, gB);
    // sums over the points; lane 0 and 1 add body A's, 2 and 3 body B's
    const F rest = groupSum(gr.rest), amu = groupSum(live ? r.amu : 0.0f);
    auto body = [&](uint32_t i, bool isStatic, bool low, const Tf<F> &t, const Q<F> &gq, const V3<F> &lin,
                    const V3<F> &ang, F aim, F im) {
        const V3<F> x = groupSum(t.p), dv = groupSum(lin), dw = groupSum(ang);
        const F qx = groupSum(t.q.x + gq.x), qy = groupSum(t.q.y + gq.y), qz = groupSum(t.q.z + gq.z),
                qw = groupSum(t.q.w + gq.w), m = groupSum(aim);
        if (isStatic) return;
        if (low) {
            atomicAdd(&adj.ax[3 * i], x.x);
            atomicAdd(&adj.ax[3 * i + 1], x.y);
            atomicAdd(&adj.ax[3 * i + 2], x.z);
            atomicAdd(&adj.aq[4 * i], qx);
            atomicAdd(&adj.aq[4 * i + 1], qy);
            atomicAdd(&adj.aq[4 * i + 2], qz);
            atomicAdd(&adj.aq[4 * i + 3], qw);
        } else {
            atomicAdd(&adj.dv[3 * i], dv.x);
            atomicAdd(&adj.dv[3 * i + 1], dv.y);
            atomicAdd(&adj.dv[3 * i + 2], dv.z);
            atomicAdd(&adj.dw[3 * i], dw.x);
            atomicAdd(&adj.dw[3 * i + 1], dw.y);
            atomicAdd(&adj.dw[3 * i + 2], dw.z);
            atomicAdd(&adj.amass[i], -(m * im * im));  // im = 1 / mass
        }
    };
    body(l.a, !act || l.sA || g.p > 1, g.p == 0, gA, gr.qA, gr.linA, gr.angA, gr.imA, imA);
    body(l.b, !act || l.sB || g.p < 2, g.p == 2, gB, gr.qB, gr.linB, gr.angB, gr.imB, imB);
    if (act && g.p == 0) {
        // restitution = max(ra, rb), friction = sqrt(max(fa, 0) * max(fb, 0))
        if (W.rest[l.a] < W.rest[l.b]) {
            if (!l.sB) atomicAdd(&adj.arest[l.b], rest);
        } else if (!l.sA) {
            atomicAdd(&adj.arest[l.a], rest);
        }
        if (l.mu > 0.0f) {
            const F fa = smax(W.mu[l.a], 0.0f), fb = smax(W.mu[l.b], 0.0f);
            const F h = amu * (0.5f / l.mu);
            if (!l.sA && !(W.mu[l.a] < 0.0f)) atomicAdd(&adj.amu[l.a], h * fb);
            if (!l.sB && !(W.mu[l.b] < 0.0f)) atomicAdd(&adj.amu[l.b], h * fa);
        }
    }
}

// last: the step is the rollout's last (its impulses have no adjoint);
// otherwise adj.acache holds the adjoint of the step's output cache on entry.
// It holds that of the input cache on exit.
__device__ __noinline__ void backwardStepBlock(const BlockWorld &bw, bool last) {
    const WorldParams<F> &W = bw.W;
    const StateView<F> &in = bw.in, &out = bw.out;
    const CacheView<F> &cin = bw.cin;
    const StepScratch<F> &sc = bw.sc;
    const AdjointView<F> &adj = bw.adj;
    const uint32_t tid = threadIdx.x, nt = blockDim.x, n = W.n;
    const uint32_t M = sc.counts[1], C = sc.counts[2];
    const size_t K = W.maxManifolds, KP = 4 * K;
    const Group g = laneGroup();
    const bool resident = M <= g.count;  // a group for every manifold
    const bool staged = n <= kStageBodies;
    F *av = staged ? reinterpret_cast<F *>(bw.dyn) : adj.av, *aw = staged ? av + 3 * n : adj.aw;
    // 1. pose integration; adjoints of the velocities into shared memory
    for (uint32_t i = tid; i < n; i += nt) {
        V3<F> v = ld3(adj.av, i), w = ld3(adj.aw, i);
        if (!W.isStatic[i]) {
            Q<F> aq = ld4q(adj.aq, i);
            poseReverse(W.dt, ld4q(in.q, i), ld3(out.w, i), ld3(adj.ax, i), aq, v, w);
            st4q(adj.aq, i, aq);
        }
        st3(av, i, v);
        st3(aw, i, w);
        st3(adj.dv, i, V3<F>{0.0f, 0.0f, 0.0f});
        st3(adj.dw, i, V3<F>{0.0f, 0.0f, 0.0f});
    }
    // adjoints of the final impulses
    auto finalImpulses = [&](uint32_t kp, F (&alam)[3]) {
        const uint32_t e = last ? kNoSlot : sc.cacheSlot[kp];
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) alam[j] = e == kNoSlot ? 0.0f : adj.acache[3 * e + j];
    };
    const uint32_t cacheN = *cin.count;
    ManifoldLane l{};
    AdjointLane r{};
    uint32_t color = 0;
    const bool live = g.id < M;
    auto clear = [&](AdjointLane &x) {
#pragma unroll
        for (int e = 0; e < kPreparedScalars; ++e) x.ac[e] = 0.0f;
        x.an = V3<F>{0.0f, 0.0f, 0.0f};
        x.amu = x.aimA = x.aimB = 0.0f;
    };
    // where a group takes several manifolds, its adjoints wait in memory
    auto loadAdjoint = [&](uint32_t kp, AdjointLane &x) {
        loadFields(x.ac, adj.app, KP, kp);
        loadFields(x.alam, adj.alam, KP, kp);
        F ex[kAdjointExtra];
        loadFields(ex, adj.aext, KP, kp);
        x.an = V3<F>{ex[0], ex[1], ex[2]};
        x.amu = ex[3];
        x.aimA = ex[4];
        x.aimB = ex[5];
    };
    auto storeAdjoint = [&](uint32_t kp, const AdjointLane &x) {
        storeFields(x.ac, adj.app, KP, kp);
        storeFields(x.alam, adj.alam, KP, kp);
        const F ex[kAdjointExtra] = {x.an.x, x.an.y, x.an.z, x.amu, x.aimA, x.aimB};
        storeFields(ex, adj.aext, KP, kp);
    };
    if (resident) {
        if (live) {
            l = loadManifold(bw, g, g.id);
            color = sc.color[l.m];
            clear(r);
            finalImpulses(l.kp, r.alam);
        }
    } else {
        for (uint32_t k = g.id; k < M; k += g.count) {
            AdjointLane x;
            clear(x);
            finalImpulses(4 * k + g.p, x.alam);
            storeAdjoint(4 * k + g.p, x);
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < 3 * cacheN; i += nt) adj.acache[i] = 0.0f;
    __syncthreads();
    // 2. velocity iterations in reverse
    for (int it = W.iterations - 1; it >= 0; --it) {
        const F *tape = sc.tape + (size_t)it * (kTapeScalars * K);
        const bool lastIt = it + 1 == W.iterations;
        auto one = [&](bool act, const ManifoldLane &ml, AdjointLane &x) {
            F c[kPreparedScalars], lam[3], lamPost[3];
            loadFields(c, sc.pp, KP, ml.kp);
            loadFields(lam, tape + (12 + 3 * g.p) * K, K, ml.k);
            if (lastIt) loadFields(lamPost, sc.lam, KP, ml.kp);
            else loadFields(lamPost, tape + (kTapeScalars + 12 + 3 * g.p) * K, K, ml.k);
            reverseGroup(g, act, ml, c, lam, lamPost, sc.pm[18 * K + ml.k], sc.pm[19 * K + ml.k], tape, K, av, aw, x);
        };
        for (int ci = (int)C - 1; ci >= 0; --ci) {
            if (resident) {
                const bool act = live && color == (uint32_t)ci;
                if (__any_sync(kWarp, act)) one(act, l, r);
            } else {
                const uint32_t end = sc.colorStart[ci + 1];
                for (uint32_t k0 = sc.colorStart[ci]; k0 < end; k0 += g.count) {
                    const bool act = k0 + g.id < end;
                    const ManifoldLane ml = loadManifold(bw, g, act ? k0 + g.id : end - 1);
                    AdjointLane x;
                    loadAdjoint(ml.kp, x);
                    one(act, ml, x);
                    if (act) storeAdjoint(ml.kp, x);
                }
            }
            __syncthreads();
        }
    }
    // 3. warm start, matching, preparation, geometry, materials
    if (resident) {
        if (__any_sync(kWarp, live)) geometryGroup(bw, av, aw, g, live, l, r);
    } else {
        for (uint32_t k0 = 0; k0 < M; k0 += g.count) {
            const bool act = k0 + g.id < M;
            const ManifoldLane ml = loadManifold(bw, g, act ? k0 + g.id : M - 1);
            AdjointLane x;
            loadAdjoint(ml.kp, x);
            geometryGroup(bw, av, aw, g, act, ml, x);
        }
    }
    __syncthreads();
    // 4. velocity integration passes the adjoints on
    for (uint32_t i = tid; i < n; i += nt) {
        st3(adj.av, i, ld3(av, i) + ld3(adj.dv, i));
        st3(adj.aw, i, ld3(aw, i) + ld3(adj.dw, i));
    }
    __syncthreads();
}

} // namespace ad
} // namespace pe
