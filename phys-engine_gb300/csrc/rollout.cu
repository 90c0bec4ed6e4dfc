// GPU differentiable rollout (rollout.h): device layout, the forward and the
// adjoint kernels, and the host driver.
#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>

#include "ad_block.cuh"
#include "rollout.h"

namespace pe {
namespace {

using namespace ad;
__host__ __device__ constexpr size_t align16(size_t v) { return (v + 15) & ~size_t(15); }

// Byte offsets inside one world's slot of the arena.
struct Layout {
    // snapshots (checkpoints first, then the segment's states)
    size_t snap0, snapStride;
    size_t sState, sCount, sKey, sA, sB, sLam;  // within a snapshot
    // step scratch (one per step of a segment)
    size_t scr0, scrStride;
    size_t aabb, mA, mB, mCount, mFeature, mNormal, mMu, mRest, mAnchorA, mAnchorB, mDepth, color, order, rank,
        sortKeys, bodyUsed, colorStart, pp, pm, lam, lamInit, match, tape, cacheSlot, counts;
    // adjoints
    size_t ax, aq, av, aw, alam, app, aext, acache, amass, amu, arest, dv, dw;
    // broadphase sort buffers, shared by the steps (not part of any record)
    size_t bpEntries, bpPairs;
    size_t stride;
};

__host__ __device__ Layout makeLayout(uint32_t nMax, uint32_t maxPairs, uint32_t maxM, int iterations, uint32_t nSnap,
                                      uint32_t nScr) {
    Layout L{};
    const uint32_t cap = 4 * maxM;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o = align16(o + bytes);
        return at;
    };
    L.sState = take(sizeof(F) * 13 * nMax);
    L.sCount = take(sizeof(uint32_t));
    L.sKey = take(sizeof(unsigned long long) * cap);
    L.sA = take(sizeof(F) * 3 * cap);
    L.sB = take(sizeof(F) * 3 * cap);
    L.sLam = take(sizeof(F) * 3 * cap);
    L.snapStride = o;
    o = 0;
    L.aabb = take(sizeof(F) * 6 * nMax);
    L.mA = take(4ull * maxM);
    L.mB = take(4ull * maxM);
    L.mCount = take(4ull * maxM);
    L.mFeature = take(16ull * maxM);
    L.mNormal = take(sizeof(F) * 3 * maxM);
    L.mMu = take(sizeof(F) * maxM);
    L.mRest = take(sizeof(F) * maxM);
    L.mAnchorA = take(sizeof(F) * 12 * maxM);
    L.mAnchorB = take(sizeof(F) * 12 * maxM);
    L.mDepth = take(sizeof(F) * 4 * maxM);
    L.color = take(4ull * maxM);
    L.order = take(4ull * maxM);
    L.rank = take(4ull * maxM);
    L.sortKeys = take(8ull * maxM);
    L.bodyUsed = take(16ull * nMax);
    L.colorStart = take(4ull * (maxM + 1));
    L.pp = take(sizeof(F) * 4 * maxM * kPreparedScalars);
    L.pm = take(sizeof(F) * maxM * kPmScalars);
    L.lam = take(sizeof(F) * 12 * maxM);
    L.lamInit = take(sizeof(F) * 12 * maxM);
    L.match = take(16ull * maxM);
    L.tape = take(sizeof(F) * (size_t)(iterations > 0 ? iterations : 1) * maxM * kTapeScalars);
    L.cacheSlot = take(4ull * cap);
    L.counts = take(16);
    L.scrStride = o;
    o = 0;
    L.snap0 = take(L.snapStride * nSnap);
    L.scr0 = take(L.scrStride * nScr);
    L.ax = take(sizeof(F) * 3 * nMax);
    L.aq = take(sizeof(F) * 4 * nMax);
    L.av = take(sizeof(F) * 3 * nMax);
    L.aw = take(sizeof(F) * 3 * nMax);
    L.alam = take(sizeof(F) * 12 * maxM);
    L.app = take(sizeof(F) * 4 * maxM * kPreparedScalars);
    L.aext = take(sizeof(F) * 4 * maxM * kAdjointExtra);
    L.acache = take(sizeof(F) * 3 * cap);
    L.amass = take(sizeof(F) * nMax);
    L.amu = take(sizeof(F) * nMax);
    L.arest = take(sizeof(F) * nMax);
    L.dv = take(sizeof(F) * 3 * nMax);
    L.dw = take(sizeof(F) * 3 * nMax);
    L.bpEntries = take(8ull * ad::nextPow2u(nMax > 0 ? nMax : 1));
    L.bpPairs = take(8ull * ad::nextPow2u(maxPairs > 0 ? maxPairs : 1));
    L.stride = o;
    return L;
}

// Capacities of a world of n bodies: candidate pairs, manifolds (a power of
// two), and its slot of the arena, sized for those.
__host__ __device__ inline uint32_t worldMaxPairs(uint32_t n) { return 8 * n + 64; }
// quarterPerBody: manifold capacity in quarter manifolds per body (8 = two
// per body, enough for boxes resting on one another).
__host__ __device__ inline uint32_t worldMaxManifolds(uint32_t n, uint32_t quarterPerBody) {
    const uint64_t need = ((uint64_t)quarterPerBody * n + 3) / 4 + 32;
    uint32_t m = 1;
    while (m < need) m <<= 1;
    return m;
}

struct Args {
    unsigned char *arena;
    const unsigned long long *worldOff;  // byte offset of each world's slot in the arena
    const uint32_t *order;               // worlds in the order blocks take them (largest first)
    const uint32_t *bodyStart;           // worlds + 1
    const uint8_t *shape, *isStatic;
    const F *dims, *iinv, *mass, *mu, *rest;
    uint32_t worlds, steps, ckEvery, nCk, quarterPerBody;
    int iterations;
    F gx, gy, gz, dt;
    uint32_t *queueHead;
    uint32_t *err;  // per world
};

// One world's slot: its layout (sized by its own body count) and base address.
struct Slot {
    Layout L;
    unsigned char *base;
    uint32_t maxPairs, maxM;
};
__device__ __forceinline__ Slot slotOf(const Args &a, uint32_t w) {
    const uint32_t n = a.bodyStart[w + 1] - a.bodyStart[w];
    Slot s;
    s.maxPairs = worldMaxPairs(n);
    s.maxM = worldMaxManifolds(n, a.quarterPerBody);
    s.L = makeLayout(n, s.maxPairs, s.maxM, a.iterations, a.nCk + a.ckEvery + 1, a.ckEvery);
    s.base = a.arena + a.worldOff[w];
    return s;
}

template <class P> __device__ __forceinline__ P *at(unsigned char *base, size_t off) {
    return reinterpret_cast<P *>(base + off);
}

struct Snap {
    ad::StateView<F> s;
    ad::CacheView<F> c;
};
__device__ __forceinline__ Snap snapshot(const Slot &ws, uint32_t j, uint32_t n) {
    unsigned char *p = ws.base + ws.L.snap0 + ws.L.snapStride * j;
    F *st = at<F>(p, ws.L.sState);
    Snap r;
    r.s = ad::StateView<F>{st, st + 3 * n, st + 7 * n, st + 10 * n};
    r.c = ad::CacheView<F>{at<uint32_t>(p, ws.L.sCount), at<unsigned long long>(p, ws.L.sKey), at<F>(p, ws.L.sA),
                       at<F>(p, ws.L.sB), at<F>(p, ws.L.sLam), 4 * ws.maxM};
    return r;
}
__device__ __forceinline__ StepScratch<F> scratch(const Slot &ws, uint32_t j) {
    unsigned char *p = ws.base + ws.L.scr0 + ws.L.scrStride * j;
    const Layout &L = ws.L;
    StepScratch<F> s;
    s.aabb = at<F>(p, L.aabb);
    s.mA = at<uint32_t>(p, L.mA);
    s.mB = at<uint32_t>(p, L.mB);
    s.mCount = at<uint32_t>(p, L.mCount);
    s.mFeature = at<uint32_t>(p, L.mFeature);
    s.mNormal = at<F>(p, L.mNormal);
    s.mMu = at<F>(p, L.mMu);
    s.mRest = at<F>(p, L.mRest);
    s.mAnchorA = at<F>(p, L.mAnchorA);
    s.mAnchorB = at<F>(p, L.mAnchorB);
    s.mDepth = at<F>(p, L.mDepth);
    s.color = at<uint32_t>(p, L.color);
    s.order = at<uint32_t>(p, L.order);
    s.rank = at<uint32_t>(p, L.rank);
    s.sortKeys = at<unsigned long long>(p, L.sortKeys);
    s.bodyUsed = at<unsigned long long>(p, L.bodyUsed);
    s.colorStart = at<uint32_t>(p, L.colorStart);
    s.pp = at<F>(p, L.pp);
    s.pm = at<F>(p, L.pm);
    s.lam = at<F>(p, L.lam);
    s.lamInit = at<F>(p, L.lamInit);
    s.match = at<int32_t>(p, L.match);
    s.tape = at<F>(p, L.tape);
    s.cacheSlot = at<uint32_t>(p, L.cacheSlot);
    s.counts = at<uint32_t>(p, L.counts);
    s.bpEntries = at<unsigned long long>(ws.base, L.bpEntries);
    s.bpPairs = at<unsigned long long>(ws.base, L.bpPairs);
    return s;
}

__device__ __forceinline__ WorldParams<F> params(const Args &a, uint32_t w, const Slot &ws) {
    const uint32_t b = a.bodyStart[w];
    WorldParams<F> W;
    W.n = a.bodyStart[w + 1] - b;
    W.shape = a.shape + b;
    W.isStatic = a.isStatic + b;
    W.dims = a.dims + 3 * b;
    W.iinv = a.iinv + 3 * b;
    W.mass = a.mass + b;
    W.mu = a.mu + b;
    W.rest = a.rest + b;
    W.gx = a.gx;
    W.gy = a.gy;
    W.gz = a.gz;
    W.dt = a.dt;
    W.iterations = a.iterations;
    W.maxPairs = ws.maxPairs;
    W.maxManifolds = ws.maxM;
    return W;
}

__device__ __forceinline__ uint32_t nextWorld(const Args &a) {
    __shared__ uint32_t s_w;
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t i = atomicAdd(a.queueHead, 1u);
        s_w = i < a.worlds ? a.order[i] : a.worlds;
    }
    __syncthreads();
    return s_w;
}

// The block's next world: its slot, parameters and adjoint arrays (thread 0
// writes them for all).  False when no world is left.
__device__ __noinline__ bool takeWorld(const Args &a, Slot &ws, BlockWorld &bw, unsigned char *dyn, uint32_t &world) {
    const uint32_t w = nextWorld(a);
    if (w >= a.worlds) return false;
    if (threadIdx.x == 0) {
        ws = slotOf(a, w);
        bw.W = params(a, w, ws);
        bw.dyn = dyn;
        const Layout &L = ws.L;
        unsigned char *p = ws.base;
        bw.adj = AdjointView<F>{};
        bw.adj.ax = at<F>(p, L.ax);
        bw.adj.aq = at<F>(p, L.aq);
        bw.adj.av = at<F>(p, L.av);
        bw.adj.aw = at<F>(p, L.aw);
        bw.adj.alam = at<F>(p, L.alam);
        bw.adj.app = at<F>(p, L.app);
        bw.adj.aext = at<F>(p, L.aext);
        bw.adj.acache = at<F>(p, L.acache);
        bw.adj.amass = at<F>(p, L.amass);
        bw.adj.amu = at<F>(p, L.amu);
        bw.adj.arest = at<F>(p, L.arest);
        bw.adj.dv = at<F>(p, L.dv);
        bw.adj.dw = at<F>(p, L.dw);
    }
    world = w;
    __syncthreads();
    return true;
}

// The step from snapshot `from` to snapshot `to` with scratch `j`.  The barrier ahead of
// the write lets every thread finish with the last step's record: without it a late warp
// read the error word of a record whose step had not run.
__device__ __noinline__ void setStep(const Slot &ws, BlockWorld &bw, uint32_t from, uint32_t to, uint32_t j) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const Snap in = snapshot(ws, from, bw.W.n), out = snapshot(ws, to, bw.W.n);
        bw.in = in.s;
        bw.cin = in.c;
        bw.out = out.s;
        bw.cout = out.c;
        bw.sc = scratch(ws, j);
    }
    __syncthreads();
}

// Forward: steps every world, keeps a checkpoint every ckEvery steps (and the
// final state), writes the final state.
template <int T, int B>
__global__ void __launch_bounds__(T, B) k_rollout_forward(const __grid_constant__ Args a, const F *x0, const F *q0,
                                                          const F *v0, const F *w0, F *xT, F *qT, F *vT, F *wT) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ BlockWorld bw;
    __shared__ Slot ws;
    uint32_t w;
    while (takeWorld(a, ws, bw, s_dyn, w)) {
        const uint32_t n = bw.W.n;
        const size_t b = a.bodyStart[w];
        {
            const Snap s = snapshot(ws, 0, n);
            for (uint32_t i = threadIdx.x; i < 3 * n; i += blockDim.x) {
                s.s.x[i] = x0[3 * b + i];
                s.s.v[i] = v0[3 * b + i];
                s.s.w[i] = w0[3 * b + i];
            }
            for (uint32_t i = threadIdx.x; i < 4 * n; i += blockDim.x) s.s.q[i] = q0[4 * b + i];
            if (threadIdx.x == 0) *s.c.count = 0;
        }
        bool failed = false;
        uint32_t cur = 0;
        for (uint32_t t = 0; t < a.steps && !failed; ++t) {
            // a checkpoint's step writes the checkpoint itself
            const uint32_t s = t + 1;
            const bool keep = s % a.ckEvery == 0 || s == a.steps;
            const uint32_t next = keep ? (s + a.ckEvery - 1) / a.ckEvery : a.nCk + (t & 1);
            setStep(ws, bw, cur, next, 0);
            forwardStepBlock(bw, false);
            const uint32_t err = bw.sc.counts[3];
            if (err) {
                if (threadIdx.x == 0) atomicOr(&a.err[w], err);
                failed = true;
            }
            cur = next;
        }
        if (failed) continue;
        const Snap s = snapshot(ws, cur, n);
        for (uint32_t i = threadIdx.x; i < 3 * n; i += blockDim.x) {
            xT[3 * b + i] = s.s.x[i];
            vT[3 * b + i] = s.s.v[i];
            wT[3 * b + i] = s.s.w[i];
        }
        for (uint32_t i = threadIdx.x; i < 4 * n; i += blockDim.x) qT[4 * b + i] = s.s.q[i];
    }
}

// Adjoint: per segment (last first) recompute from the checkpoint with the
// tape, then reverse step by step.
template <int T, int B>
__global__ void __launch_bounds__(T, B) k_rollout_backward(const __grid_constant__ Args a, const F *gx, const F *gq,
                                                           const F *gv, const F *gw, F *gx0, F *gq0, F *gv0, F *gw0,
                                                           F *gmass, F *gmu, F *grest) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ BlockWorld bw;
    __shared__ Slot ws;
    uint32_t w;
    while (takeWorld(a, ws, bw, s_dyn, w)) {
        const uint32_t n = bw.W.n;
        const size_t b = a.bodyStart[w];
        const AdjointView<F> &adj = bw.adj;
        for (uint32_t i = threadIdx.x; i < 3 * n; i += blockDim.x) {
            adj.ax[i] = gx ? gx[3 * b + i] : 0.0f;
            adj.av[i] = gv ? gv[3 * b + i] : 0.0f;
            adj.aw[i] = gw ? gw[3 * b + i] : 0.0f;
        }
        for (uint32_t i = threadIdx.x; i < 4 * n; i += blockDim.x) adj.aq[i] = gq ? gq[4 * b + i] : 0.0f;
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) adj.amass[i] = adj.amu[i] = adj.arest[i] = 0.0f;
        const uint32_t nSeg = (a.steps + a.ckEvery - 1) / a.ckEvery;
        bool failed = false;
        for (int s = (int)nSeg - 1; s >= 0 && !failed; --s) {
            const uint32_t t0 = (uint32_t)s * a.ckEvery;
            const uint32_t L = min(a.steps, t0 + a.ckEvery) - t0;
            // state i of the segment: its checkpoint, then the recomputed steps
            auto state = [&](uint32_t i) { return i == 0 ? (uint32_t)s : a.nCk + i; };
            for (uint32_t i = 0; i < L && !failed; ++i) {
                setStep(ws, bw, state(i), state(i + 1), i);
                forwardStepBlock(bw, true);
                const uint32_t err = bw.sc.counts[3];
                if (err) {
                    if (threadIdx.x == 0) atomicOr(&a.err[w], err);
                    failed = true;
                }
            }
            for (int i = (int)L - 1; i >= 0 && !failed; --i) {
                setStep(ws, bw, state((uint32_t)i), state((uint32_t)i + 1), (uint32_t)i);
                backwardStepBlock(bw, t0 + (uint32_t)i + 1 == a.steps);
            }
        }
        if (failed) continue;
        for (uint32_t i = threadIdx.x; i < 3 * n; i += blockDim.x) {
            if (gx0) gx0[3 * b + i] = adj.ax[i];
            if (gv0) gv0[3 * b + i] = adj.av[i];
            if (gw0) gw0[3 * b + i] = adj.aw[i];
        }
        if (gq0)
            for (uint32_t i = threadIdx.x; i < 4 * n; i += blockDim.x) gq0[4 * b + i] = adj.aq[i];
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
            if (gmass) gmass[b + i] = adj.amass[i];
            if (gmu) gmu[b + i] = adj.amu[i];
            if (grest) grest[b + i] = adj.arest[i];
        }
    }
}

// Block size and register budget.  With more work for an SM than its largest
// world (bodies over SMs above the largest count) the SMs stay full: two blocks
// of 256 threads an SM at 128 registers, or four of 128 where a world has at
// most 33 bodies (32 manifolds a block at once).  Otherwise the longest world
// decides, and a block takes the registers it wants.  Measured, forward +
// adjoint, ms: 1,024 worlds of 64 boxes 5.4 + 16.7 at two blocks, 8.0 + 20.3 at
// one; 8 worlds of 33 boxes 0.94 + 2.30 and 0.90 + 1.97; 512 worlds of 16 to
// 1,024 bodies 2.21 + 3.83 and 2.03 + 3.84.
constexpr uint32_t kSmallWorld = 33;
using ForwardKernel = void (*)(Args, const F *, const F *, const F *, const F *, F *, F *, F *, F *);
using BackwardKernel = void (*)(Args, const F *, const F *, const F *, const F *, F *, F *, F *, F *, F *, F *, F *);

// Blocks that the device holds at once, at most one a world.
template <class Kernel> uint32_t residentBlocks(Kernel k, int threads, size_t smem, uint32_t worlds, int device) {
    int sms = 0, per = 0;
    PE_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    PE_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, threads, smem));
    return std::min<uint32_t>(worlds, (uint32_t)(std::max(1, per) * sms));
}

template <class T> void uploadVec(DeviceArray<T> &d, const std::vector<T> &h) {
    d.reserve(h.size());
    if (!h.empty()) PE_CHECK(cudaMemcpy(d.ptr, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
}

} // namespace

Rollout::Rollout(int device) : device_(device) {
    PE_CHECK(cudaSetDevice(device_));
    PE_CHECK(cudaEventCreate(&e0_));
    PE_CHECK(cudaEventCreate(&e1_));
    PE_CHECK(cudaMallocHost(&hostErr_, sizeof(uint32_t)));
}

Rollout::~Rollout() {
    if (e0_) cudaEventDestroy(e0_);
    if (e1_) cudaEventDestroy(e1_);
    if (hostErr_) cudaFreeHost(hostErr_);
}

void Rollout::create(const std::vector<uint32_t> &worldBodies, const std::vector<uint8_t> &shape,
                     const std::vector<uint8_t> &isStatic, const std::vector<float> &halfExtents,
                     const std::vector<float> &invInertia, uint32_t steps, float dt, int iterations,
                     uint32_t checkpointEvery) {
    PE_CHECK(cudaSetDevice(device_));
    if (worldBodies.empty()) throw std::invalid_argument("a rollout needs at least one world");
    if (steps == 0) throw std::invalid_argument("a rollout needs at least one step");
    if (checkpointEvery == 0) throw std::invalid_argument("checkpoint interval must be positive");
    if (iterations < 0 || iterations > 256) throw std::invalid_argument("iterations out of range");
    uint64_t total = 0;
    nMax_ = 0;
    std::vector<uint32_t> start(worldBodies.size() + 1, 0);
    for (size_t w = 0; w < worldBodies.size(); ++w) {
        if (worldBodies[w] == 0 || worldBodies[w] > kRolloutMaxBodies)
            throw std::invalid_argument("a differentiable world holds 1 to " + std::to_string(kRolloutMaxBodies) +
                                        " bodies");
        start[w] = (uint32_t)total;
        total += worldBodies[w];
        nMax_ = std::max(nMax_, worldBodies[w]);
    }
    start.back() = (uint32_t)total;
    if (shape.size() != total || isStatic.size() != total || halfExtents.size() != 3 * total ||
        invInertia.size() != 3 * total)
        throw std::invalid_argument("per-body arrays must hold the sum of the world body counts");
    for (uint8_t s : shape)
        if (s > 1) throw std::invalid_argument("differentiable worlds hold spheres and boxes");
    nb_ = total;
    worldBodies_ = worldBodies;
    steps_ = steps;
    dt_ = dt;
    iterations_ = iterations;
    ckEvery_ = std::min(checkpointEvery, steps);
    nCk_ = (steps + ckEvery_ - 1) / ckEvery_ + 1;
    // worlds are taken largest first
    std::vector<uint32_t> order(worldBodies.size());
    for (size_t w = 0; w < order.size(); ++w) order[w] = (uint32_t)w;
    std::stable_sort(order.begin(), order.end(),
                     [&](uint32_t x, uint32_t y) { return worldBodies[x] > worldBodies[y]; });
    uploadVec(order_, order);
    uploadVec(bodyStart_, start);
    uploadVec(shape_, shape);
    uploadVec(static_, isStatic);
    uploadVec(dims_, halfExtents);
    uploadVec(iinv_, invInertia);
    mass_.reserve(total);
    mu_.reserve(total);
    rest_.reserve(total);
    queue_.reserve(1);
    err_.reserve(worldBodies.size());
    arena_.release();
    haveForward_ = false;
}

void Rollout::setManifoldCapacity(float perBody) {
    if (!(perBody >= 0.25f && perBody <= 64.0f))
        throw std::invalid_argument("manifold capacity must be 0.25 to 64 manifolds per body");
    const uint32_t q = (uint32_t)(perBody * 4.0f + 0.5f);
    if (q == quarterPerBody_) return;
    quarterPerBody_ = q;
    arena_.release();  // laid out again at the next forward call
    haveForward_ = false;
}

// Every world's slot is sized by its own body count (checkpoints, one
// segment's step scratch and tape, adjoints), allocated at the first forward
// call after creation or a capacity change.
void Rollout::ensureArena() {
    if (arena_.ptr) return;
    std::vector<unsigned long long> off(worldBodies_.size());
    unsigned long long arenaBytes = 0;
    for (size_t w = 0; w < worldBodies_.size(); ++w) {
        const uint32_t n = worldBodies_[w];
        const Layout L = makeLayout(n, worldMaxPairs(n), worldMaxManifolds(n, quarterPerBody_), iterations_,
                                    nCk_ + ckEvery_ + 1, ckEvery_);
        off[w] = arenaBytes;
        arenaBytes += align16(L.stride);
    }
    uploadVec(worldOff_, off);
    arena_.reserve(arenaBytes);
    bytes_ = arenaBytes + nb_ * 64;
}

void Rollout::checkErrors(cudaStream_t s, const char *what) {
    std::vector<uint32_t> e(worldBodies_.size());
    PE_CHECK(cudaMemcpyAsync(e.data(), err_.ptr, e.size() * 4, cudaMemcpyDeviceToHost, s));
    PE_CHECK(cudaStreamSynchronize(s));
    for (size_t w = 0; w < e.size(); ++w)
        if (e[w]) {
            const uint32_t b = e[w];
            const char *m = (b & kAdErrPairs)       ? "candidate pairs exceed the world's capacity"
                            : (b & kAdErrManifolds) ? "contact manifolds exceed the world's capacity"
                                                    : "warm-start cache overflow";
            throw std::runtime_error(std::string(what) + ": world " + std::to_string(w) + ": " + m);
        }
}

void Rollout::forward(const float *x0, const float *q0, const float *v0, const float *w0, const float *mass,
                      const float *friction, const float *restitution, float *xT, float *qT, float *vT, float *wT,
                      cudaStream_t s) {
    PE_CHECK(cudaSetDevice(device_));
    if (!x0 || !q0 || !v0 || !w0 || !mass || !friction || !restitution || !xT || !qT || !vT || !wT)
        throw std::invalid_argument("null argument");
    ensureArena();
    PE_CHECK(cudaMemcpyAsync(mass_.ptr, mass, nb_ * 4, cudaMemcpyDeviceToDevice, s));
    PE_CHECK(cudaMemcpyAsync(mu_.ptr, friction, nb_ * 4, cudaMemcpyDeviceToDevice, s));
    PE_CHECK(cudaMemcpyAsync(rest_.ptr, restitution, nb_ * 4, cudaMemcpyDeviceToDevice, s));
    PE_CHECK(cudaMemsetAsync(queue_.ptr, 0, 4, s));
    PE_CHECK(cudaMemsetAsync(err_.ptr, 0, worldBodies_.size() * 4, s));
    Args a{};
    a.arena = arena_.ptr;
    a.quarterPerBody = quarterPerBody_;
    a.worldOff = worldOff_.ptr;
    a.order = order_.ptr;
    a.bodyStart = bodyStart_.ptr;
    a.shape = shape_.ptr;
    a.isStatic = static_.ptr;
    a.dims = dims_.ptr;
    a.iinv = iinv_.ptr;
    a.mass = mass_.ptr;
    a.mu = mu_.ptr;
    a.rest = rest_.ptr;
    a.worlds = (uint32_t)worldBodies_.size();
    a.steps = steps_;
    a.ckEvery = ckEvery_;
    a.nCk = nCk_;
    a.iterations = iterations_;
    a.gx = gravity[0];
    a.gy = gravity[1];
    a.gz = gravity[2];
    a.dt = dt_;
    a.queueHead = queue_.ptr;
    a.err = err_.ptr;
    const bool full = nb_ > (uint64_t)nMax_ * smCount(), small = full && nMax_ <= kSmallWorld;
    const ForwardKernel kernel = small  ? k_rollout_forward<128, 4>
                                 : full ? k_rollout_forward<256, 2>
                                        : k_rollout_forward<256, 1>;
    const int threads = small ? 128 : 256;
    const size_t smem = sharedBytes(nMax_);
    const uint32_t blocks = residentBlocks(kernel, threads, smem, a.worlds, device_);
    PE_CHECK(cudaEventRecord(e0_, s));
    kernel<<<blocks, threads, smem, s>>>(a, x0, q0, v0, w0, xT, qT, vT, wT);
    PE_LAUNCHED();
    PE_CHECK(cudaEventRecord(e1_, s));
    checkErrors(s, "rollout forward");
    float ms = 0;
    PE_CHECK(cudaEventElapsedTime(&ms, e0_, e1_));
    fwdMs_ = ms;
    haveForward_ = true;
}

void Rollout::backward(const float *gx, const float *gq, const float *gv, const float *gw, float *gx0, float *gq0,
                       float *gv0, float *gw0, float *gmass, float *gfriction, float *grestitution, cudaStream_t s) {
    PE_CHECK(cudaSetDevice(device_));
    if (!haveForward_) throw std::invalid_argument("backward needs a forward call first");
    PE_CHECK(cudaMemsetAsync(queue_.ptr, 0, 4, s));
    PE_CHECK(cudaMemsetAsync(err_.ptr, 0, worldBodies_.size() * 4, s));
    Args a{};
    a.arena = arena_.ptr;
    a.quarterPerBody = quarterPerBody_;
    a.worldOff = worldOff_.ptr;
    a.order = order_.ptr;
    a.bodyStart = bodyStart_.ptr;
    a.shape = shape_.ptr;
    a.isStatic = static_.ptr;
    a.dims = dims_.ptr;
    a.iinv = iinv_.ptr;
    a.mass = mass_.ptr;
    a.mu = mu_.ptr;
    a.rest = rest_.ptr;
    a.worlds = (uint32_t)worldBodies_.size();
    a.steps = steps_;
    a.ckEvery = ckEvery_;
    a.nCk = nCk_;
    a.iterations = iterations_;
    a.gx = gravity[0];
    a.gy = gravity[1];
    a.gz = gravity[2];
    a.dt = dt_;
    a.queueHead = queue_.ptr;
    a.err = err_.ptr;
    const bool full = nb_ > (uint64_t)nMax_ * smCount(), small = full && nMax_ <= kSmallWorld;
    const BackwardKernel kernel = small  ? k_rollout_backward<128, 4>
                                  : full ? k_rollout_backward<256, 2>
                                         : k_rollout_backward<256, 1>;
    const int threads = small ? 128 : 256;
    const size_t smem = sharedBytes(nMax_);
    const uint32_t blocks = residentBlocks(kernel, threads, smem, a.worlds, device_);
    PE_CHECK(cudaEventRecord(e0_, s));
    kernel<<<blocks, threads, smem, s>>>(a, gx, gq, gv, gw, gx0, gq0, gv0, gw0, gmass, gfriction, grestitution);
    PE_LAUNCHED();
    PE_CHECK(cudaEventRecord(e1_, s));
    checkErrors(s, "rollout backward");
    float ms = 0;
    PE_CHECK(cudaEventElapsedTime(&ms, e0_, e1_));
    bwdMs_ = ms;
}

} // namespace pe
