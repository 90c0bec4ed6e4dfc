// BroadPhaseAlgorithm::DynamicTree on the device: a linear BVH rebuilt every
// step.  The reference keeps an incremental AABB tree with fattened node bounds
// (src/collision/dynamic_aabb_tree.cpp) and reports every leaf pair whose tight
// bounds overlap, sorted lexicographically (:276-327) — the same pair set as
// sweep-and-prune, so only the way it is found differs here:
//
//   k_lbvh_bounds : bounds of the AABB centres (ordered-float atomics)
//   k_lbvh_codes  : 30-bit Morton code of each centre, key = code << b | index
//                   (unique keys), then a radix sort of the keys
//   k_lbvh_build  : binary radix tree over the sorted keys (Karras, "Maximizing
//                   Parallelism in the Construction of BVHs, Octrees, and k-d
//                   Trees", HPG 2012): one thread per internal node finds its
//                   range and split from common-prefix lengths
//   k_lbvh_refit  : node bounds bottom-up (the second child to arrive at a node
//                   unites both children, writes the node's record and climbs on)
//   k_lbvh_front  : the four above in one block for up to kFrontMax boxes
//   k_lbvh_pairs  : two to eight lanes per leaf walk the tree with its AABB and emit
//                   the overlapping leaves of a higher size class, and of its
//                   own class those after it in sorted order (each pair once),
//                   touching counting as overlap (Aabb::overlaps)
//
// The size class decides who reports a pair because a walk is serial: a floor
// that every body touches found its n partners in one thread (686 us of a
// 1,179 us step of 1,501 bodies over a floor; the step takes 531 us when each
// body finds the floor).  A class spans a factor of four, so boxes of similar size keep the
// rule of the sorted order, which prunes half of the tree.
//
// The emitted pairs are ordered by lists (k_broad.cu): in one block for a small world,
// over the grid where collider i is on body i; otherwise they go through the common
// finalize (sort, mapping to collider slots, same-body filter).
//
// What bounds a small tree is latency, in a dozen launches and in chains of loads.
// Measured on 1,501 bodies over a floor (us, profiled launch by launch): bounds,
// codes, sort, tree and node bounds in eleven launches 85, in one block 36; the
// walk with a thread a leaf and two dependent loads a node 103, with eight lanes a
// leaf and one 64-byte record a node 17; pair order from a sort of 64-bit keys 41,
// from lists 19.  The step went from 380 to 242; with 12,259 mixed bodies (eleven
// launches, few pairs) from 222 to 168, with 100,000 from 330 to 305.
#include "pe_block.cuh"
#include "pe_kernels.cuh"
#include "pe_math.cuh"
#include "pe_prims.cuh"
#include "pe_stages.h"

namespace pe {

namespace {

constexpr int kLbvhThreads = 256;
constexpr uint32_t kLeafBit = 0x80000000u;

inline int lbvhGrid(uint32_t n) {
    uint32_t b = (n + kLbvhThreads - 1) / kLbvhThreads;
    const uint32_t maxGrid = 8u * (uint32_t)smCount();
    return (int)(b ? (b < maxGrid ? b : maxGrid) : 1u);
}

__device__ __forceinline__ float orderedFloatDecode(uint32_t k) {
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    return __uint_as_float(u);
}

// Spreads the low 10 bits of v to every third bit.
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
    uint32_t r = 0;
#pragma unroll
    for (int b = 0; b < 10; ++b) r |= ((v >> b) & 1u) << (3 * b);
    return r;
}

__device__ __forceinline__ bool boxOverlap(const float4 &amn, const float4 &amx, const float4 &bmn, const float4 &bmx) {
    // Aabb::overlaps (include/phys/collision/aabb.hpp:15-19)
    return amn.x <= bmx.x && amx.x >= bmn.x && amn.y <= bmx.y && amx.y >= bmn.y && amn.z <= bmx.z && amx.z >= bmn.z;
}

// Reporting order of sorted leaf l: its box's size class (the exponent of the
// extents' sum over two, a factor of four a class; NaN counts as infinite, so every
// pair has one reporter) above the leaf's index, shifted to 24 bits.
__device__ __forceinline__ uint32_t reportKey(const float4 &mn, const float4 &mx, uint32_t l, uint32_t shift) {
    const float e = (mx.x - mn.x) + (mx.y - mn.y) + (mx.z - mn.z);
    const uint32_t u = __float_as_uint(e) & 0x7FFFFFFFu;
    return (u < 0x7F800000u ? u : 0x7F800000u) >> 24 << 24 | l >> shift;
}

// Bounds of two boxes, the higher of their reporting keys in mx.w.
__device__ __forceinline__ void unite(const float4 (&mn)[2], const float4 (&mx)[2], float4 &omn, float4 &omx) {
    omn = make_float4(INFINITY, INFINITY, INFINITY, 0.0f);
    omx = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.0f);
    uint32_t top = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        omn = make_float4(fminf(omn.x, mn[k].x), fminf(omn.y, mn[k].y), fminf(omn.z, mn[k].z), 0.0f);
        omx = make_float4(fmaxf(omx.x, mx[k].x), fmaxf(omx.y, mx[k].y), fmaxf(omx.z, mx[k].z), 0.0f);
        top = max(top, __float_as_uint(mx[k].w));
    }
    omx.w = __uint_as_float(top);
}

// A node's record: both children's bounds in one 64-byte line, the child (leaf
// children flagged) in mn.w, the highest reporting key below it in mx.w.
__device__ __forceinline__ void uniteChildren(const float4 (&mn)[2], const float4 (&mx)[2], const uint32_t (&c)[2],
                                              float4 *rec, float4 &omn, float4 &omx) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        rec[2 * k] = make_float4(mn[k].x, mn[k].y, mn[k].z, __uint_as_float(c[k]));
        rec[2 * k + 1] = mx[k];
    }
    unite(mn, mx, omn, omx);
}

// Common-prefix length of sorted keys i and j; -1 outside [0, n).
__device__ __forceinline__ int prefixLen(const unsigned long long *keys, uint32_t n, int i, int j) {
    if (j < 0 || j >= (int)n) return -1;
    return __clzll(keys[i] ^ keys[j]);
}

} // namespace

// box[0..2] = ordered-float minima of the centres, box[3..5] maxima.
__global__ void k_lbvh_init(uint32_t *box) {
    if (threadIdx.x < 3) box[threadIdx.x] = 0xFFFFFFFFu;
    else if (threadIdx.x < 6) box[threadIdx.x] = 0u;
}

__global__ void k_lbvh_bounds(BroadInput in, uint32_t *box) {
    const uint32_t n = *in.d_n;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = in.mn[i], b = in.mx[i];
        const float c[3] = {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], c[k]);
            hi[k] = fmaxf(hi[k], c[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    }
    if ((threadIdx.x & 31) == 0 && lo[0] <= hi[0]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            atomicMin(&box[k], orderedFloatKey(lo[k]));
            atomicMax(&box[3 + k], orderedFloatKey(hi[k]));
        }
    }
}

// Morton key of a box's centre (10 bits per axis) above the index bits.
__device__ __forceinline__ unsigned long long mortonKey(const float4 &a, const float4 &b, const float (&lo)[3],
                                                        const float (&scale)[3], uint32_t indexBits, uint32_t i) {
    const float c[3] = {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float t = fminf(fmaxf((c[k] - lo[k]) * scale[k], 0.0f), 1023.0f);  // NaN -> 0
        q[k] = (uint32_t)t;
    }
    const uint32_t code = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
    return ((unsigned long long)code << indexBits) | i;
}

__global__ void k_lbvh_codes(BroadInput in, const uint32_t *box, unsigned long long *keys, uint32_t indexBits,
                             uint32_t *counts) {
    const uint32_t n = *in.d_n;
    float lo[3], scale[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = orderedFloatDecode(box[k]);
        const float ext = orderedFloatDecode(box[3 + k]) - lo[k];
        scale[k] = ext > 0.0f ? 1024.0f / ext : 0.0f;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        keys[i] = mortonKey(in.mn[i], in.mx[i], lo, scale, indexBits, i);
        if (counts) counts[i] = 0u;  // for the walk's pairs
    }
}

// Internal node i of n - 1 over the sorted keys: the leaves lo .. hi it covers,
// gamma the last of the left child's.
__device__ __forceinline__ void nodeSplit(const unsigned long long *keys, uint32_t n, int i, int &lo, int &hi,
                                          int &gamma) {
    const int d = prefixLen(keys, n, i, i + 1) - prefixLen(keys, n, i, i - 1) > 0 ? 1 : -1;
    const int dmin = prefixLen(keys, n, i, i - d);
    int lmax = 2;
    while (prefixLen(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int s = lmax >> 1; s >= 1; s >>= 1)
        if (prefixLen(keys, n, i, i + (l + s) * d) > dmin) l += s;
    const int j = i + l * d;
    const int dnode = prefixLen(keys, n, i, j);
    int split = 0;
    for (int s = (l + 1) >> 1;; s = (s + 1) >> 1) {
        if (prefixLen(keys, n, i, i + (split + s) * d) > dnode) split += s;
        if (s == 1) break;
    }
    gamma = i + split * d + (d < 0 ? -1 : 0);
    lo = i < j ? i : j;
    hi = i < j ? j : i;
}

// Children (leaf children flagged with kLeafBit) and parents of the internal
// nodes, and the sorted leaves' bounds (reporting key in leafMx.w).
__global__ void k_lbvh_build(BroadInput in, const unsigned long long *keys, uint32_t indexBits, uint32_t *childL,
                             uint32_t *childR, uint32_t *parent, uint32_t *leafParent, uint32_t *visit,
                             float4 *leafMn, float4 *leafMx) {
    const uint32_t n = *in.d_n, shift = indexBits > 24 ? indexBits - 24 : 0;
    const unsigned long long idxMask = (1ull << indexBits) - 1ull;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const uint32_t idx = (uint32_t)(keys[t] & idxMask);
        leafMn[t] = in.mn[idx];
        float4 mx = in.mx[idx];
        mx.w = __uint_as_float(reportKey(in.mn[idx], mx, t, shift));
        leafMx[t] = mx;
        if (t + 1 >= n) continue;
        visit[t] = 0u;
        int lo, hi, gamma;
        nodeSplit(keys, n, (int)t, lo, hi, gamma);
        const bool leafL = lo == gamma, leafR = hi == gamma + 1;
        childL[t] = (leafL ? kLeafBit : 0u) | (uint32_t)gamma;
        childR[t] = (leafR ? kLeafBit : 0u) | (uint32_t)(gamma + 1);
        (leafL ? leafParent : parent)[gamma] = t;
        (leafR ? leafParent : parent)[gamma + 1] = t;
    }
}

// Node records from the leaves up; the second arrival at a node unites both
// children: its own bounds, which it carries, and the sibling's, from the sibling's
// record (published before the arrival counter moves).  What bounds it is traffic
// and the fences (300,000 leaves 71 us; 80 with bounds of the nodes kept beside the
// records, 57 before there were records).
__global__ void k_lbvh_refit(const uint32_t *d_n, const uint32_t *childL, const uint32_t *childR,
                             const uint32_t *parent, const uint32_t *leafParent, uint32_t *visit, const float4 *leafMn,
                             const float4 *leafMx, float4 *rec) {
    const uint32_t n = *d_n;
    if (n < 2) return;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        uint32_t node = leafParent[t], from = kLeafBit | t;
        float4 ownMn = leafMn[t], ownMx = leafMx[t];  // of the child that this thread comes from
        for (uint32_t depth = 0; depth < n; ++depth) {
            __threadfence();
            if (atomicAdd(&visit[node], 1u) == 0u) break;  // the sibling finishes this node
            __threadfence();
            const uint32_t c[2] = {childL[node], childR[node]};
            const bool second = c[1] == from;
            const uint32_t other = second ? c[0] : c[1], l = other & ~kLeafBit;
            float4 mn[2], mx[2];
            if (other & kLeafBit) {
                mn[0] = leafMn[l];
                mx[0] = leafMx[l];
            } else {  // the sibling's bounds are those of its record's two children
                const float4 *r = rec + 4 * (size_t)l;
                const float4 a = __ldcg(r), b = __ldcg(r + 1), e = __ldcg(r + 2), f = __ldcg(r + 3);
                const float4 cmn[2] = {a, e}, cmx[2] = {b, f};
                unite(cmn, cmx, mn[0], mx[0]);
            }
            mn[1] = second ? ownMn : mn[0];
            mx[1] = second ? ownMx : mx[0];
            if (!second) {
                mn[0] = ownMn;
                mx[0] = ownMx;
            }
            uniteChildren(mn, mx, c, rec + 4 * (size_t)node, ownMn, ownMx);
            if (node == 0) break;
            from = node;
            node = parent[node];
        }
    }
}

// Bounds, codes, sort, tree and node bounds of up to kFrontMax boxes in one
// block: keys, links (16 bits) and node bounds in shared memory.
constexpr uint32_t kFrontMax = 4 * kRegSortThreads;
constexpr uint32_t kLeafBit16 = 0x8000u;
constexpr size_t frontBytes(uint32_t N) { return (size_t)N * (2 * 8 + 32) + N / 8; }

template <int E>
__global__ void __launch_bounds__(kRegSortThreads)
k_lbvh_front(BroadInput in, unsigned long long *keys, uint32_t indexBits, float4 *leafMn, float4 *leafMx,
             float4 *rec) {
    constexpr uint32_t N = kRegSortThreads * E;
    extern __shared__ __align__(16) unsigned char s_front[];
    float4 *sMn = reinterpret_cast<float4 *>(s_front), *sMx = sMn + N;
    unsigned long long *sKeys = reinterpret_cast<unsigned long long *>(sMx + N), *sTmp = sKeys + N;
    uint16_t *sL = reinterpret_cast<uint16_t *>(sTmp), *sR = sL + N, *sParent = sR + N, *sLeafParent = sParent + N;
    uint32_t *sVisit = reinterpret_cast<uint32_t *>(sTmp + N);
    __shared__ float s_box[6][32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n = min(*in.d_n, N);  // the host launches this for at most N boxes
    float4 a[E], b[E];
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, scale[3];
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const uint32_t i = tid * E + r;
        if (i >= n) continue;
        a[r] = in.mn[i];
        b[r] = in.mx[i];
        const float c[3] = {(a[r].x + b[r].x) * 0.5f, (a[r].y + b[r].y) * 0.5f, (a[r].z + b[r].z) * 0.5f};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], c[k]);
            hi[k] = fmaxf(hi[k], c[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
        if (lane == 0) {
            s_box[k][warp] = lo[k];
            s_box[3 + k][warp] = hi[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = s_box[k][lane];
        hi[k] = s_box[3 + k][lane];
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
        const float ext = hi[k] - lo[k];
        scale[k] = ext > 0.0f ? 1024.0f / ext : 0.0f;
    }
    unsigned long long v[E];
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const uint32_t i = tid * E + r;
        v[r] = i < n ? mortonKey(a[r], b[r], lo, scale, indexBits, i) : ~0ull;
    }
    blockRegisterSort<unsigned long long, E>(v, sKeys, sTmp);
    __syncthreads();  // the last shared-memory stage's reads are done
    const unsigned long long idxMask = (1ull << indexBits) - 1ull;
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const uint32_t t = tid * E + r;
        sKeys[t] = v[r];
        if (t >= n) continue;
        keys[t] = v[r];
        const uint32_t idx = (uint32_t)(v[r] & idxMask);
        const float4 mn = in.mn[idx];
        float4 mx = in.mx[idx];
        mx.w = __uint_as_float(reportKey(mn, mx, t, 0));
        leafMn[t] = mn;
        leafMx[t] = mx;
    }
    for (uint32_t i = tid; i < N / 32; i += kRegSortThreads) sVisit[i] = 0u;
    __syncthreads();
    for (uint32_t t = tid; t + 1 < n; t += kRegSortThreads) {
        int first, last, gamma;
        nodeSplit(sKeys, n, (int)t, first, last, gamma);
        const bool leafL = first == gamma, leafR = last == gamma + 1;
        sL[t] = (uint16_t)((leafL ? kLeafBit16 : 0u) | (uint32_t)gamma);
        sR[t] = (uint16_t)((leafR ? kLeafBit16 : 0u) | (uint32_t)(gamma + 1));
        (leafL ? sLeafParent : sParent)[gamma] = (uint16_t)t;
        (leafR ? sLeafParent : sParent)[gamma + 1] = (uint16_t)t;
    }
    __syncthreads();
    if (n < 2) return;
    for (uint32_t t = tid; t < n; t += kRegSortThreads) {
        uint32_t node = sLeafParent[t];
        for (uint32_t depth = 0; depth < n; ++depth) {
            __threadfence_block();
            const uint32_t bit = 1u << (node & 31);
            if (!(atomicOr(&sVisit[node >> 5], bit) & bit)) break;  // the sibling finishes this node
            __threadfence_block();
            const uint32_t link[2] = {sL[node], sR[node]};
            uint32_t c[2];
            float4 mn[2], mx[2], omn, omx;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t l = link[k] & ~kLeafBit16;
                const bool leaf = (link[k] & kLeafBit16) != 0;
                c[k] = leaf ? kLeafBit | l : l;
                mn[k] = leaf ? leafMn[l] : sMn[l];
                mx[k] = leaf ? leafMx[l] : sMx[l];
            }
            uniteChildren(mn, mx, c, rec + 4 * (size_t)node, omn, omx);
            sMn[node] = omn;
            sMx[node] = omx;
            if (node == 0) break;
            node = sParent[node];
        }
    }
}

// Walks are long and uneven, and each step waits for its node's record: up to eight
// lanes a leaf take as many nodes off the leaf's stack at a time, and 64-thread
// blocks spread the leaves of a small world over the SMs.  Once the leaves fill the chip,
// lanes that find no node on the stack take the place of other leaves: a leaf then has
// four lanes, or two.  Broadphase in us with eight, four and two lanes: 20,000 mixed bodies
// 116, 112, 117, of a settled field 142, 147, 166; 40,000 135, 125, 128 and 190, 183, 202;
// 66,000 159, 144, 141 and 230, 215, 214; a falling field of 140,000 218, 177, 160 (a
// thread a leaf in the kernel before the lanes 199), of 300,000 388, 293, 250 (247).
constexpr int kLbvhWalkThreads = 64;
// Stack of a leaf: with fewer than kTreeDepth free entries beyond what a round can
// push, one node is taken at a time, and what that pushes is at most the tree's depth
// (a key has 30 + index bits).
constexpr uint32_t kTreeDepth = 64;
constexpr uint32_t kWalkThreadsPerSm = 1536;  // three quarters of what an SM holds

// Leaf t's AABB against the tree; pairs with the leaves of a higher size class
// and the later leaves of its own.
template <uint32_t kWalkLanes>
__global__ void __launch_bounds__(kLbvhWalkThreads)
k_lbvh_pairs(const uint32_t *d_n, const unsigned long long *keys, uint32_t indexBits, const float4 *leafMn,
             const float4 *leafMx, const float4 *rec, unsigned long long *pkeys, uint32_t cap, uint32_t bits,
             uint32_t *counts, uint32_t *ranks, DevStats *st) {
    constexpr uint32_t kWalkLeaves = kLbvhWalkThreads / kWalkLanes, kWalkStack = kTreeDepth + 16 * kWalkLanes;
    constexpr uint32_t kWalkMask = (1u << kWalkLanes) - 1u;
    __shared__ uint32_t s_stack[kWalkLeaves][kWalkStack + kWalkLanes];  // (rows on different banks)
    const uint32_t n = *d_n;
    if (n < 2) return;
    const unsigned long long idxMask = (1ull << indexBits) - 1ull;
    const uint32_t lane = threadIdx.x & 31, p = lane & (kWalkLanes - 1), shift = lane & ~(kWalkLanes - 1);
    const uint32_t leaf = threadIdx.x / kWalkLanes;
    uint32_t *stack = s_stack[leaf];
    const uint32_t below = (1u << p) - 1u;
    for (uint32_t t0 = blockIdx.x * kWalkLeaves; t0 < n; t0 += gridDim.x * kWalkLeaves) {
        const uint32_t t = t0 + leaf, tt = t < n ? t : n - 1;
        const float4 qmn = leafMn[tt], qmx = leafMx[tt];
        const uint32_t qk = __float_as_uint(qmx.w), qc = qk >> 24, qi = (uint32_t)(keys[tt] & idxMask);
        uint32_t sp = t < n ? 1u : 0u, pops = 0;
        __syncwarp();
        if (p == 0) stack[0] = 0u;
        __syncwarp();
        while (__any_sync(0xffffffffu, sp > 0)) {
            const uint32_t room = kWalkStack - kTreeDepth;
            const uint32_t k = min(min(sp, kWalkLanes), sp < room - kWalkLanes ? kWalkLanes : 1u);
            const bool act = p < k;
            const uint32_t node = act ? stack[sp - 1 - p] : 0u;
            sp -= k;
            __syncwarp();
            bool push[2] = {false, false}, hit[2] = {false, false};
            uint32_t c[2] = {0u, 0u};
            if (act) {
                const float4 *r = rec + 4 * (size_t)node;
                const float4 b[4] = {r[0], r[1], r[2], r[3]};
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint32_t id = __float_as_uint(b[2 * e].w), key = __float_as_uint(b[2 * e + 1].w);
                    c[e] = id & ~kLeafBit;
                    const bool over = boxOverlap(qmn, qmx, b[2 * e], b[2 * e + 1]);
                    if (id & kLeafBit) hit[e] = over && (key >> 24 > qc || (key >> 24 == qc && c[e] > t));
                    else push[e] = over && key >= qk;
                }
            }
            const uint32_t push0 = (__ballot_sync(0xffffffffu, push[0]) >> shift) & kWalkMask;
            const uint32_t push1 = (__ballot_sync(0xffffffffu, push[1]) >> shift) & kWalkMask;
            const uint32_t at0 = sp + __popc(push0 & below), at1 = sp + __popc(push0) + __popc(push1 & below);
            sp += __popc(push0) + __popc(push1);
            pops += k;
            if (sp > kWalkStack || pops >= n) {  // a tree visits each of its n - 1 internal nodes at most once
                if (p == 0) atomicOr(&st->err, kErrTreeDepth);
                sp = 0;
            } else {
                if (push[0]) stack[at0] = c[0];
                if (push[1]) stack[at1] = c[1];
            }
            __syncwarp();
            const uint32_t hit0 = __ballot_sync(0xffffffffu, hit[0]), hit1 = __ballot_sync(0xffffffffu, hit[1]);
            if (hit0 | hit1) {
                uint32_t slot = 0;
                if (lane == 0) slot = atomicAdd(&st->rawPairs, (uint32_t)(__popc(hit0) + __popc(hit1)));
                slot = __shfl_sync(0xffffffffu, slot, 0);
                const uint32_t before = (1u << lane) - 1u;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (!hit[e]) continue;
                    const uint32_t at = slot + (e ? __popc(hit0) + __popc(hit1 & before) : __popc(hit0 & before));
                    const uint32_t oi = (uint32_t)(keys[c[e]] & idxMask);
                    if (at >= cap) continue;
                    pkeys[at] = ((unsigned long long)min(qi, oi) << bits) | max(qi, oi);
                    if (counts) ranks[at] = aggregatedAppendKeyed(counts, min(qi, oi));
                }
            }
        }
    }
}

template <int E> static void launchFront(const BroadInput &in, const LbvhBuffers &lb, uint32_t indexBits, cudaStream_t s) {
    constexpr size_t bytes = frontBytes(kRegSortThreads * E);
    static PerDevice raised;
    allowSharedBytes(raised, k_lbvh_front<E>, bytes);
    k_lbvh_front<E><<<1, kRegSortThreads, bytes, s>>>(in, lb.keys, indexBits, lb.leafMn, lb.leafMx, lb.rec);
    PE_LAUNCHED();
}

template <uint32_t LANES>
static void launchWalk(const BroadInput &in, const LbvhBuffers &lb, uint32_t indexBits, PairBuffers &pb, bool lists,
                       DevStats *st, cudaStream_t s) {
    constexpr uint32_t leaves = kLbvhWalkThreads / LANES;
    const uint32_t b = (in.maxN + leaves - 1) / leaves, maxGrid = 32u * (uint32_t)smCount();
    k_lbvh_pairs<LANES><<<(b ? (b < maxGrid ? b : maxGrid) : 1u), kLbvhWalkThreads, 0, s>>>(
        in.d_n, lb.keys, indexBits, lb.leafMn, lb.leafMx, lb.rec, pb.keys, pb.cap, pb.bits,
        lists ? pb.count : nullptr, pb.flags, st);
    PE_LAUNCHED();
}

bool launchLbvh(const BroadInput &in, const LbvhBuffers &lb, PairBuffers &pb, DevStats *st, Scratch &ws,
                cudaStream_t s, const PairMapping &finalize) {
    uint32_t indexBits = 1;
    while (indexBits < 32 && (1ull << indexBits) < (unsigned long long)(in.maxN > 2 ? in.maxN : 2)) ++indexBits;
    const bool lists = in.maxN > kFrontMax && pairListsFit(in, finalize);
    if (in.maxN <= kRegSortThreads) {
        launchFront<1>(in, lb, indexBits, s);
    } else if (in.maxN <= 2 * kRegSortThreads) {
        launchFront<2>(in, lb, indexBits, s);
    } else if (in.maxN <= kFrontMax) {
        launchFront<4>(in, lb, indexBits, s);
    } else {
        const int g = lbvhGrid(in.maxN);
        k_lbvh_init<<<1, 32, 0, s>>>(lb.box);
        PE_LAUNCHED();
        k_lbvh_bounds<<<g, kLbvhThreads, 0, s>>>(in, lb.box);
        PE_LAUNCHED();
        k_lbvh_codes<<<g, kLbvhThreads, 0, s>>>(in, lb.box, lb.keys, indexBits, lists ? pb.count : nullptr);
        PE_LAUNCHED();
        // The index bits are already ascending (keys are laid out by index) and the
        // sort is stable, so sorting the 30 code bits orders the whole keys.
        launchRadixSort<unsigned long long>(lb.keys, lb.keysTmp, nullptr, nullptr, in.d_n, in.maxN, (int)indexBits,
                                            (int)indexBits + 30, ws, &st->err, s);
        k_lbvh_build<<<g, kLbvhThreads, 0, s>>>(in, lb.keys, indexBits, lb.childL, lb.childR, lb.parent,
                                                lb.leafParent, lb.visit, lb.leafMn, lb.leafMx);
        PE_LAUNCHED();
        k_lbvh_refit<<<g, kLbvhThreads, 0, s>>>(in.d_n, lb.childL, lb.childR, lb.parent, lb.leafParent, lb.visit,
                                                lb.leafMn, lb.leafMx, lb.rec);
        PE_LAUNCHED();
    }
    const uint32_t threads = kWalkThreadsPerSm * (uint32_t)smCount();
    if (in.maxN <= threads / 8) launchWalk<8>(in, lb, indexBits, pb, lists, st, s);
    else if (in.maxN <= threads / 4) launchWalk<4>(in, lb, indexBits, pb, lists, st, s);
    else launchWalk<2>(in, lb, indexBits, pb, lists, st, s);
    if (lists) {
        launchPairsOrder(in, pb, st, ws, s);
        return true;
    }
    return launchPairsLists(in, finalize, pb, st, s);
}

} // namespace pe
