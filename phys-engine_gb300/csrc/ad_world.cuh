// Differentiable world step: PhysicsWorld::step (src/world/physics_world.cpp:
// 518-782) for a small world of sphere/box bodies over a scalar type S, plus
// its hand-written reverse (adjoint) with the contact set of the forward pass
// frozen: the pairs, the separating axes / kept vertices, the colour order, the
// warm-start matches and every clamp branch are the ones the forward evaluation
// took; everything continuous is differentiated, including the contact points,
// normals and depths as functions of the poses.
//
// Forward (mirrors the engine stage by stage): velocity integration, AABBs,
// sweep along x with the pairs in lexicographic order, narrowphase in pair
// order, greedy colouring by manifold priority (= the engine's colouring),
// solve order (colour, index), prepare + warm-start matching, warm start,
// velocity iterations, cache rebuild, pose integration.
//
// Reverse, per step, given the adjoints of the step's outputs (poses,
// velocities, and the final impulses that the next step's warm start read):
//   pose integration -> velocity iterations (colours in reverse, points in
//   reverse, from a tape of the pre-update velocities and impulses) -> warm
//   start -> warm-start matching (to the previous step's impulses) -> contact
//   preparation -> contact geometry -> materials (friction = sqrt(fa fb),
//   restitution = max) -> velocity integration.
//
// This file holds the pieces of the step and its evaluation by one host thread
// (double precision); ad_block.cuh runs the same pieces on a thread block.
#pragma once
#include "ad_geom.cuh"

#if !defined(__CUDACC__)
#include <algorithm>
#include <cstring>
#include <vector>
#endif

namespace pe {
namespace ad {

constexpr uint32_t kAdMaxColors = 128;  // colours per window of the per-body colour masks
constexpr uint32_t kNoSlot = 0xFFFFFFFFu;
constexpr int kTapeScalars = 24; // vA, wA, vB, wB, then 4 x (n, t1, t2)
constexpr int kPmScalars = 20;   // IA (9), IB (9), imA, imB

enum : uint32_t { kAdErrPairs = 1, kAdErrManifolds = 2, kAdErrCache = 8 };

AD_HD uint32_t nextPow2u(uint32_t v) {
    uint32_t p = 1;
    while (p < v) p <<= 1;
    return p;
}

// Manifold priority for the colouring (a bijective 32-bit mix of the index).
AD_HD uint32_t adColorPriority(uint32_t m) {
    uint32_t h = m;
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

// ------------------------------------------------------------------ views ---
template <class S> struct WorldParams {
    uint32_t n;
    const uint8_t *shape;     // 0 sphere, 1 box
    const uint8_t *isStatic;
    const S *dims;            // radius / half extents, 3 per body
    const S *iinv;            // diagonal local inverse inertia, 3 per body
    const S *mass, *mu, *rest;
    S gx, gy, gz, dt;
    int iterations;
    uint32_t maxPairs, maxManifolds;  // maxManifolds is a power of two
};

template <class S> struct StateView {
    S *x, *q, *v, *w;  // 3, 4, 3, 3 per body
};

// Warm-start cache (sorted by (body A, body B), stable in solve order).
template <class S> struct CacheView {
    uint32_t *count;
    unsigned long long *key;  // body A << 32 | body B
    S *anchorA, *anchorB;     // 3 per entry
    S *lam;                   // normal, tangent 1, tangent 2
    uint32_t cap;
};

template <class S> struct StepScratch {
    S *aabb;                        // 6 per body
    uint32_t *mA, *mB, *mCount;     // manifolds in pair order
    uint32_t *mFeature;             // 4 per manifold
    S *mNormal;                     // 3
    S *mMu, *mRest;
    S *mAnchorA, *mAnchorB;         // 12 each
    S *mDepth;                      // 4
    uint32_t *color, *order;        // maxManifolds
    uint32_t *rank;                 // maxManifolds: place of a manifold in the order (thread blocks)
    unsigned long long *sortKeys;   // maxManifolds
    unsigned long long *bodyUsed;   // 2 per body
    uint32_t *colorStart;           // maxManifolds + 1 (colours <= manifolds)
    S *pp;                          // kPreparedScalars per (k, p)
    S *pm;                          // kPmScalars per k
    S *lam;                         // 3 per (k, p)
    S *lamInit;                     // 3 per (k, p)
    int32_t *match;                 // per (k, p): matched cache entry or -1
    S *tape;                        // iterations * maxManifolds * kTapeScalars
    uint32_t *cacheSlot;            // per (k, p): its entry of the output cache, or kNoSlot
    uint32_t *counts;               // [0] pairs, [1] manifolds, [2] colours, [3] error bits
    // broadphase scratch (not recorded: it may be shared by the steps of a segment)
    unsigned long long *bpEntries;  // nextPow2(n): (min.x key << 32) | body
    unsigned long long *bpPairs;    // nextPow2(maxPairs): (first << 32) | second
};

// Order-preserving 32-bit key of a float (the sort order of the sweep).
AD_HD uint32_t adOrderedKey(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
AD_HD uint32_t adOrderedKey(double d) { return adOrderedKey((float)d); }

template <class S> struct AdjointView {
    S *ax, *aq, *av, *aw;        // per body (3, 4, 3, 3)
    S *alam;                     // 3 per (k, p)
    S *app;                      // kPreparedScalars per (k, p)
    S *acache;                   // 3 per entry of the step's input cache
    // one host thread
    S *apm;                      // kPmScalars per k
    S *an;                       // 3 per k
    S *amuM;                     // per k
    // thread blocks
    S *aext;                     // kAdjointExtra per (k, p)
    S *dv, *dw;                  // 3 per body: additions to av, aw
    S *amass, *amu, *arest;      // per body, accumulated over steps
};

template <class S> AD_HD V3<S> ld3(const S *p, uint32_t i) { return {p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
template <class S> AD_HD void st3(S *p, uint32_t i, const V3<S> &v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}
template <class S> AD_HD Q<S> ld4q(const S *p, uint32_t i) { return {p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]}; }
template <class S> AD_HD void st4q(S *p, uint32_t i, const Q<S> &q) {
    p[4 * i] = q.x;
    p[4 * i + 1] = q.y;
    p[4 * i + 2] = q.z;
    p[4 * i + 3] = q.w;
}
template <class S> AD_HD M3<S> ldm(const S *p) { return {p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8]}; }

// RigidBody::getInverseMass (rigid_body.hpp:74-77)
template <class S> AD_HD S inverseMass(bool isStatic, const S &m) {
    return (isStatic || val(m) <= 0.0f) ? ADL(S, 0.0f) : ADL(S, 1.0f) / m;
}

// ------------------------------------------------------ velocity iterations --
// One contact point of solvePrepared (sequential_impulse_solver.cpp:520-603).
template <class S> struct PointIn {
    V3<S> vA, wA, vB, wB;
    S ln, l1, l2;
};
template <class S>
AD_HD void pointForward(const V3<S> &n, const S &friction, const S *c, const S &imA, const S &imB, bool sA, bool sB,
                        PointIn<S> &st) {
    const S iem = c[kPIem];
    if (val(iem) <= 0.0f) return;
    const V3<S> offA = pv(c, kPOffA), offB = pv(c, kPOffB), t1 = pv(c, kPT1), t2 = pv(c, kPT2);
    const V3<S> vA = st.vA + cross(st.wA, offA), vB = st.vB + cross(st.wB, offB);
    const V3<S> rel = vB - vA;
    const S vn = dot(rel, n);
    const S delta = -(vn + c[kPRv] - c[kPBias]) / iem;
    const S prev = st.ln;
    st.ln = smax(prev + delta, ADL(S, 0.0f));
    const S applied = st.ln - prev;
    const V3<S> impulse = n * applied;
    if (!sA) {
        st.vA += (-impulse) * imA;
        st.wA += pv(c, kPNrA) * (-applied);
    }
    if (!sB) {
        st.vB += impulse * imB;
        st.wB += pv(c, kPNrB) * applied;
    }
    if (val(c[kPItm00]) <= 0.0f || val(c[kPItm11]) <= 0.0f) return;
    const S limit = smax(friction, ADL(S, 0.0f)) * st.ln;
    const S tv1 = dot(rel, t1) + c[kPNtr1] * applied;
    const S tv2 = dot(rel, t2) + c[kPNtr2] * applied;
    const S d1 = -(c[kPItm00] * tv1 + c[kPItm01] * tv2);
    const S d2 = -(c[kPItm01] * tv1 + c[kPItm11] * tv2);
    const S p1 = st.l1, p2 = st.l2;
    st.l1 = st.l1 + d1;
    st.l2 = st.l2 + d2;
    const S lsq = st.l1 * st.l1 + st.l2 * st.l2;
    if (val(lsq) > val(limit * limit)) {
        const S s = limit / ssqrt(lsq);
        st.l1 = st.l1 * s;
        st.l2 = st.l2 * s;
    }
    const S a1 = st.l1 - p1, a2 = st.l2 - p2;
    const V3<S> ti = t1 * a1 + t2 * a2;
    const V3<S> rA = pv(c, kPTrA1) * a1 + pv(c, kPTrA2) * a2;
    const V3<S> rB = pv(c, kPTrB1) * a1 + pv(c, kPTrB2) * a2;
    if (!sA) {
        st.vA += (-ti) * imA;
        st.wA += -rA;
    }
    if (!sB) {
        st.vB += ti * imB;
        st.wB += rB;
    }
}

// Reverse of pointForward, in three parts so that a thread block can run the
// first and the last for all points of a manifold at once and only the second
// point after point.
//
// Part 1: the forward intermediates at the point's inputs.
template <class S> struct PointMid {
    V3<S> rel;
    S num, raw, ln, applied, mu0, limit, tv1, tv2, a1, a2, u1, u2, kq;
    bool live, fric, scaled;
};
template <class S>
AD_HD PointMid<S> pointMid(const V3<S> &n, const S &friction, const S *c, const PointIn<S> &in) {
    PointMid<S> m;
    const S z = S(0), iem = c[kPIem];
    m.live = !(iem <= 0.0f);
    m.fric = false;
    m.scaled = false;
    if (!m.live) return m;
    const V3<S> offA = pv(c, kPOffA), offB = pv(c, kPOffB), t1 = pv(c, kPT1), t2 = pv(c, kPT2);
    const V3<S> vAp = in.vA + cross(in.wA, offA), vBp = in.vB + cross(in.wB, offB);
    m.rel = vBp - vAp;
    const S vn = dot(m.rel, n);
    m.num = vn + c[kPRv] - c[kPBias];
    const S delta = -m.num / iem;
    const S prev = in.ln;
    m.raw = prev + delta;
    m.ln = smax(m.raw, z);
    m.applied = m.ln - prev;
    m.fric = !(c[kPItm00] <= z || c[kPItm11] <= z);
    if (m.fric) {
        m.mu0 = smax(friction, z);
        m.limit = m.mu0 * m.ln;
        m.tv1 = dot(m.rel, t1) + c[kPNtr1] * m.applied;
        m.tv2 = dot(m.rel, t2) + c[kPNtr2] * m.applied;
        const S d1 = -(c[kPItm00] * m.tv1 + c[kPItm01] * m.tv2);
        const S d2 = -(c[kPItm01] * m.tv1 + c[kPItm11] * m.tv2);
        const S r1 = in.l1 + d1, r2 = in.l2 + d2;
        const S lsq = r1 * r1 + r2 * r2;
        m.scaled = lsq > m.limit * m.limit;
        S f1 = r1, f2 = r2;
        if (m.scaled) {
            const S L = ssqrt(lsq);
            m.kq = m.limit / L;
            f1 = r1 * m.kq;
            f2 = r2 * m.kq;
            m.u1 = r1 / L;
            m.u2 = r2 / L;
        }
        m.a1 = f1 - in.l1;
        m.a2 = f2 - in.l2;
    }
    return m;
}

// Part 2: `a` holds the adjoints of the point's outputs on entry and of its
// inputs on exit; what part 3 needs is kept in the return value.
template <class S> struct PointAdj {
    V3<S> vA, wA, vB, wB;  // adjoints of the point's output velocities
    V3<S> ati, arel;
    S aa1, aa2, ar1, ar2, alimit, atv1, atv2, adelta, anum;
};
template <class S>
AD_HD PointAdj<S> pointChain(const V3<S> &n, const S *c, const S &imA, const S &imB, bool sA, bool sB,
                             const PointMid<S> &m, PointIn<S> &a) {
    PointAdj<S> r{};
    if (!m.live) return r;
    const S z = S(0), iem = c[kPIem];
    r.vA = a.vA;
    r.wA = a.wA;
    r.vB = a.vB;
    r.wB = a.wB;
    V3<S> ati{z, z, z};
    if (!sB) ati += a.vB * imB;
    if (!sA) ati += -(a.vA * imA);
    r.ati = ati;
    r.aa1 = r.aa2 = r.ar1 = r.ar2 = r.alimit = r.atv1 = r.atv2 = z;
    S aln = a.ln, aapplied = z, aprev = z;
    V3<S> arel{z, z, z};
    if (m.fric) {
        V3<S> arA{z, z, z}, arB{z, z, z};
        if (!sB) arB = a.wB;
        if (!sA) arA = -a.wA;
        r.aa1 = dot(ati, pv(c, kPT1)) + dot(arA, pv(c, kPTrA1)) + dot(arB, pv(c, kPTrB1));
        r.aa2 = dot(ati, pv(c, kPT2)) + dot(arA, pv(c, kPTrA2)) + dot(arB, pv(c, kPTrB2));
        // a = f - p; the outputs l1, l2 are f
        const S af1 = a.l1 + r.aa1, af2 = a.l2 + r.aa2;
        r.ar1 = af1;
        r.ar2 = af2;
        if (m.scaled) {
            const S ua = m.u1 * af1 + m.u2 * af2;
            r.ar1 = m.kq * (af1 - m.u1 * ua);
            r.ar2 = m.kq * (af2 - m.u2 * ua);
            r.alimit = ua;
        }
        a.l1 = -r.aa1 + r.ar1;
        a.l2 = -r.aa2 + r.ar2;
        r.atv1 = -(r.ar1 * c[kPItm00] + r.ar2 * c[kPItm01]);
        r.atv2 = -(r.ar1 * c[kPItm01] + r.ar2 * c[kPItm11]);
        arel += pv(c, kPT1) * r.atv1 + pv(c, kPT2) * r.atv2;
        aapplied = aapplied + r.atv1 * c[kPNtr1] + r.atv2 * c[kPNtr2];
        aln = aln + r.alimit * m.mu0;
    }
    // normal update
    if (!sB) aapplied = aapplied + dot(a.wB, pv(c, kPNrB));
    if (!sA) aapplied = aapplied - dot(a.wA, pv(c, kPNrA));
    aapplied = aapplied + dot(ati, n);
    aln = aln + aapplied;
    aprev = aprev - aapplied;
    const S araw = (m.raw < z) ? z : aln;
    aprev = aprev + araw;
    r.adelta = araw;
    r.anum = -araw / iem;
    arel += n * r.anum;
    r.arel = arel;
    // rel = (vB + wB x offB) - (vA + wA x offA)
    a.vB += arel;
    a.vA += -arel;
    a.wB += cross(pv(c, kPOffB), arel);
    a.wA += cross(pv(c, kPOffA), -arel);
    a.ln = aprev;
    return r;
}

// Part 3: adjoints of the prepared constants to ac[], of the normal to an, of
// the friction to amu, of the inverse masses to aimA / aimB.
template <class S>
AD_HD void pointAccumulate(const V3<S> &n, const S &friction, const S *c, const PointIn<S> &in, bool sA, bool sB,
                           const PointMid<S> &m, const PointAdj<S> &r, S *ac, V3<S> &an, S &amu, S &aimA, S &aimB) {
    if (!m.live) return;
    const S z = S(0), iem = c[kPIem];
    auto acc3 = [&](int f, const V3<S> &v) {
        ac[3 * f] = ac[3 * f] + v.x;
        ac[3 * f + 1] = ac[3 * f + 1] + v.y;
        ac[3 * f + 2] = ac[3 * f + 2] + v.z;
    };
    if (m.fric) {
        const V3<S> ti = pv(c, kPT1) * m.a1 + pv(c, kPT2) * m.a2;
        V3<S> arA{z, z, z}, arB{z, z, z};
        if (!sB) {
            aimB = aimB + dot(r.vB, ti);
            arB = r.wB;
        }
        if (!sA) {
            aimA = aimA - dot(r.vA, ti);
            arA = -r.wA;
        }
        acc3(kPT1, r.ati * m.a1);
        acc3(kPT2, r.ati * m.a2);
        acc3(kPTrA1, arA * m.a1);
        acc3(kPTrA2, arA * m.a2);
        acc3(kPTrB1, arB * m.a1);
        acc3(kPTrB2, arB * m.a2);
        ac[kPItm00] = ac[kPItm00] - r.ar1 * m.tv1;
        ac[kPItm01] = ac[kPItm01] - (r.ar1 * m.tv2 + r.ar2 * m.tv1);
        ac[kPItm11] = ac[kPItm11] - r.ar2 * m.tv2;
        acc3(kPT1, m.rel * r.atv1);
        acc3(kPT2, m.rel * r.atv2);
        ac[kPNtr1] = ac[kPNtr1] + r.atv1 * m.applied;
        ac[kPNtr2] = ac[kPNtr2] + r.atv2 * m.applied;
        if (!(friction < z)) amu = amu + r.alimit * m.ln;
    }
    const V3<S> impulse = n * m.applied;
    if (!sB) {
        aimB = aimB + dot(r.vB, impulse);
        acc3(kPNrB, r.wB * m.applied);
    }
    if (!sA) {
        aimA = aimA - dot(r.vA, impulse);
        acc3(kPNrA, r.wA * (-m.applied));
    }
    an += r.ati * m.applied;
    ac[kPIem] = ac[kPIem] + r.adelta * m.num / (iem * iem);
    ac[kPRv] = ac[kPRv] + r.anum;
    ac[kPBias] = ac[kPBias] - r.anum;
    an += m.rel * r.anum;
    acc3(kPOffB, cross(r.arel, in.wB));
    acc3(kPOffA, cross(-r.arel, in.wA));
}

// Velocities after the forward pass's integration (integrateVelocity without an
// applied force).
template <class S> AD_HD V3<S> integratedVelocity(const WorldParams<S> &W, uint32_t i, V3<S> v) {
    if (!W.isStatic[i]) {
        const S z = ADL(S, 0.0f);
        const V3<S> g{W.gx, W.gy, W.gz}, f{z, z, z};
        const V3<S> acc = g + f * inverseMass(false, W.mass[i]);
        v += acc * W.dt;
    }
    return v;
}

template <class S> AD_HD void bodyAabb(const WorldParams<S> &W, uint32_t i, const V3<S> &p, const Q<S> &q, V3<S> &mn,
                                       V3<S> &mx) {
    if (W.shape[i] == 0) {
        const S r = W.dims[3 * i];
        const V3<S> rr{r, r, r};
        mn = p - rr;
        mx = p + rr;
    } else {
        const M3<S> m = toMat3(q);
        const S hx = W.dims[3 * i], hy = W.dims[3 * i + 1], hz = W.dims[3 * i + 2];
        const V3<S> e{sabs(m.m00) * hx + sabs(m.m01) * hy + sabs(m.m02) * hz,
                      sabs(m.m10) * hx + sabs(m.m11) * hy + sabs(m.m12) * hz,
                      sabs(m.m20) * hx + sabs(m.m21) * hy + sabs(m.m22) * hz};
        mn = p - e;
        mx = p + e;
    }
}

// Pose integration (rigid_body.cpp:103-125) of one body and its reverse.
template <class S> AD_HD void poseForward(const S &dt, const V3<S> &lin, const V3<S> &ang, V3<S> &pos, Q<S> &rot) {
    pos += lin * dt;
    const Q<S> spin{ang.x, ang.y, ang.z, ADL(S, 0.0f)};
    const Q<S> d = qmul(spin, rot);
    const S h = ADL(S, 0.5f) * dt;
    rot.x = rot.x + h * d.x;
    rot.y = rot.y + h * d.y;
    rot.z = rot.z + h * d.z;
    rot.w = rot.w + h * d.w;
    rot = qnormalized(rot);
}
// rot, ang: the inputs; aq: adjoint of the new rotation in, of the old one out;
// av, aw: adjoints of the velocities, added to.
template <class S>
AD_HD void poseReverse(const S &dt, const Q<S> &rot, const V3<S> &ang, const V3<S> &ax, Q<S> &aq, V3<S> &av, V3<S> &aw) {
    const S z = S(0);
    av += ax * dt;
    const Q<S> spin{ang.x, ang.y, ang.z, z};
    const Q<S> d = qmul(spin, rot);
    const S h = S(0.5f) * dt;
    const Q<S> u{rot.x + h * d.x, rot.y + h * d.y, rot.z + h * d.z, rot.w + h * d.w};
    const S len = ssqrt(u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w);
    Q<S> au{z, z, z, z};
    if (len != z) {
        const Q<S> q1{u.x / len, u.y / len, u.z / len, u.w / len};
        const S qa = q1.x * aq.x + q1.y * aq.y + q1.z * aq.z + q1.w * aq.w;
        au = Q<S>{(aq.x - q1.x * qa) / len, (aq.y - q1.y * qa) / len, (aq.z - q1.z * qa) / len,
                  (aq.w - q1.w * qa) / len};
    }
    Q<S> arot = au, aspin{z, z, z, z};
    const Q<S> ad{h * au.x, h * au.y, h * au.z, h * au.w};
    qmulAdj(spin, rot, ad, aspin, arot);
    aw += V3<S>{aspin.x, aspin.y, aspin.z};
    aq = arot;
}

// Impulses of a matched cache entry (normal, tangents) clamped to the friction
// cone (sequential_impulse_solver.cpp:448-490), and the reverse: adjoints of
// the clamped impulses in, of the entry's out; the friction's is added to.
template <class S> AD_HD void warmClamp(const S &friction, const S &cn, const S &c1, const S &c2, S &l0, S &l1, S &l2) {
    const S z = ADL(S, 0.0f);
    const S ni = smax(cn, z);
    const S limit = smax(friction, z) * ni;
    const S tlsq = c1 * c1 + c2 * c2;
    const S scale = val(tlsq) > val(limit * limit) ? limit / ssqrt(tlsq) : ADL(S, 1.0f);
    l0 = ni;
    l1 = c1 * scale;
    l2 = c2 * scale;
}
template <class S>
AD_HD V3<S> warmClampReverse(const S &mu, const S &cn, const S &c1, const S &c2, const V3<S> &alam, S &amu) {
    const S z = S(0);
    const S ni = smax(cn, z);
    const S mu0 = smax(mu, z);
    const S limit = mu0 * ni;
    const S tlsq = c1 * c1 + c2 * c2;
    S ani = alam.x;
    const S af1 = alam.y, af2 = alam.z;
    S ac1 = af1, ac2 = af2;
    if (tlsq > limit * limit) {
        const S L = ssqrt(tlsq);
        const S u1 = c1 / L, u2 = c2 / L;
        const S ua = u1 * af1 + u2 * af2;
        ac1 = (limit / L) * (af1 - u1 * ua);
        ac2 = (limit / L) * (af2 - u2 * ua);
        ani = ani + ua * mu0;
        if (!(mu < z)) amu = amu + ua * ni;
    }
    return {(cn < z) ? z : ani, ac1, ac2};
}

// The warm start's application of one matched point in reverse (the body
// adjoints pass through): adjoints of the initial impulses, of the prepared
// constants, of the normal and of the inverse masses and inertias are added to.
template <class S>
AD_HD void warmReverse(const V3<S> &n, const S *pp, const V3<S> &lam, const M3<S> &IA, const M3<S> &IB, const S &imA,
                       const S &imB, bool sA, bool sB, const V3<S> &avA, const V3<S> &awA, const V3<S> &avB,
                       const V3<S> &awB, V3<S> &alam, S *ac, V3<S> &an, M3<S> &aIA, M3<S> &aIB, S &aimA, S &aimB) {
    const S z = S(0);
    const V3<S> t1 = pv(pp, kPT1), t2 = pv(pp, kPT2), offA = pv(pp, kPOffA), offB = pv(pp, kPOffB);
    const V3<S> wi = n * lam.x + t1 * lam.y + t2 * lam.z;
    const V3<S> nw = -wi;
    V3<S> awi{z, z, z};
    auto acc3 = [&](int f, const V3<S> &v) {
        ac[3 * f] = ac[3 * f] + v.x;
        ac[3 * f + 1] = ac[3 * f + 1] + v.y;
        ac[3 * f + 2] = ac[3 * f + 2] + v.z;
    };
    if (!sB) {
        awi += avB * imB;
        aimB = aimB + dot(avB, wi);
        V3<S> ay{z, z, z}, aoff{z, z, z};
        mulAdj(IB, cross(offB, wi), awB, aIB, ay);
        crossAdj(offB, wi, ay, aoff, awi);
        acc3(kPOffB, aoff);
    }
    if (!sA) {
        V3<S> anw = avA * imA;
        aimA = aimA + dot(avA, nw);
        V3<S> ay{z, z, z}, aoff{z, z, z};
        mulAdj(IA, cross(offA, nw), awA, aIA, ay);
        crossAdj(offA, nw, ay, aoff, anw);
        acc3(kPOffA, aoff);
        awi += -anw;
    }
    alam.x = alam.x + dot(awi, n);
    alam.y = alam.y + dot(awi, t1);
    alam.z = alam.z + dot(awi, t2);
    an += awi * lam.x;
    acc3(kPT1, awi * lam.y);
    acc3(kPT2, awi * lam.z);
}

// --------------------------------------- one host thread: forward, reverse --
#if !defined(__CUDACC__)
template <class S>
inline void forwardStep(const WorldParams<S> &W, const StateView<S> &in, const CacheView<S> &cin, StateView<S> out,
                       CacheView<S> cout, StepScratch<S> sc, bool record) {
    const uint32_t n = W.n;
    const S z = ADL(S, 0.0f);
    // 1. velocity integration (RigidBody::integrateVelocity, no applied force) and AABBs
    for (uint32_t i = 0; i < n; ++i) {
        st3(out.v, i, integratedVelocity(W, i, ld3(in.v, i)));
        st3(out.w, i, ld3(in.w, i));
        V3<S> mn, mx;
        bodyAabb(W, i, ld3(in.x, i), ld4q(in.q, i), mn, mx);
        st3(sc.aabb, 2 * i, mn);
        st3(sc.aabb, 2 * i + 1, mx);
    }
    sc.counts[0] = sc.counts[1] = sc.counts[3] = 0;
    // 2. every pair (i < j) with overlapping AABBs (touching counts), in
    // lexicographic order: sort and sweep along x (broadphase.cpp:195-291) —
    // bodies sorted by min.x, each tested against the later ones whose min.x
    // does not exceed its max.x (the one of an overlapping pair sorted first
    // always meets the other) — then the pairs sorted by (first, second).
    for (uint32_t i = 0; i < n; ++i)
        sc.bpEntries[i] = ((unsigned long long)adOrderedKey(val(sc.aabb[6 * i])) << 32) | i;
    std::sort(sc.bpEntries, sc.bpEntries + n);
    auto overlapsYZ = [&](uint32_t a, uint32_t b) {
        const V3<S> amn = ld3(sc.aabb, 2 * a), amx = ld3(sc.aabb, 2 * a + 1);
        const V3<S> bmn = ld3(sc.aabb, 2 * b), bmx = ld3(sc.aabb, 2 * b + 1);
        return val(amn.y) <= val(bmx.y) && val(amx.y) >= val(bmn.y) && val(amn.z) <= val(bmx.z) &&
               val(amx.z) >= val(bmn.z);
    };
    uint32_t P = 0;
    for (uint32_t k = 0; k < n; ++k) {
        const uint32_t i = (uint32_t)sc.bpEntries[k];
        const auto maxX = val(sc.aabb[6 * i + 3]);
        for (uint32_t kk = k + 1; kk < n; ++kk) {
            const uint32_t j = (uint32_t)sc.bpEntries[kk];
            if (val(sc.aabb[6 * j]) > maxX) break;
            if (!overlapsYZ(i, j)) continue;
            if (P < W.maxPairs) sc.bpPairs[P] = ((unsigned long long)(i < j ? i : j) << 32) | (i < j ? j : i);
            ++P;
        }
    }
    if (P > W.maxPairs) {
        sc.counts[3] |= kAdErrPairs;
        P = W.maxPairs;
    }
    std::sort(sc.bpPairs, sc.bpPairs + P);
    sc.counts[0] = P;
    // 3. narrowphase in pair order, manifolds compacted in that order
    uint32_t M = 0;
    for (uint32_t p = 0; p < P; ++p) {
        const uint32_t a = (uint32_t)(sc.bpPairs[p] >> 32), b = (uint32_t)sc.bpPairs[p];
        Contact<S> c{};
        const Tf<S> tA{ld3(in.x, a), ld4q(in.q, a)}, tB{ld3(in.x, b), ld4q(in.q, b)};
        if (!contactPair<S>(W.shape[a], ld3(W.dims, a), tA, W.shape[b], ld3(W.dims, b), tB, c)) continue;
        const uint32_t m = M++;
        if (m >= W.maxManifolds) continue;
        sc.mA[m] = a;
        sc.mB[m] = b;
        sc.mCount[m] = c.count;
        st3(sc.mNormal, m, c.normal);
        sc.mRest[m] = smax(W.rest[a], W.rest[b]);
        sc.mMu[m] = ssqrt(smax(W.mu[a], z) * smax(W.mu[b], z));
        for (uint32_t k = 0; k < 4; ++k) {
            const bool live = k < c.count;
            st3(sc.mAnchorA, 4 * m + k, live ? c.anchorA[k] : V3<S>{z, z, z});
            st3(sc.mAnchorB, 4 * m + k, live ? c.anchorB[k] : V3<S>{z, z, z});
            sc.mDepth[4 * m + k] = live ? c.depth[k] : z;
            sc.mFeature[4 * m + k] = live ? c.feature[k] | (c.axis << kAdAxisShift) : 0u;
        }
    }
    if (M > W.maxManifolds) {
        sc.counts[3] |= kAdErrManifolds;
        M = W.maxManifolds;
    }
    sc.counts[1] = M;
    // 4. colouring: greedy in decreasing priority over manifolds that share a
    // dynamic body (the engine's colouring), then order = (colour, index)
    for (uint32_t i = 0; i < M; ++i) sc.sortKeys[i] = ((unsigned long long)(~adColorPriority(i)) << 32) | i;
    for (uint32_t i = 0; i < 2 * n; ++i) sc.bodyUsed[i] = 0ull;
    std::sort(sc.sortKeys, sc.sortKeys + M);
    {
        // Colour windows of kAdMaxColors: a manifold whose higher-priority
        // neighbours use the whole window waits for the next window, in which
        // only the waiting manifolds take colours (the engine's rule, so the
        // same colouring); no colour limit.
        constexpr uint32_t kWaiting = 0xFFFFFFFFu;
        for (uint32_t r = 0; r < M; ++r) sc.color[(uint32_t)sc.sortKeys[r]] = kWaiting;
        uint32_t colors = 0, base = 0, waiting = M;
        while (waiting) {
            uint32_t deferred = 0;
            for (uint32_t r = 0; r < M; ++r) {
                const uint32_t m = (uint32_t)sc.sortKeys[r];
                if (sc.color[m] != kWaiting) continue;
                const uint32_t a = sc.mA[m], b = sc.mB[m];
                const bool da = !W.isStatic[a], db = !W.isStatic[b];
                unsigned long long u0 = 0, u1 = 0;
                if (da) {
                    u0 |= sc.bodyUsed[2 * a];
                    u1 |= sc.bodyUsed[2 * a + 1];
                }
                if (db) {
                    u0 |= sc.bodyUsed[2 * b];
                    u1 |= sc.bodyUsed[2 * b + 1];
                }
                uint32_t local = kAdMaxColors;
                for (uint32_t k = 0; k < kAdMaxColors && local == kAdMaxColors; ++k) {
                    const unsigned long long w = k < 64 ? u0 : u1;
                    if (!((w >> (k & 63)) & 1ull)) local = k;
                }
                if (local == kAdMaxColors) {
                    ++deferred;
                    continue;
                }
                const uint32_t c = base + local;
                sc.color[m] = c;
                const unsigned long long bit = 1ull << (local & 63);
                if (da) sc.bodyUsed[2 * a + (local >> 6)] |= bit;
                if (db) sc.bodyUsed[2 * b + (local >> 6)] |= bit;
                if (c + 1 > colors) colors = c + 1;
            }
            waiting = deferred;
            if (waiting) {
                base += kAdMaxColors;
                for (uint32_t i = 0; i < 2 * n; ++i) sc.bodyUsed[i] = 0ull;
            }
        }
        sc.counts[2] = colors;
    }
    for (uint32_t i = 0; i < M; ++i) sc.sortKeys[i] = ((unsigned long long)sc.color[i] << 32) | i;
    std::sort(sc.sortKeys, sc.sortKeys + M);
    const uint32_t C = sc.counts[2];
    for (uint32_t k = 0; k < M; ++k) {
        sc.order[k] = (uint32_t)sc.sortKeys[k];
        const uint32_t ck = (uint32_t)(sc.sortKeys[k] >> 32);
        const uint32_t cp = k == 0 ? 0xFFFFFFFFu : (uint32_t)(sc.sortKeys[k - 1] >> 32);
        for (uint32_t c = (k == 0 ? 0 : cp + 1); c <= ck; ++c) sc.colorStart[c] = k;
    }
    sc.colorStart[C] = M;
    // 5. prepare + warm-start matching (sequential_impulse_solver.cpp:101-214, :448-490)
    const S inverseDt = ADL(S, 1.0f) / smax(W.dt, ADL(S, 1e-6f));
    const uint32_t cacheN = *cin.count;
    for (uint32_t k = 0; k < M; ++k) {
        const uint32_t m = sc.order[k];
        const uint32_t a = sc.mA[m], b = sc.mB[m];
        const bool sA = W.isStatic[a] != 0, sB = W.isStatic[b] != 0;
        const Q<S> qA = ld4q(in.q, a), qB = ld4q(in.q, b);
        const M3<S> IA = inverseInertiaWorld(qA, W.iinv[3 * a], W.iinv[3 * a + 1], W.iinv[3 * a + 2]);
        const M3<S> IB = inverseInertiaWorld(qB, W.iinv[3 * b], W.iinv[3 * b + 1], W.iinv[3 * b + 2]);
        const S imA = inverseMass(sA, W.mass[a]), imB = inverseMass(sB, W.mass[b]);
        S *pm = sc.pm + (size_t)k * kPmScalars;
        const S *ia = &IA.m00, *ib = &IB.m00;
        for (int e = 0; e < 9; ++e) {
            pm[e] = ia[e];
            pm[9 + e] = ib[e];
        }
        pm[18] = imA;
        pm[19] = imB;
        const V3<S> n3 = ld3(sc.mNormal, m);
        const V3<S> linA = ld3(out.v, a), angA = ld3(out.w, a), linB = ld3(out.v, b), angB = ld3(out.w, b);
        const unsigned long long key = ((unsigned long long)a << 32) | b;
        uint32_t lo = 0, hi = cacheN;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (cin.key[mid] < key) lo = mid + 1;
            else hi = mid;
        }
        uint32_t re = lo;
        while (re < cacheN && cin.key[re] == key) ++re;
        const S friction = sc.mMu[m];
        const uint32_t npts = sc.mCount[m];
        for (uint32_t p = 0; p < 4; ++p) {
            const size_t kp = (size_t)k * 4 + p;
            S *pp = sc.pp + kp * kPreparedScalars;
            for (int e = 0; e < kPreparedScalars; ++e) pp[e] = z;
            S l0 = z, l1 = z, l2 = z;
            int32_t match = -1;
            if (p < npts) {
                const V3<S> anA = ld3(sc.mAnchorA, 4 * m + p), anB = ld3(sc.mAnchorB, 4 * m + p);
                Prepared<S> pr;
                preparePoint(n3, anA, anB, sc.mDepth[4 * m + p], qA, qB, IA, IB, imA, imB, linA, angA, linB, angB,
                             sc.mRest[m], inverseDt, pr);
                preparedPack(pr, pp);
                if (pr.tangentValid && !(val(pr.iem) <= 0.0f)) {
                    const float matchSq = 0.05f * 0.05f;
                    for (uint32_t e = lo; e < re; ++e) {
                        const V3<S> da = ld3(cin.anchorA, e) - anA, db = ld3(cin.anchorB, e) - anB;
                        if (val(dot(da, da)) > matchSq || val(dot(db, db)) > matchSq) continue;
                        const S cn = cin.lam[3 * e], c1 = cin.lam[3 * e + 1], c2 = cin.lam[3 * e + 2];
                        warmClamp(friction, cn, c1, c2, l0, l1, l2);
                        match = (int32_t)e;
                        break;
                    }
                }
            }
            sc.match[kp] = match;
            sc.lamInit[3 * kp] = sc.lam[3 * kp] = l0;
            sc.lamInit[3 * kp + 1] = sc.lam[3 * kp + 1] = l1;
            sc.lamInit[3 * kp + 2] = sc.lam[3 * kp + 2] = l2;
        }
    }
    // 6. warm start, colour by colour (warmStartPrepared :453-490)
    for (uint32_t c = 0; c < C; ++c) {
        for (uint32_t k = sc.colorStart[c]; k < sc.colorStart[c + 1]; ++k) {
            const uint32_t m = sc.order[k];
            const uint32_t a = sc.mA[m], b = sc.mB[m];
            const bool sA = W.isStatic[a] != 0, sB = W.isStatic[b] != 0;
            const S *pm = sc.pm + (size_t)k * kPmScalars;
            const M3<S> IA = ldm(pm), IB = ldm(pm + 9);
            const V3<S> n3 = ld3(sc.mNormal, m);
            V3<S> linA = ld3(out.v, a), angA = ld3(out.w, a), linB = ld3(out.v, b), angB = ld3(out.w, b);
            bool any = false;
            for (uint32_t p = 0; p < sc.mCount[m]; ++p) {
                const size_t kp = (size_t)k * 4 + p;
                if (sc.match[kp] < 0) continue;
                const S *pp = sc.pp + kp * kPreparedScalars;
                const V3<S> wi = n3 * sc.lamInit[3 * kp] + pv(pp, kPT1) * sc.lamInit[3 * kp + 1] +
                                 pv(pp, kPT2) * sc.lamInit[3 * kp + 2];
                const V3<S> nw = -wi;
                if (!sA) {
                    linA += nw * pm[18];
                    angA += mul(IA, cross(pv(pp, kPOffA), nw));
                }
                if (!sB) {
                    linB += wi * pm[19];
                    angB += mul(IB, cross(pv(pp, kPOffB), wi));
                }
                any = true;
            }
            if (!any) continue;
            if (!sA) {
                st3(out.v, a, linA);
                st3(out.w, a, angA);
            }
            if (!sB) {
                st3(out.v, b, linB);
                st3(out.w, b, angB);
            }
        }
    }
    // 7. velocity iterations in colour order, with the tape of each manifold update
    for (int it = 0; it < W.iterations; ++it)
        for (uint32_t c = 0; c < C; ++c) {
            for (uint32_t k = sc.colorStart[c]; k < sc.colorStart[c + 1]; ++k) {
                const uint32_t m = sc.order[k];
                const uint32_t a = sc.mA[m], b = sc.mB[m];
                const bool sA = W.isStatic[a] != 0, sB = W.isStatic[b] != 0;
                const S *pm = sc.pm + (size_t)k * kPmScalars;
                const V3<S> n3 = ld3(sc.mNormal, m);
                PointIn<S> s{ld3(out.v, a), ld3(out.w, a), ld3(out.v, b), ld3(out.w, b), z, z, z};
                if (record) {
                    S *tp = sc.tape + ((size_t)it * W.maxManifolds + k) * kTapeScalars;
                    st3(tp, 0, s.vA);
                    st3(tp, 1, s.wA);
                    st3(tp, 2, s.vB);
                    st3(tp, 3, s.wB);
                    for (int e = 0; e < 12; ++e) tp[12 + e] = sc.lam[(size_t)k * 12 + e];
                }
                for (uint32_t p = 0; p < sc.mCount[m]; ++p) {
                    const size_t kp = (size_t)k * 4 + p;
                    s.ln = sc.lam[3 * kp];
                    s.l1 = sc.lam[3 * kp + 1];
                    s.l2 = sc.lam[3 * kp + 2];
                    pointForward(n3, sc.mMu[m], sc.pp + kp * kPreparedScalars, pm[18], pm[19], sA, sB, s);
                    sc.lam[3 * kp] = s.ln;
                    sc.lam[3 * kp + 1] = s.l1;
                    sc.lam[3 * kp + 2] = s.l2;
                }
                if (!sA) {
                    st3(out.v, a, s.vA);
                    st3(out.w, a, s.wA);
                }
                if (!sB) {
                    st3(out.v, b, s.vB);
                    st3(out.w, b, s.wB);
                }
            }
        }
    // 8. cache rebuild: entries sorted by (body A, body B), stable in solve order (:623-681)
    for (uint32_t i = 0; i < M; ++i) {
        const uint32_t m = sc.order[i];
        sc.sortKeys[i] = ((unsigned long long)sc.mA[m] << 44) | ((unsigned long long)sc.mB[m] << 24) | i;
    }
    std::sort(sc.sortKeys, sc.sortKeys + M);
    {
        uint32_t e = 0;
        for (uint32_t kp = 0; kp < 4 * M; ++kp) sc.cacheSlot[kp] = kNoSlot;
        for (uint32_t r = 0; r < M; ++r) {
            const uint32_t k = (uint32_t)(sc.sortKeys[r] & 0xFFFFFFu);
            const uint32_t m = sc.order[k];
            for (uint32_t p = 0; p < sc.mCount[m]; ++p, ++e) {
                if (e >= cout.cap) {
                    sc.counts[3] |= kAdErrCache;
                    break;
                }
                const size_t kp = (size_t)k * 4 + p;
                cout.key[e] = ((unsigned long long)sc.mA[m] << 32) | sc.mB[m];
                st3(cout.anchorA, e, ld3(sc.mAnchorA, 4 * m + p));
                st3(cout.anchorB, e, ld3(sc.mAnchorB, 4 * m + p));
                cout.lam[3 * e] = sc.lam[3 * kp];
                cout.lam[3 * e + 1] = sc.lam[3 * kp + 1];
                cout.lam[3 * e + 2] = sc.lam[3 * kp + 2];
                sc.cacheSlot[kp] = e;
            }
        }
        *cout.count = e < cout.cap ? e : cout.cap;
    }
    // 9. pose integration (rigid_body.cpp:103-125)
    for (uint32_t i = 0; i < n; ++i) {
        V3<S> pos = ld3(in.x, i);
        Q<S> rot = ld4q(in.q, i);
        if (!W.isStatic[i]) poseForward(W.dt, ld3(out.v, i), ld3(out.w, i), pos, rot);
        st3(out.x, i, pos);
        st4q(out.q, i, rot);
    }
}

// ------------------------------------------------------------------ reverse --
template <class S>
inline void backwardStep(const WorldParams<S> &W, const StateView<S> &in, const CacheView<S> &cin,
                         const StateView<S> &out, const StepScratch<S> &sc, AdjointView<S> adj) {
    const uint32_t n = W.n;
    const S z = S(0);
    const uint32_t M = sc.counts[1], C = sc.counts[2];
    // clear the per-step adjoints of constants
    for (uint32_t i = 0; i < M * 4 * kPreparedScalars; ++i) adj.app[i] = z;
    for (uint32_t i = 0; i < M * kPmScalars; ++i) adj.apm[i] = z;
    for (uint32_t i = 0; i < 3 * M; ++i) adj.an[i] = z;
    for (uint32_t i = 0; i < M; ++i) adj.amuM[i] = z;
    for (uint32_t i = 0; i < 3 * (*cin.count); ++i) adj.acache[i] = z;
    // 1. pose integration
    for (uint32_t i = 0; i < n; ++i) {
        if (W.isStatic[i]) continue;
        Q<S> aq = ld4q(adj.aq, i);
        V3<S> av = ld3(adj.av, i), aw = ld3(adj.aw, i);
        poseReverse(W.dt, ld4q(in.q, i), ld3(out.w, i), ld3(adj.ax, i), aq, av, aw);
        st3(adj.av, i, av);
        st3(adj.aw, i, aw);
        st4q(adj.aq, i, aq);
    }
    // 2. velocity iterations in reverse
    for (int it = W.iterations - 1; it >= 0; --it)
        for (int ci = (int)C - 1; ci >= 0; --ci) {
            const uint32_t c = (uint32_t)ci;
            for (uint32_t k = sc.colorStart[c]; k < sc.colorStart[c + 1]; ++k) {
                const uint32_t m = sc.order[k];
                const uint32_t a = sc.mA[m], b = sc.mB[m];
                const bool sA = W.isStatic[a] != 0, sB = W.isStatic[b] != 0;
                const S *pm = sc.pm + (size_t)k * kPmScalars;
                const V3<S> n3 = ld3(sc.mNormal, m);
                const S mu = sc.mMu[m];
                const S *tp = sc.tape + ((size_t)it * W.maxManifolds + k) * kTapeScalars;
                const uint32_t npts = sc.mCount[m];
                PointIn<S> ins[4];
                PointIn<S> s{ld3(tp, 0), ld3(tp, 1), ld3(tp, 2), ld3(tp, 3), z, z, z};
                for (uint32_t p = 0; p < npts; ++p) {
                    s.ln = tp[12 + 3 * p];
                    s.l1 = tp[12 + 3 * p + 1];
                    s.l2 = tp[12 + 3 * p + 2];
                    ins[p] = s;
                    pointForward(n3, mu, sc.pp + ((size_t)k * 4 + p) * kPreparedScalars, pm[18], pm[19], sA, sB, s);
                }
                PointIn<S> ab{sA ? V3<S>{z, z, z} : ld3(adj.av, a), sA ? V3<S>{z, z, z} : ld3(adj.aw, a),
                              sB ? V3<S>{z, z, z} : ld3(adj.av, b), sB ? V3<S>{z, z, z} : ld3(adj.aw, b), z, z, z};
                V3<S> an = ld3(adj.an, k);
                S amu = adj.amuM[k];
                S *apm = adj.apm + (size_t)k * kPmScalars;
                S aimA = apm[18], aimB = apm[19];
                for (int p = (int)npts - 1; p >= 0; --p) {
                    const size_t kp = (size_t)k * 4 + p;
                    const S *c = sc.pp + kp * kPreparedScalars;
                    ab.ln = adj.alam[3 * kp];
                    ab.l1 = adj.alam[3 * kp + 1];
                    ab.l2 = adj.alam[3 * kp + 2];
                    const PointMid<S> mid = pointMid(n3, mu, c, ins[p]);
                    const PointAdj<S> r = pointChain(n3, c, pm[18], pm[19], sA, sB, mid, ab);
                    pointAccumulate(n3, mu, c, ins[p], sA, sB, mid, r, adj.app + kp * kPreparedScalars, an, amu, aimA,
                                    aimB);
                    adj.alam[3 * kp] = ab.ln;
                    adj.alam[3 * kp + 1] = ab.l1;
                    adj.alam[3 * kp + 2] = ab.l2;
                }
                apm[18] = aimA;
                apm[19] = aimB;
                st3(adj.an, k, an);
                adj.amuM[k] = amu;
                if (!sA) {
                    st3(adj.av, a, ab.vA);
                    st3(adj.aw, a, ab.wA);
                }
                if (!sB) {
                    st3(adj.av, b, ab.vB);
                    st3(adj.aw, b, ab.wB);
                }
            }
        }
    // 3. warm start and its matching, 4. preparation, 5. contact geometry, 6. materials.
    // The preparation's velocity adjoints wait until every warm start has read
    // the body adjoints.
    std::vector<V3<S>> dv(n, V3<S>{z, z, z}), dw(n, V3<S>{z, z, z});
    const S inverseDt = S(1) / smax(W.dt, ADL(S, 1e-6f));
    for (uint32_t k = 0; k < M; ++k) {
        const uint32_t m = sc.order[k];
        const uint32_t a = sc.mA[m], b = sc.mB[m];
        const bool sA = W.isStatic[a] != 0, sB = W.isStatic[b] != 0;
        const S *pm = sc.pm + (size_t)k * kPmScalars;
        const S *apm = adj.apm + (size_t)k * kPmScalars;
        const M3<S> IA = ldm(pm), IB = ldm(pm + 9);
        const V3<S> n3 = ld3(sc.mNormal, m);
        const V3<S> avA = ld3(adj.av, a), awA = ld3(adj.aw, a), avB = ld3(adj.av, b), awB = ld3(adj.aw, b);
        const S mu = sc.mMu[m], rest = sc.mRest[m];
        const Tf<S> tA{ld3(in.x, a), ld4q(in.q, a)}, tB{ld3(in.x, b), ld4q(in.q, b)};
        const V3<S> linA = integratedVelocity(W, a, ld3(in.v, a)), angA = ld3(in.w, a);
        const V3<S> linB = integratedVelocity(W, b, ld3(in.v, b)), angB = ld3(in.w, b);
        S amu = adj.amuM[k];
        PrepareGrad<S> g{};
        g.n = ld3(adj.an, k);
        g.imA = apm[18];
        g.imB = apm[19];
        Tf<S> gA{{z, z, z}, {z, z, z, z}}, gB = gA;
        V3<S> gn{z, z, z};
        for (uint32_t p = 0; p < sc.mCount[m]; ++p) {
            const size_t kp = (size_t)k * 4 + p;
            const S *pp = sc.pp + kp * kPreparedScalars;
            S *ac = adj.app + kp * kPreparedScalars;
            const int32_t e = sc.match[kp];
            if (e >= 0) {
                V3<S> alam = ld3(adj.alam, (uint32_t)kp);
                warmReverse(n3, pp, ld3(sc.lamInit, (uint32_t)kp), IA, IB, pm[18], pm[19], sA, sB, avA, awA, avB, awB,
                            alam, ac, g.n, g.IA, g.IB, g.imA, g.imB);
                const V3<S> o = warmClampReverse(mu, cin.lam[3 * e], cin.lam[3 * e + 1], cin.lam[3 * e + 2], alam, amu);
                st3(adj.acache, (uint32_t)e, ld3(adj.acache, (uint32_t)e) + o);
            }
            g.anchorA = g.anchorB = V3<S>{z, z, z};
            g.depth = z;
            const V3<S> anchorA = ld3(sc.mAnchorA, 4 * m + p), anchorB = ld3(sc.mAnchorB, 4 * m + p);
            preparePointReverse(n3, anchorA, anchorB, sc.mDepth[4 * m + p], tA.q, tB.q, IA, IB, pm[18] + pm[19], linA,
                                angA, linB, angB, rest, inverseDt, pp, ac, g);
            // a one-point manifold's normal goes with its point; the points of
            // two boxes only add to it
            const bool last = p + 1 == sc.mCount[m];
            if (last) gn += g.n;
            contactPointReverse(W.shape[a], ld3(W.dims, a), tA, W.shape[b], ld3(W.dims, b), tB, n3,
                                sc.mFeature[4 * m + p], PointGrad<S>{g.anchorA, g.anchorB, g.depth}, gn, gA, gB);
        }
        if (W.shape[a] == 1 && W.shape[b] == 1)
            boxNormalReverse(tA, tB, (sc.mFeature[4 * m] & kAdAxisMask) >> kAdAxisShift, n3, gn, gA, gB);
        inverseInertiaAdj(tA.q, ld3(W.iinv, a), g.IA, g.qA);
        inverseInertiaAdj(tB.q, ld3(W.iinv, b), g.IB, g.qB);
        auto body = [&](uint32_t i, const Tf<S> &t, const Q<S> &gq, const V3<S> &lin, const V3<S> &ang, const S &im,
                        const S &aim) {
            st3(adj.ax, i, ld3(adj.ax, i) + t.p);
            const Q<S> q = ld4q(adj.aq, i);
            st4q(adj.aq, i, Q<S>{q.x + (t.q.x + gq.x), q.y + (t.q.y + gq.y), q.z + (t.q.z + gq.z), q.w + (t.q.w + gq.w)});
            dv[i] += lin;
            dw[i] += ang;
            adj.amass[i] = adj.amass[i] - aim * im * im;  // im = 1 / mass
        };
        if (!sA) body(a, gA, g.qA, g.linA, g.angA, pm[18], g.imA);
        if (!sB) body(b, gB, g.qB, g.linB, g.angB, pm[19], g.imB);
        if (W.rest[a] < W.rest[b]) {
            if (!sB) adj.arest[b] = adj.arest[b] + g.rest;
        } else if (!sA) {
            adj.arest[a] = adj.arest[a] + g.rest;
        }
        if (mu > z) {
            const S fa = smax(W.mu[a], z), fb = smax(W.mu[b], z);
            const S h = amu * (S(0.5f) / mu);
            if (!sA && !(W.mu[a] < z)) adj.amu[a] = adj.amu[a] + h * fb;
            if (!sB && !(W.mu[b] < z)) adj.amu[b] = adj.amu[b] + h * fa;
        }
    }
    for (uint32_t i = 0; i < n; ++i) {
        st3(adj.av, i, ld3(adj.av, i) + dv[i]);
        st3(adj.aw, i, ld3(adj.aw, i) + dw[i]);
    }
}
#endif // host

} // namespace ad
} // namespace pe
