// Device narrowphase: one call produces one contact manifold for one collider
// pair.  Operation order follows src/collision/narrowphase.cpp (sphere-sphere
// :132-160, sphere-box :162-248, box-box :250-324, dispatch/swap :326-374) and
// src/collision/sat.cpp:38-102, so results are bit-identical to the reference
// under --fmad=false.  Feature ids (which the reference lacks) are
// (kind << 24) | (source << 16) | (face axis << 8) | (face sign << 4) | vertex.
// Convex hulls go through GJK (src/collision/gjk.cpp:11-158) and EPA
// (src/collision/epa.cpp:29-130) over support maps, with bounded polytope storage.
#pragma once
#include "pe_engine.h"
#include "pe_math.cuh"

namespace pe {

struct LocalManifold {
    V3 normal;
    uint32_t count;
    V3 anchorA[4];
    V3 anchorB[4];
    float depth[4];
    uint32_t feature[4];
};

__device__ __forceinline__ V3 boxSupport(const V3 &he, const Tf &tf, const V3 &dir) {
    V3 ld = rotate(conj(tf.q), dir);
    V3 lp{ld.x >= 0.0f ? he.x : -he.x, ld.y >= 0.0f ? he.y : -he.y, ld.z >= 0.0f ? he.z : -he.z};
    return toWorld(lp, tf);
}

__device__ __forceinline__ float boxProjectedRadius(const V3 &he, const M3 &r, const V3 &axis) {
    V3 a0{r.m00, r.m10, r.m20}, a1{r.m01, r.m11, r.m21}, a2{r.m02, r.m12, r.m22};
    return fabsf(dot(a0, axis)) * he.x + fabsf(dot(a1, axis)) * he.y + fabsf(dot(a2, axis)) * he.z;
}

// intersectSphereSphere (narrowphase.cpp:132-160)
__device__ __forceinline__ bool sphereSphere(float rA, const Tf &tA, float rB, const Tf &tB, LocalManifold &m) {
    V3 delta = tB.p - tA.p;
    float distance = length(delta);
    float radii = rA + rB;
    if (distance >= radii) return false;
    m.normal = distance > 1e-6f ? delta / distance : V3{1.0f, 0.0f, 0.0f};
    m.count = 1;
    m.depth[0] = radii - distance;
    V3 pA = tA.p + m.normal * rA;
    V3 pB = tB.p - m.normal * rB;
    V3 wc = (pA + pB) * 0.5f;
    m.anchorA[0] = toLocal(wc, tA);
    m.anchorB[0] = toLocal(wc, tB);
    m.feature[0] = kFeatSphereSphere << 24;
    return true;
}

// intersectSphereBox (narrowphase.cpp:162-248); region: 0..5 nearest face when
// the centre is inside, 6 outside.
__device__ __forceinline__ bool sphereBox(float r, const Tf &tS, const V3 &he, const Tf &tB, LocalManifold &m) {
    V3 c = rotate(conj(tB.q), tS.p - tB.p);
    V3 cl{clampv(c.x, -he.x, he.x), clampv(c.y, -he.y, he.y), clampv(c.z, -he.z, he.z)};
    V3 dl = cl - c;
    float distance = length(dl);
    V3 nl;
    float pen;
    uint32_t region;
    if (distance > 1e-6f) {
        if (distance >= r) return false;
        nl = dl / distance;
        pen = r - distance;
        region = 6;
    } else {
        float dpx = he.x - c.x, dnx = he.x + c.x, dpy = he.y - c.y, dny = he.y + c.y, dpz = he.z - c.z,
              dnz = he.z + c.z;
        float nearest = dpx;
        nl = {-1.0f, 0.0f, 0.0f};
        region = 0;
        if (dnx < nearest) { nearest = dnx; nl = {1.0f, 0.0f, 0.0f}; region = 1; }
        if (dpy < nearest) { nearest = dpy; nl = {0.0f, -1.0f, 0.0f}; region = 2; }
        if (dny < nearest) { nearest = dny; nl = {0.0f, 1.0f, 0.0f}; region = 3; }
        if (dpz < nearest) { nearest = dpz; nl = {0.0f, 0.0f, -1.0f}; region = 4; }
        if (dnz < nearest) { nearest = dnz; nl = {0.0f, 0.0f, 1.0f}; region = 5; }
        pen = r + nearest;
    }
    m.normal = rotate(tB.q, nl);
    m.count = 1;
    m.depth[0] = pen;
    V3 bp = toWorld(cl, tB);
    V3 sp = tS.p + m.normal * r;
    V3 wc = (sp + bp) * 0.5f;
    m.anchorA[0] = toLocal(wc, tS);
    m.anchorB[0] = toLocal(wc, tB);
    m.feature[0] = (kFeatSphereBox << 24) | region;
    return true;
}

// overlapOnAxis (sat.cpp:45-62); axes of a box are the columns of its matrix.
__device__ __forceinline__ bool satAxis(const M3 &rA, const V3 &heA, const M3 &rB, const V3 &heB, const V3 &cd,
                                        const V3 &axis, V3 &bestAxis, float &bestDepth) {
    float lsq = dot(axis, axis);
    if (lsq < 1e-8f) return true; // degenerate axis: depth = FLT_MAX never wins
    V3 na = axis * (1.0f / sqrtf(lsq));
    float distance = fabsf(dot(cd, na));
    float d = (boxProjectedRadius(heA, rA, na) + boxProjectedRadius(heB, rB, na)) - distance;
    if (d < 0.0f) return false;
    if (d < bestDepth) {
        bestDepth = d;
        bestAxis = na;
    }
    return true;
}

// Column j of a rotation matrix (a box's local axis j in world space).
__device__ __forceinline__ V3 matColumn(const M3 &r, int j) {
    return j == 0 ? V3{r.m00, r.m10, r.m20} : j == 1 ? V3{r.m01, r.m11, r.m21} : V3{r.m02, r.m12, r.m22};
}

// testOBBOBB (sat.cpp:66-102): face axes of A, of B, then A_i x B_j, in that
// order.  One rolled loop over the 15 axes: the kernel runs this once per pair,
// so a single copy of the axis test (fetched once) beats 15 unrolled copies.
__device__ __forceinline__ bool satBoxBox(const V3 &heA, const Tf &tA, const M3 &rA, const V3 &heB, const Tf &tB,
                                          const M3 &rB, V3 &axis, float &depth) {
    depth = 3.402823466e+38f;
    V3 cd = tB.p - tA.p;
#pragma unroll 1
    for (int t = 0; t < 15; ++t) {
        V3 ax;
        if (t < 3) ax = matColumn(rA, t);
        else if (t < 6) ax = matColumn(rB, t - 3);
        else ax = cross(matColumn(rA, (t - 6) / 3), matColumn(rB, (t - 6) % 3));
        if (!satAxis(rA, heA, rB, heB, cd, ax, axis, depth)) return false;
    }
    return true;
}

// addFaceCandidates (narrowphase.cpp:281-304) for one source box face.
// (not inlined: its two calls per box pair share one copy of the code)
static __device__ __noinline__ void boxFaceCandidates(const V3 &srcHe, const Tf &srcTf, const V3 &othHe, const Tf &othTf,
                                                  const V3 &dir, uint32_t source, V3 *contacts, float *depths,
                                                  uint32_t *feats, uint32_t &count) {
    float otherSurface = dot(boxSupport(othHe, othTf, -dir), dir);
    // supportFaceVertices (narrowphase.cpp:60-98)
    V3 ld = rotate(conj(srcTf.q), dir);
    int faceAxis = 0;
    float largest = fabsf(ld.x);
    if (fabsf(ld.y) > largest) { faceAxis = 1; largest = fabsf(ld.y); }
    if (fabsf(ld.z) > largest) faceAxis = 2;
    float comp = faceAxis == 0 ? ld.x : faceAxis == 1 ? ld.y : ld.z;
    float faceSign = comp >= 0.0f ? 1.0f : -1.0f;
    uint32_t signBit = comp >= 0.0f ? 0u : 1u;
    float ext[3] = {srcHe.x, srcHe.y, srcHe.z};
    int fa = (faceAxis + 1) % 3, sa = (faceAxis + 2) % 3;
    Q cq = conj(othTf.q);
    for (uint32_t vi = 0; vi < 4; ++vi) {
        float c[3] = {0.0f, 0.0f, 0.0f};
        c[faceAxis] = faceSign * ext[faceAxis];
        c[fa] = (vi & 1) ? ext[fa] : -ext[fa];
        c[sa] = (vi & 2) ? ext[sa] : -ext[sa];
        V3 v = toWorld(V3{c[0], c[1], c[2]}, srcTf);
        // pointInsideBox (narrowphase.cpp:100-107)
        V3 l = rotate(cq, v - othTf.p);
        const float tol = 1e-4f;
        if (!(fabsf(l.x) <= othHe.x + tol && fabsf(l.y) <= othHe.y + tol && fabsf(l.z) <= othHe.z + tol)) continue;
        float depth = smax(dot(v, dir) - otherSurface, 0.0f);
        V3 cand = v - dir * (depth * 0.5f);
        if (count >= 4) continue;
        // duplicatePoint (narrowphase.cpp:109-120)
        bool dup = false;
        for (uint32_t k = 0; k < count; ++k) {
            V3 dd = contacts[k] - cand;
            if (dot(dd, dd) <= 1e-6f) dup = true;
        }
        if (dup) continue;
        depths[count] = depth;
        feats[count] = (kFeatBoxFace << 24) | (source << 16) | ((uint32_t)faceAxis << 8) | (signBit << 4) | vi;
        contacts[count++] = cand;
    }
}

// overlapMidpoint (narrowphase.cpp:48-58)
__device__ __forceinline__ float boxOverlapMidpoint(const V3 &heA, const Tf &tA, const M3 &rA, const V3 &heB,
                                                    const Tf &tB, const M3 &rB, const V3 &ax) {
    float cA = dot(tA.p, ax), cB = dot(tB.p, ax);
    float ra = boxProjectedRadius(heA, rA, ax), rb = boxProjectedRadius(heB, rB, ax);
    float lower = smax(cA - ra, cB - rb);
    float upper = smin(cA + ra, cB + rb);
    return (lower + upper) * 0.5f;
}

// intersectBoxBox (narrowphase.cpp:250-324)
__device__ __forceinline__ bool boxBox(const V3 &heA, const Tf &tA, const V3 &heB, const Tf &tB, LocalManifold &m) {
    M3 rA = toMat3(tA.q), rB = toMat3(tB.q);
    V3 normal;
    float penetration;
    if (!satBoxBox(heA, tA, rA, heB, tB, rB, normal, penetration)) return false;
    V3 cd = tB.p - tA.p;
    if (dot(cd, normal) < 0.0f) normal = -normal;
    m.normal = normal;
    V3 contacts[4];
    float depths[4];
    uint32_t feats[4];
    uint32_t count = 0;
    boxFaceCandidates(heA, tA, heB, tB, normal, 0, contacts, depths, feats, count);
    boxFaceCandidates(heB, tB, heA, tA, -normal, 1, contacts, depths, feats, count);
    if (count == 0) {
        // Fallback contact (narrowphase.cpp:270-276, 308-312).
        V3 tref = fabsf(normal.x) < 0.9f ? V3{1.0f, 0.0f, 0.0f} : V3{0.0f, 1.0f, 0.0f};
        V3 t1 = normalize(cross(normal, tref));
        V3 t2 = cross(normal, t1);
        float nc = (dot(tA.p, normal) + boxProjectedRadius(heA, rA, normal) + dot(tB.p, normal) -
                    boxProjectedRadius(heB, rB, normal)) *
                   0.5f;
        contacts[0] = normal * nc + t1 * boxOverlapMidpoint(heA, tA, rA, heB, tB, rB, t1) +
                      t2 * boxOverlapMidpoint(heA, tA, rA, heB, tB, rB, t2);
        depths[0] = penetration;
        feats[0] = kFeatBoxFallback << 24;
        count = 1;
    }
    m.count = count;
    for (uint32_t i = 0; i < count; ++i) {
        m.depth[i] = depths[i];
        m.anchorA[i] = toLocal(contacts[i], tA);
        m.anchorB[i] = toLocal(contacts[i], tB);
        m.feature[i] = feats[i];
    }
    return true;
}

// ---------------------------------------------------------------------------
// GJK / EPA over support maps (box: boxSupportPoint; sphere: centre +
// normalize(d) * r; hull: first vertex of maximal d . v in body space).
// ---------------------------------------------------------------------------
constexpr int kEpaMaxVertices = 4 + 64;
constexpr int kEpaMaxFaces = 256;
constexpr int kEpaMaxHorizon = 128;

struct SupportShape {
    uint32_t shape;
    float radius;
    V3 he;
    const float4 *verts;
    uint32_t nverts;
    Tf tf;
};

__device__ __forceinline__ V3 support(const SupportShape &s, const V3 &dir, uint32_t &index) {
    if (s.shape == kShapeBox) return boxSupport(s.he, s.tf, dir);
    if (s.shape == kShapeSphere) return s.tf.p + normalize(dir) * s.radius;
    V3 ld = rotate(conj(s.tf.q), dir);
    uint32_t best = 0;
    float4 v0 = s.verts[0];
    float bd = dot(V3{v0.x, v0.y, v0.z}, ld);
    for (uint32_t i = 1; i < s.nverts; ++i) {
        float4 v = s.verts[i];
        float d = dot(V3{v.x, v.y, v.z}, ld);
        if (d > bd) { bd = d; best = i; }
    }
    index = best;
    float4 vb = s.verts[best];
    return toWorld(V3{vb.x, vb.y, vb.z}, s.tf);
}

struct Simplex {
    V3 p[4];
    uint32_t size;
};

__device__ __forceinline__ V3 tripleCross(const V3 &a, const V3 &b, const V3 &c) { return cross(cross(a, b), c); }

// setLineDirection (gjk.cpp:21-41)
__device__ inline void gjkLine(Simplex &s, V3 &dir) {
    V3 A = s.p[0], B = s.p[1];
    V3 toO = -A;
    V3 e = B - A;
    if (dot(e, toO) > 0.0f) {
        dir = tripleCross(e, toO, e);
        if (dot(dir, dir) < 1e-12f) dir = cross(e, V3{1.0f, 0.0f, 0.0f});
        if (dot(dir, dir) < 1e-12f) dir = cross(e, V3{0.0f, 1.0f, 0.0f});
    } else {
        s.size = 1;
        dir = toO;
    }
}
// setTriangleDirection (gjk.cpp:43-74)
__device__ inline void gjkTriangle(Simplex &s, V3 &dir) {
    V3 A = s.p[0], B = s.p[1], C = s.p[2];
    V3 toO = -A;
    V3 ab = B - A, ac = C - A;
    V3 n = cross(ab, ac);
    if (dot(cross(n, ac), toO) > 0.0f) {
        if (dot(ac, toO) > 0.0f) {
            s.p[1] = C;
            s.size = 2;
            dir = tripleCross(ac, toO, ac);
            return;
        }
        gjkLine(s, dir);
        return;
    }
    if (dot(cross(ab, n), toO) > 0.0f) {
        gjkLine(s, dir);
        return;
    }
    if (dot(n, toO) > 0.0f) {
        dir = n;
    } else {
        V3 t = s.p[1];
        s.p[1] = s.p[2];
        s.p[2] = t;
        dir = -n;
    }
}
// containsOrigin (gjk.cpp:76-124), including its third-face assignment through
// aliased references (the simplex becomes {A, D, D}).
__device__ inline bool gjkContains(Simplex &s, V3 &dir) {
    if (s.size == 1) {
        dir = -s.p[0];
        return false;
    }
    if (s.size == 2) {
        gjkLine(s, dir);
        return false;
    }
    if (s.size == 3) {
        gjkTriangle(s, dir);
        return false;
    }
    V3 A = s.p[0];
    V3 toO = -A;
    auto outside = [&](const V3 &fb, const V3 &fc, const V3 &op) {
        V3 n = cross(fb - A, fc - A);
        if (dot(n, op - A) > 0.0f) n = -n;
        return dot(n, toO) > 0.0f;
    };
    if (outside(s.p[1], s.p[2], s.p[3])) {
        s.size = 3;
        gjkTriangle(s, dir);
        return false;
    }
    if (outside(s.p[2], s.p[3], s.p[1])) {
        s.p[1] = s.p[2];
        s.p[2] = s.p[3];
        s.size = 3;
        gjkTriangle(s, dir);
        return false;
    }
    if (outside(s.p[3], s.p[1], s.p[2])) {
        s.p[1] = s.p[3];
        s.p[2] = s.p[1];
        s.size = 3;
        gjkTriangle(s, dir);
        return false;
    }
    return true;
}

__device__ inline bool gjk(const SupportShape &A, const SupportShape &B, Simplex &s) {
    s.size = 0;
    V3 dir{1.0f, 0.0f, 0.0f};
    uint32_t ia, ib;
    for (uint32_t it = 0; it < 32; ++it) {
        if (dot(dir, dir) < 1e-12f) break;
        V3 p = support(A, dir, ia) - support(B, -dir, ib);
        if (dot(p, dir) <= 0.0f) break;
        for (uint32_t i = s.size < 3u ? s.size : 3u; i > 0; --i) s.p[i] = s.p[i - 1];
        s.p[0] = p;
        s.size = s.size + 1 < 4u ? s.size + 1 : 4u;
        if (gjkContains(s, dir)) return true;
    }
    return false;
}

struct EpaFace {
    uint16_t a, b, c;
    V3 n;
    float d;
};

__device__ __forceinline__ EpaFace epaFace(const V3 *v, uint32_t a, uint32_t b, uint32_t c) {
    V3 n = cross(v[b] - v[a], v[c] - v[a]);
    float len = length(n);
    if (len > 1e-8f) n = n * (1.0f / len);
    float d = dot(n, v[a]);
    if (d < 0.0f) {
        uint32_t t = b;
        b = c;
        c = t;
        n = -n;
        d = -d;
    }
    return {(uint16_t)a, (uint16_t)b, (uint16_t)c, n, d};
}

// computeEpa (epa.cpp:64-130); 1 on success, 0 on failure (degenerate,
// iteration cap, or bounded storage exhausted).  Storage is per thread.
__device__ inline int epa(const SupportShape &A, const SupportShape &B, const Simplex &s, V3 &normal, float &depth) {
    normal = V3{0.0f, 0.0f, 0.0f};
    depth = 0.0f;
    if (s.size < 4) return 0;
    V3 v[kEpaMaxVertices];
    EpaFace faces[kEpaMaxFaces];
    uint16_t he[kEpaMaxHorizon][2];
    uint32_t nv = 0, nf = 0;
    for (uint32_t i = 0; i < s.size; ++i) v[nv++] = s.p[i];
    faces[nf++] = epaFace(v, 0, 1, 2);
    faces[nf++] = epaFace(v, 0, 3, 1);
    faces[nf++] = epaFace(v, 0, 2, 3);
    faces[nf++] = epaFace(v, 1, 3, 2);
    const float tol = 1e-4f;
    uint32_t ia, ib;
    for (uint32_t it = 0; it < 64; ++it) {
        if (nf == 0) return 0;
        uint32_t ci = 0;
        for (uint32_t f = 1; f < nf; ++f)
            if (faces[f].d < faces[ci].d) ci = f;
        EpaFace cf = faces[ci];
        V3 sup = support(A, cf.n, ia) - support(B, -cf.n, ib);
        float sd = dot(sup, cf.n);
        if (sd - cf.d <= tol) {
            normal = cf.n;
            depth = smax(cf.d, 0.0f);
            return 1;
        }
        if (nv >= (uint32_t)kEpaMaxVertices) return 0;
        uint32_t si = nv;
        v[nv++] = sup;
        uint32_t nh = 0;
        bool overflow = false;
        uint32_t kept = 0;
        for (uint32_t f = 0; f < nf; ++f) {
            const EpaFace face = faces[f];
            float vis = dot(face.n, sup - v[face.a]);
            if (vis > tol) {
                uint32_t e[3][2] = {{face.a, face.b}, {face.b, face.c}, {face.c, face.a}};
                for (int k = 0; k < 3; ++k) {
                    uint32_t a = e[k][0], b = e[k][1];
                    bool removed = false;
                    for (uint32_t q = 0; q < nh; ++q)
                        if (he[q][0] == b && he[q][1] == a) {
                            for (uint32_t r = q + 1; r < nh; ++r) {
                                he[r - 1][0] = he[r][0];
                                he[r - 1][1] = he[r][1];
                            }
                            --nh;
                            removed = true;
                            break;
                        }
                    if (!removed) {
                        if (nh >= (uint32_t)kEpaMaxHorizon) {
                            overflow = true;
                        } else {
                            he[nh][0] = (uint16_t)a;
                            he[nh][1] = (uint16_t)b;
                            ++nh;
                        }
                    }
                }
            } else {
                faces[kept++] = face;
            }
        }
        if (overflow || nh == 0) return 0;
        nf = kept;
        if (nf + nh > (uint32_t)kEpaMaxFaces) return 0;
        for (uint32_t k = 0; k < nh; ++k) faces[nf++] = epaFace(v, he[k][0], he[k][1], si);
    }
    return 0;
}

// Hull contact (project-defined): normal and depth from EPA (A toward B), one
// point midway between A's support along n and B's support along -n.
__device__ inline bool hullContact(const SupportShape &A, const SupportShape &B, LocalManifold &m, bool &epaFailed) {
    epaFailed = false;
    Simplex s;
    if (!gjk(A, B, s)) return false;
    V3 n;
    float depth;
    if (!epa(A, B, s, n, depth)) {
        epaFailed = true;
        return false;
    }
    uint32_t ia = 0xFFu, ib = 0xFFu;
    V3 pa = support(A, n, ia);
    V3 pb = support(B, -n, ib);
    if (A.shape != kShapeHull) ia = 0xFFu;
    if (B.shape != kShapeHull) ib = 0xFFu;
    V3 wc = (pa + pb) * 0.5f;
    m.normal = n;
    m.count = 1;
    m.depth[0] = depth;
    m.anchorA[0] = toLocal(wc, A.tf);
    m.anchorB[0] = toLocal(wc, B.tf);
    m.feature[0] = (kFeatHull << 24) | ((ia & 0xFFu) << 8) | (ib & 0xFFu);
    return true;
}


// The world's generateContact lambda (src/world/physics_world.cpp:645-691) for
// collider slots ca, cb (spheres and boxes: a batch's worlds) of bodies ba, bb: world
// transforms, shape dispatch with the box-sphere swap (narrowphase.cpp:353-365),
// anchors to body space, restitution = max, friction = sqrt(max(fa,0) * max(fb,0)).
// category: 0 sphere-sphere, 1 sphere-box, 2 box-box.
__device__ __forceinline__ bool narrowphasePair(const WorldView &w, uint32_t ca, uint32_t cb, uint32_t ba, uint32_t bb,
                                                LocalManifold &lm, float &restitution, float &friction,
                                                uint32_t &category) {
    lm.count = 0;
    const uint32_t sa = colliderShape(w.cflags[ca]), sb = colliderShape(w.cflags[cb]);
    V3 lpa = w.clpos ? f4xyz(w.clpos[ca]) : V3{0.0f, 0.0f, 0.0f};
    Q lqa = w.clrot ? f4q(w.clrot[ca]) : qidentity();
    V3 lpb = w.clpos ? f4xyz(w.clpos[cb]) : V3{0.0f, 0.0f, 0.0f};
    Q lqb = w.clrot ? f4q(w.clrot[cb]) : qidentity();
    V3 pa = f4xyz(w.cur.pos[ba]), pb = f4xyz(w.cur.pos[bb]);
    Q qa = f4q(w.cur.rot[ba]), qb = f4q(w.cur.rot[bb]);
    Tf tA{pa + rotate(qa, lpa), qmul(qa, lqa)};
    Tf tB{pb + rotate(qb, lpb), qmul(qb, lqb)};
    const float4 sha = w.cshape[ca], shb = w.cshape[cb];
    const V3 ha{sha.x, sha.y, sha.z}, hb{shb.x, shb.y, shb.z};
    category = sa + sb;
    bool hit;
    if (sa == kShapeSphere && sb == kShapeSphere) {
        hit = sphereSphere(sha.x, tA, shb.x, tB, lm);
    } else if (sa == kShapeSphere) {
        hit = sphereBox(sha.x, tA, hb, tB, lm);
    } else if (sb == kShapeSphere) {
        hit = sphereBox(shb.x, tB, ha, tA, lm);
        if (hit) {
            lm.normal = -lm.normal;
            const V3 t = lm.anchorA[0];
            lm.anchorA[0] = lm.anchorB[0];
            lm.anchorB[0] = t;
        }
    } else {
        hit = boxBox(ha, tA, hb, tB, lm);
    }
    if (hit) {
        for (uint32_t k = 0; k < lm.count; ++k) {
            lm.anchorA[k] = lpa + rotate(lqa, lm.anchorA[k]);
            lm.anchorB[k] = lpb + rotate(lqb, lm.anchorB[k]);
        }
        const float4 ma = w.mat[ba], mb = w.mat[bb];
        restitution = smax(ma.y, mb.y);
        friction = sqrtf(smax(ma.z, 0.0f) * smax(mb.z, 0.0f));
    }
    return hit;
}

// ------------------------------------------------------------------ lanes ---
// A pair on eight lanes of a warp (the multi-kernel step's narrowphase).
//
// A box pair is some 7,000 cycles of dependent arithmetic on one thread: fifteen
// axes with a square root and two divisions each, then eight face vertices, with
// the contacts in local memory.  The lanes take two axes and one vertex each, and
// a contact stays in its lane's registers.  The operations of an axis and of a
// vertex are those of satBoxBox and boxFaceCandidates; what those decide in order
// (the first smallest depth; a vertex is dropped when it is close to one kept
// before it or four are kept) is decided here from the lanes' results in that
// order.
constexpr uint32_t kPairLanes = 8;

// What a pair's lanes hold of its manifold: the lane's contact, if it has one.
struct LaneManifold {
    bool hit;
    uint32_t count;  // of the manifold
    V3 normal;
    bool mine;       // the lane has contact `slot`
    uint32_t slot;
    V3 anchorA, anchorB;
    float depth;
    uint32_t feature;
};

__device__ __forceinline__ V3 laneShfl(const V3 &v, uint32_t from) {
    return {__shfl_sync(0xffffffffu, v.x, from, kPairLanes), __shfl_sync(0xffffffffu, v.y, from, kPairLanes),
            __shfl_sync(0xffffffffu, v.z, from, kPairLanes)};
}
__device__ __forceinline__ V3 pick(bool first, const V3 &a, const V3 &b) {
    return {first ? a.x : b.x, first ? a.y : b.y, first ? a.z : b.z};
}

// boxBox on the lanes of a pair; whole warps call it, act: the lane's pair is
// one of two boxes.  Anchors in collider space.
__device__ __forceinline__ void boxBoxLanes(bool act, const V3 &heA, const Tf &tA, const V3 &heB, const Tf &tB,
                                            LaneManifold &o) {
    const uint32_t t = threadIdx.x & (kPairLanes - 1), shift = threadIdx.x & 24u;
    const M3 rA = toMat3(tA.q), rB = toMat3(tB.q);
    const V3 cd = tB.p - tA.p;
    // two axes a lane (satBoxBox's order: t, then t + 8)
    float best = 3.402823466e+38f;
    uint32_t bestAxis = 16;
    V3 normal{0.0f, 0.0f, 0.0f};
    bool apart = false;
#pragma unroll
    for (uint32_t r = 0; r < 2; ++r) {
        const uint32_t k = t + r * kPairLanes;
        V3 ax;
        if (r == 0 && k < 6) {
            ax = k < 3 ? matColumn(rA, (int)k) : matColumn(rB, (int)k - 3);
        } else {
            const uint32_t e = k - 6, i = e < 3 ? 0 : e < 6 ? 1 : 2;
            ax = cross(matColumn(rA, (int)i), matColumn(rB, (int)(e - 3 * i)));
        }
        if (k < 15) {
            const float before = best;
            if (!satAxis(rA, heA, rB, heB, cd, ax, normal, best)) apart = true;
            if (best < before) bestAxis = k;
        }
    }
    const uint32_t separated = (__ballot_sync(0xffffffffu, apart) >> shift) & 0xFFu;
    const bool hit = act && separated == 0;
#pragma unroll
    for (uint32_t j = 1; j < kPairLanes; j <<= 1) {
        const float d = __shfl_xor_sync(0xffffffffu, best, j);
        const uint32_t k = __shfl_xor_sync(0xffffffffu, bestAxis, j);
        if (d < best || (d == best && k < bestAxis)) {
            best = d;
            bestAxis = k;
        }
    }
    normal = laneShfl(normal, bestAxis & (kPairLanes - 1));
    if (dot(cd, normal) < 0.0f) normal = -normal;
    // one face vertex a lane: box A's face along the normal, then box B's
    const bool fromA = t < 4;
    const uint32_t vi = t & 3;
    const V3 dir = pick(fromA, normal, -normal);
    const V3 srcHe = pick(fromA, heA, heB), othHe = pick(fromA, heB, heA);
    const Tf srcTf{pick(fromA, tA.p, tB.p), fromA ? tA.q : tB.q}, othTf{pick(fromA, tB.p, tA.p), fromA ? tB.q : tA.q};
    const float otherSurface = dot(boxSupport(othHe, othTf, -dir), dir);
    const V3 ld = rotate(conj(srcTf.q), dir);
    int faceAxis = 0;
    float largest = fabsf(ld.x);
    if (fabsf(ld.y) > largest) { faceAxis = 1; largest = fabsf(ld.y); }
    if (fabsf(ld.z) > largest) faceAxis = 2;
    const float comp = faceAxis == 0 ? ld.x : faceAxis == 1 ? ld.y : ld.z;
    const bool positive = comp >= 0.0f, first = vi & 1, second = vi & 2;
    // (the face's first side axis follows the face axis, the second follows that)
    const bool upX = faceAxis == 0 ? positive : faceAxis == 2 ? first : second;
    const bool upY = faceAxis == 1 ? positive : faceAxis == 0 ? first : second;
    const bool upZ = faceAxis == 2 ? positive : faceAxis == 1 ? first : second;
    const V3 v = toWorld(V3{upX ? srcHe.x : -srcHe.x, upY ? srcHe.y : -srcHe.y, upZ ? srcHe.z : -srcHe.z}, srcTf);
    const V3 l = rotate(conj(othTf.q), v - othTf.p);
    const float tol = 1e-4f;
    const bool inside = fabsf(l.x) <= othHe.x + tol && fabsf(l.y) <= othHe.y + tol && fabsf(l.z) <= othHe.z + tol;
    float depth = smax(dot(v, dir) - otherSurface, 0.0f);
    V3 contact = v - dir * (depth * 0.5f);
    uint32_t feature = (kFeatBoxFace << 24) | ((fromA ? 0u : 1u) << 16) | ((uint32_t)faceAxis << 8) |
                       ((positive ? 0u : 1u) << 4) | vi;
    uint32_t near = 0;  // vertices within the duplicate distance of this lane's
#pragma unroll
    for (uint32_t q = 0; q < kPairLanes; ++q) {
        const V3 d = laneShfl(contact, q) - contact;
        if (dot(d, d) <= 1e-6f) near |= 1u << q;
    }
    const uint32_t in = (__ballot_sync(0xffffffffu, inside) >> shift) & 0xFFu;
    uint32_t kept = 0, count = 0;
#pragma unroll
    for (uint32_t q = 0; q < kPairLanes; ++q) {
        const uint32_t nq = __shfl_sync(0xffffffffu, near, q, kPairLanes);
        if (((in >> q) & 1u) && count < 4 && !(nq & kept)) {
            kept |= 1u << q;
            ++count;
        }
    }
    if (!act) return;
    o.hit = hit;
    o.normal = normal;
    o.count = count;
    o.mine = (kept >> t) & 1u;
    o.slot = __popc(kept & ((1u << t) - 1u));
    if (hit && count == 0) {
        // Fallback contact (narrowphase.cpp:270-276, 308-312), as in boxBox.
        V3 tref = fabsf(normal.x) < 0.9f ? V3{1.0f, 0.0f, 0.0f} : V3{0.0f, 1.0f, 0.0f};
        V3 t1 = normalize(cross(normal, tref));
        V3 t2 = cross(normal, t1);
        float nc = (dot(tA.p, normal) + boxProjectedRadius(heA, rA, normal) + dot(tB.p, normal) -
                    boxProjectedRadius(heB, rB, normal)) *
                   0.5f;
        contact = normal * nc + t1 * boxOverlapMidpoint(heA, tA, rA, heB, tB, rB, t1) +
                  t2 * boxOverlapMidpoint(heA, tA, rA, heB, tB, rB, t2);
        depth = best;
        feature = kFeatBoxFallback << 24;
        o.count = 1;
        o.mine = t == 0;
        o.slot = 0;
    }
    o.depth = depth;
    o.anchorA = toLocal(contact, tA);
    o.anchorB = toLocal(contact, tB);
    o.feature = feature;
}

// One contact of a pair that is not two boxes, on its first lane.
__device__ __forceinline__ bool singleContact(const WorldView &w, uint32_t sa, const float4 &sha, const Tf &tA,
                                              uint32_t sb, const float4 &shb, const Tf &tB, LocalManifold &lm,
                                              bool &epaFailed) {
    if (sa == kShapeHull || sb == kShapeHull) {
        auto support = [&](uint32_t shape, const float4 &sh, const Tf &t) {
            SupportShape s;
            s.shape = shape;
            s.radius = sh.x;
            s.he = V3{sh.x, sh.y, sh.z};
            s.tf = t;
            s.verts = nullptr;
            s.nverts = 0;
            if (shape == kShapeHull) {
                const uint32_t h = __float_as_uint(sh.w);
                const uint32_t b = w.hullOffset[h];
                s.verts = w.hullVerts + b;
                s.nverts = w.hullOffset[h + 1] - b;
            }
            return s;
        };
        return hullContact(support(sa, sha, tA), support(sb, shb, tB), lm, epaFailed);
    }
    if (sa == kShapeSphere && sb == kShapeSphere) return sphereSphere(sha.x, tA, shb.x, tB, lm);
    if (sa == kShapeSphere) return sphereBox(sha.x, tA, V3{shb.x, shb.y, shb.z}, tB, lm);
    if (!sphereBox(shb.x, tB, V3{sha.x, sha.y, sha.z}, tA, lm)) return false;
    lm.normal = -lm.normal;
    const V3 t = lm.anchorA[0];
    lm.anchorA[0] = lm.anchorB[0];
    lm.anchorB[0] = t;
    return true;
}

// A collider's packed record (WorldView::npRec, written by the integrate kernel:
// world transform, shape, material, body): one 64-byte line instead of a gather
// from a dozen arrays.
struct PairSide {
    Tf t;
    float4 dims;
    float restitution, friction;
    uint32_t shape, body, gen;
};
__device__ __forceinline__ PairSide loadPairSide(const WorldView &w, uint32_t collider) {
    const float4 *r = w.npRec + 4 * (size_t)collider;
    const float4 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
    return {Tf{f4xyz(r0), f4q(r1)}, make_float4(r0.w, r2.x, r2.y, r2.z), r3.x, r3.y,
            colliderShape(__float_as_uint(r2.w)), __float_as_uint(r3.z), __float_as_uint(r3.w)};
}
// Category of a pair's counters, and what a contact takes from both materials.
__device__ __forceinline__ uint32_t pairCategory(const PairSide &a, const PairSide &b) {
    return a.shape == kShapeHull || b.shape == kShapeHull ? 3u : a.shape + b.shape;
}
__device__ __forceinline__ void pairMaterial(const PairSide &a, const PairSide &b, float &restitution,
                                             float &friction) {
    restitution = smax(a.restitution, b.restitution);
    friction = sqrtf(smax(a.friction, 0.0f) * smax(b.friction, 0.0f));
}
// An anchor from collider space to body space (local transforms only when some
// collider has one).
__device__ __forceinline__ V3 bodyAnchor(const WorldView &w, uint32_t collider, const V3 &anchor) {
    const V3 lp = w.clpos ? f4xyz(w.clpos[collider]) : V3{0.0f, 0.0f, 0.0f};
    const Q lq = w.clrot ? f4q(w.clrot[collider]) : qidentity();
    return lp + rotate(lq, anchor);
}

// The world's generateContact lambda from the records, on one thread and on the lanes of a pair
// (whole warps call it; act: the lanes have a pair).
__device__ __forceinline__ bool narrowphaseRecords(const WorldView &w, uint32_t ca, uint32_t cb, const PairSide &a,
                                                   const PairSide &b, LocalManifold &lm, float &restitution,
                                                   float &friction, bool &epaFailed) {
    epaFailed = false;
    lm.count = 0;
    const bool boxes = a.shape == kShapeBox && b.shape == kShapeBox;
    if (!(boxes ? boxBox(V3{a.dims.x, a.dims.y, a.dims.z}, a.t, V3{b.dims.x, b.dims.y, b.dims.z}, b.t, lm)
                : singleContact(w, a.shape, a.dims, a.t, b.shape, b.dims, b.t, lm, epaFailed)))
        return false;
    for (uint32_t k = 0; k < lm.count; ++k) {
        lm.anchorA[k] = bodyAnchor(w, ca, lm.anchorA[k]);
        lm.anchorB[k] = bodyAnchor(w, cb, lm.anchorB[k]);
    }
    pairMaterial(a, b, restitution, friction);
    return true;
}
__device__ __forceinline__ void narrowphaseLanes(const WorldView &w, bool act, uint32_t ca, uint32_t cb,
                                                 const PairSide &a, const PairSide &b, LaneManifold &o,
                                                 float &restitution, float &friction, bool &epaFailed) {
    epaFailed = false;
    o.hit = o.mine = false;
    o.count = o.slot = 0;
    const bool boxes = act && a.shape == kShapeBox && b.shape == kShapeBox;
    if (__any_sync(0xffffffffu, boxes))
        boxBoxLanes(boxes, V3{a.dims.x, a.dims.y, a.dims.z}, a.t, V3{b.dims.x, b.dims.y, b.dims.z}, b.t, o);
    if (act && !boxes && (threadIdx.x & (kPairLanes - 1)) == 0) {
        LocalManifold lm;
        o.hit = singleContact(w, a.shape, a.dims, a.t, b.shape, b.dims, b.t, lm, epaFailed);
        if (o.hit) {
            o.mine = true;
            o.count = 1;
            o.normal = lm.normal;
            o.anchorA = lm.anchorA[0];
            o.anchorB = lm.anchorB[0];
            o.depth = lm.depth[0];
            o.feature = lm.feature[0];
        }
    }
    if (!o.hit) return;
    o.anchorA = bodyAnchor(w, ca, o.anchorA);
    o.anchorB = bodyAnchor(w, cb, o.anchorB);
    pairMaterial(a, b, restitution, friction);
}

// Writes one manifold record in pair order: body handles, collider-space
// anchors already moved to body space, zero impulses.
__device__ __forceinline__ void storeManifoldGen(const ManifoldView &out, uint32_t m, uint32_t ba, uint32_t genA,
                                                 uint32_t bb, uint32_t genB, const LocalManifold &lm,
                                                 float restitution, float friction) {
    out.bodyA[m] = ba;
    out.genA[m] = genA;
    out.bodyB[m] = bb;
    out.genB[m] = genB;
    out.normalFriction[m] = make4(lm.normal, friction);
    out.restitution[m] = restitution;
    out.pointCount[m] = lm.count;
    for (uint32_t k = 0; k < 4; ++k) {
        const bool live = k < lm.count;
        out.anchorA[4 * m + k] = live ? make4(lm.anchorA[k], lm.depth[k]) : make_float4(0, 0, 0, 0);
        out.anchorB[4 * m + k] = live ? make4(lm.anchorB[k], 0.0f) : make_float4(0, 0, 0, 0);
        out.impulse[4 * m + k] = make_float4(0, 0, 0, 0);
        out.feature[4 * m + k] = live ? lm.feature[k] : 0u;
    }
}

// storeManifold with the body handles taken from the colliders.
__device__ __forceinline__ void storeManifold(const ManifoldView &out, uint32_t m, const WorldView &w, uint32_t ca,
                                              uint32_t cb, uint32_t ba, uint32_t bb, const LocalManifold &lm,
                                              float restitution, float friction) {
    storeManifoldGen(out, m, ba, w.cbgen[ca], bb, w.cbgen[cb], lm, restitution, friction);
}

} // namespace pe
