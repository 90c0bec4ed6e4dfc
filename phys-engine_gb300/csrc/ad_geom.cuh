// Scalar-generic contact geometry and contact preparation for the
// differentiable rollout (sphere / box colliders, one per body, identity local
// transforms).  The operations mirror the engine's device narrowphase and
// prepare step, which follow src/collision/narrowphase.cpp (sphere-sphere
// :132-160, sphere-box :162-248, box-box :250-324, dispatch :326-374),
// src/collision/sat.cpp:38-102 and sequential_impulse_solver.cpp:101-214.
// The reverse functions differentiate the contact that the forward evaluation
// produced with its discrete choices (separating axis, kept vertices, clamps)
// held; the axis and the vertex travel in the feature ids.
#pragma once
#include "ad_math.cuh"

namespace pe {
namespace ad {

enum : uint32_t { kAdFeatSphereSphere = 1, kAdFeatSphereBox = 2, kAdFeatBoxFace = 3, kAdFeatBoxFallback = 4 };

template <class S> struct Contact {
    V3<S> normal;
    uint32_t count;
    V3<S> anchorA[4];
    V3<S> anchorB[4];
    S depth[4];
    uint32_t feature[4];
    uint32_t axis;  // box-box: separating axis kept, in the order they are tested (0-14)
};
// The axis in a feature id (bits 20-23 are free there).
constexpr uint32_t kAdAxisShift = 20, kAdAxisMask = 0xFu << kAdAxisShift;

template <class S> AD_HD V3<S> cst(float x, float y, float z) { return {ADL(S, x), ADL(S, y), ADL(S, z)}; }

template <class S> AD_HD V3<S> boxSupport(const V3<S> &he, const Tf<S> &tf, const V3<S> &dir) {
    V3<S> ld = rotate(conj(tf.q), dir);
    V3<S> lp{val(ld.x) >= 0.0f ? he.x : -he.x, val(ld.y) >= 0.0f ? he.y : -he.y, val(ld.z) >= 0.0f ? he.z : -he.z};
    return toWorld(lp, tf);
}

template <class S> AD_HD S boxProjectedRadius(const V3<S> &he, const M3<S> &r, const V3<S> &axis) {
    V3<S> a0{r.m00, r.m10, r.m20}, a1{r.m01, r.m11, r.m21}, a2{r.m02, r.m12, r.m22};
    return sabs(dot(a0, axis)) * he.x + sabs(dot(a1, axis)) * he.y + sabs(dot(a2, axis)) * he.z;
}

// intersectSphereSphere (narrowphase.cpp:132-160)
template <class S>
AD_HDN bool sphereSphere(const S &rA, const Tf<S> &tA, const S &rB, const Tf<S> &tB, Contact<S> &m) {
    V3<S> delta = tB.p - tA.p;
    S distance = length(delta);
    S radii = rA + rB;
    if (val(distance) >= val(radii)) return false;
    m.normal = val(distance) > 1e-6f ? delta / distance : cst<S>(1.0f, 0.0f, 0.0f);
    m.count = 1;
    m.depth[0] = radii - distance;
    V3<S> pA = tA.p + m.normal * rA;
    V3<S> pB = tB.p - m.normal * rB;
    V3<S> wc = (pA + pB) * ADL(S, 0.5f);
    m.anchorA[0] = toLocal(wc, tA);
    m.anchorB[0] = toLocal(wc, tB);
    m.feature[0] = kAdFeatSphereSphere << 24;
    return true;
}

// intersectSphereBox (narrowphase.cpp:162-248)
template <class S>
AD_HDN bool sphereBox(const S &r, const Tf<S> &tS, const V3<S> &he, const Tf<S> &tB, Contact<S> &m) {
    V3<S> c = rotate(conj(tB.q), tS.p - tB.p);
    V3<S> cl{clampv(c.x, -he.x, he.x), clampv(c.y, -he.y, he.y), clampv(c.z, -he.z, he.z)};
    V3<S> dl = cl - c;
    S distance = length(dl);
    V3<S> nl;
    S pen;
    uint32_t region;
    if (val(distance) > 1e-6f) {
        if (val(distance) >= val(r)) return false;
        nl = dl / distance;
        pen = r - distance;
        region = 6;
    } else {
        S dpx = he.x - c.x, dnx = he.x + c.x, dpy = he.y - c.y, dny = he.y + c.y, dpz = he.z - c.z, dnz = he.z + c.z;
        S nearest = dpx;
        nl = cst<S>(-1.0f, 0.0f, 0.0f);
        region = 0;
        if (val(dnx) < val(nearest)) { nearest = dnx; nl = cst<S>(1.0f, 0.0f, 0.0f); region = 1; }
        if (val(dpy) < val(nearest)) { nearest = dpy; nl = cst<S>(0.0f, -1.0f, 0.0f); region = 2; }
        if (val(dny) < val(nearest)) { nearest = dny; nl = cst<S>(0.0f, 1.0f, 0.0f); region = 3; }
        if (val(dpz) < val(nearest)) { nearest = dpz; nl = cst<S>(0.0f, 0.0f, -1.0f); region = 4; }
        if (val(dnz) < val(nearest)) { nearest = dnz; nl = cst<S>(0.0f, 0.0f, 1.0f); region = 5; }
        pen = r + nearest;
    }
    m.normal = rotate(tB.q, nl);
    m.count = 1;
    m.depth[0] = pen;
    V3<S> bp = toWorld(cl, tB);
    V3<S> sp = tS.p + m.normal * r;
    V3<S> wc = (sp + bp) * ADL(S, 0.5f);
    m.anchorA[0] = toLocal(wc, tS);
    m.anchorB[0] = toLocal(wc, tB);
    m.feature[0] = (kAdFeatSphereBox << 24) | region;
    return true;
}

// overlapOnAxis (sat.cpp:45-62)
template <class S>
AD_HD bool satAxis(const M3<S> &rA, const V3<S> &heA, const M3<S> &rB, const V3<S> &heB, const V3<S> &cd,
                   const V3<S> &axis, uint32_t index, V3<S> &bestAxis, S &bestDepth, uint32_t &bestIndex) {
    S lsq = dot(axis, axis);
    if (val(lsq) < 1e-8f) return true;
    V3<S> na = axis * (ADL(S, 1.0f) / ssqrt(lsq));
    S distance = sabs(dot(cd, na));
    S d = (boxProjectedRadius(heA, rA, na) + boxProjectedRadius(heB, rB, na)) - distance;
    if (val(d) < 0.0f) return false;
    if (val(d) < val(bestDepth)) {
        bestDepth = d;
        bestAxis = na;
        bestIndex = index;
    }
    return true;
}

// testOBBOBB (sat.cpp:66-102)
template <class S>
AD_HDN bool satBoxBox(const V3<S> &heA, const Tf<S> &tA, const M3<S> &rA, const V3<S> &heB, const Tf<S> &tB,
                     const M3<S> &rB, V3<S> &axis, S &depth, uint32_t &index) {
    index = 0;
    depth = ADL(S, 3.402823466e+38f);
    V3<S> cd = tB.p - tA.p;
    V3<S> ax[3] = {{rA.m00, rA.m10, rA.m20}, {rA.m01, rA.m11, rA.m21}, {rA.m02, rA.m12, rA.m22}};
    V3<S> bx[3] = {{rB.m00, rB.m10, rB.m20}, {rB.m01, rB.m11, rB.m21}, {rB.m02, rB.m12, rB.m22}};
    for (int i = 0; i < 3; ++i)
        if (!satAxis(rA, heA, rB, heB, cd, ax[i], (uint32_t)i, axis, depth, index)) return false;
    for (int i = 0; i < 3; ++i)
        if (!satAxis(rA, heA, rB, heB, cd, bx[i], 3u + i, axis, depth, index)) return false;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            if (!satAxis(rA, heA, rB, heB, cd, cross(ax[i], bx[j]), 6u + 3u * i + j, axis, depth, index)) return false;
    return true;
}

// addFaceCandidates (narrowphase.cpp:281-304) for one source box face.
template <class S>
AD_HDN void boxFaceCandidates(const V3<S> &srcHe, const Tf<S> &srcTf, const V3<S> &othHe, const Tf<S> &othTf,
                             const V3<S> &dir, uint32_t source, V3<S> *contacts, S *depths, uint32_t *feats,
                             uint32_t &count) {
    S otherSurface = dot(boxSupport(othHe, othTf, -dir), dir);
    V3<S> ld = rotate(conj(srcTf.q), dir);
    int faceAxis = 0;
    float largest = sabs(val(ld.x));
    if (sabs(val(ld.y)) > largest) { faceAxis = 1; largest = sabs(val(ld.y)); }
    if (sabs(val(ld.z)) > largest) faceAxis = 2;
    const S comp = faceAxis == 0 ? ld.x : faceAxis == 1 ? ld.y : ld.z;
    const S one = ADL(S, 1.0f);
    S faceSign = val(comp) >= 0.0f ? one : -one;
    uint32_t signBit = val(comp) >= 0.0f ? 0u : 1u;
    S ext[3] = {srcHe.x, srcHe.y, srcHe.z};
    int fa = (faceAxis + 1) % 3, sa = (faceAxis + 2) % 3;
    Q<S> cq = conj(othTf.q);
    for (uint32_t vi = 0; vi < 4; ++vi) {
        S c[3] = {ADL(S, 0.0f), ADL(S, 0.0f), ADL(S, 0.0f)};
        c[faceAxis] = faceSign * ext[faceAxis];
        c[fa] = (vi & 1) ? ext[fa] : -ext[fa];
        c[sa] = (vi & 2) ? ext[sa] : -ext[sa];
        V3<S> v = toWorld(V3<S>{c[0], c[1], c[2]}, srcTf);
        V3<S> l = rotate(cq, v - othTf.p);
        const float tol = 1e-4f;
        if (!(sabs(val(l.x)) <= val(othHe.x) + tol && sabs(val(l.y)) <= val(othHe.y) + tol &&
              sabs(val(l.z)) <= val(othHe.z) + tol))
            continue;
        S depth = smax(dot(v, dir) - otherSurface, ADL(S, 0.0f));
        V3<S> cand = v - dir * (depth * ADL(S, 0.5f));
        if (count >= 4) continue;
        bool dup = false;
        for (uint32_t k = 0; k < count; ++k) {
            V3<S> dd = contacts[k] - cand;
            if (val(dot(dd, dd)) <= 1e-6f) dup = true;
        }
        if (dup) continue;
        depths[count] = depth;
        feats[count] = (kAdFeatBoxFace << 24) | (source << 16) | ((uint32_t)faceAxis << 8) | (signBit << 4) | vi;
        contacts[count++] = cand;
    }
}

// intersectBoxBox (narrowphase.cpp:250-324)
template <class S>
AD_HDN bool boxBox(const V3<S> &heA, const Tf<S> &tA, const V3<S> &heB, const Tf<S> &tB, Contact<S> &m) {
    M3<S> rA = toMat3(tA.q), rB = toMat3(tB.q);
    V3<S> normal;
    S penetration;
    if (!satBoxBox(heA, tA, rA, heB, tB, rB, normal, penetration, m.axis)) return false;
    V3<S> cd = tB.p - tA.p;
    if (val(dot(cd, normal)) < 0.0f) normal = -normal;
    m.normal = normal;
    V3<S> contacts[4];
    S depths[4];
    uint32_t feats[4];
    uint32_t count = 0;
    boxFaceCandidates(heA, tA, heB, tB, normal, 0, contacts, depths, feats, count);
    boxFaceCandidates(heB, tB, heA, tA, -normal, 1, contacts, depths, feats, count);
    if (count == 0) {
        V3<S> tref = sabs(val(normal.x)) < 0.9f ? cst<S>(1.0f, 0.0f, 0.0f) : cst<S>(0.0f, 1.0f, 0.0f);
        V3<S> t1 = normalize(cross(normal, tref));
        V3<S> t2 = cross(normal, t1);
        S nc = (dot(tA.p, normal) + boxProjectedRadius(heA, rA, normal) + dot(tB.p, normal) -
                boxProjectedRadius(heB, rB, normal)) *
               ADL(S, 0.5f);
        auto mid = [&](const V3<S> &ax) {
            S cA = dot(tA.p, ax), cB = dot(tB.p, ax);
            S ra = boxProjectedRadius(heA, rA, ax), rb = boxProjectedRadius(heB, rB, ax);
            S lower = smax(cA - ra, cB - rb);
            S upper = smin(cA + ra, cB + rb);
            return (lower + upper) * ADL(S, 0.5f);
        };
        contacts[0] = normal * nc + t1 * mid(t1) + t2 * mid(t2);
        depths[0] = penetration;
        feats[0] = kAdFeatBoxFallback << 24;
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

// Shape dispatch with the box-sphere swap (narrowphase.cpp:326-374).
// shape: 0 sphere (dims.x = radius), 1 box (dims = half extents).
template <class S>
AD_HDN bool contactPair(uint32_t sa, const V3<S> &da, const Tf<S> &tA, uint32_t sb, const V3<S> &db,
                       const Tf<S> &tB, Contact<S> &m) {
    m.count = 0;
    m.axis = 0;
    bool hit;
    if (sa == 0 && sb == 0) {
        hit = sphereSphere(da.x, tA, db.x, tB, m);
    } else if (sa == 0) {
        hit = sphereBox(da.x, tA, db, tB, m);
    } else if (sb == 0) {
        hit = sphereBox(db.x, tB, da, tA, m);
        if (hit) {
            m.normal = -m.normal;
            for (uint32_t k = 0; k < m.count; ++k) {
                V3<S> t = m.anchorA[k];
                m.anchorA[k] = m.anchorB[k];
                m.anchorB[k] = t;
            }
        }
    } else {
        hit = boxBox(da, tA, db, tB, m);
    }
    return hit;
}

// ------------------------------------------------------ reverse: geometry ---
// Adjoint of one contact point: anchors, depth.  Every function adds to the
// adjoints of the two poses; the normal's goes through normalReverse*, once a
// manifold.
template <class S> struct PointGrad {
    V3<S> anchorA, anchorB;
    S depth;
};

template <class S> AD_HD V3<S> column(const M3<S> &m, uint32_t k) {
    return k == 0 ? V3<S>{m.m00, m.m10, m.m20} : k == 1 ? V3<S>{m.m01, m.m11, m.m21} : V3<S>{m.m02, m.m12, m.m22};
}
template <class S> AD_HD void addColumn(M3<S> &m, uint32_t k, const V3<S> &v) {
    const S z = S(0), s0 = k == 0 ? S(1) : z, s1 = k == 1 ? S(1) : z, s2 = k == 2 ? S(1) : z;
    m.m00 = m.m00 + s0 * v.x;
    m.m10 = m.m10 + s0 * v.y;
    m.m20 = m.m20 + s0 * v.z;
    m.m01 = m.m01 + s1 * v.x;
    m.m11 = m.m11 + s1 * v.y;
    m.m21 = m.m21 + s1 * v.z;
    m.m02 = m.m02 + s2 * v.x;
    m.m12 = m.m12 + s2 * v.y;
    m.m22 = m.m22 + s2 * v.z;
}
// d = delta / |delta|
template <class S> AD_HD V3<S> unitAdj(const V3<S> &unit, const S &len, const V3<S> &g) {
    return (g - unit * dot(unit, g)) / len;
}

// wc -> both anchors.
template <class S>
AD_HD V3<S> anchorsReverse(const V3<S> &wc, const Tf<S> &tA, const Tf<S> &tB, const PointGrad<S> &g, Tf<S> &gA,
                           Tf<S> &gB) {
    V3<S> w{S(0), S(0), S(0)};
    toLocalAdj(wc, tA, g.anchorA, gA, w);
    toLocalAdj(wc, tB, g.anchorB, gB, w);
    return w;
}

template <class S>
AD_HD void sphereSphereReverse(const S &rA, const Tf<S> &tA, const S &rB, const Tf<S> &tB, const V3<S> &normal,
                               const PointGrad<S> &g, V3<S> gn, Tf<S> &gA, Tf<S> &gB) {
    const V3<S> delta = tB.p - tA.p;
    const S distance = length(delta), half = S(0.5f);
    const V3<S> pA = tA.p + normal * rA, pB = tB.p - normal * rB;
    const V3<S> w = anchorsReverse((pA + pB) * half, tA, tB, g, gA, gB) * half;
    gn += w * (rA - rB);
    gA.p += w;
    gB.p += w;
    if (distance > S(0)) {
        V3<S> gd = delta * (-g.depth / distance);
        if (distance > 1e-6f) gd += unitAdj(normal, distance, gn);
        gB.p += gd;
        gA.p += -gd;
    }
}

// Sphere S against box B in that order (the caller swaps anchors and normal).
template <class S>
AD_HD void sphereBoxReverse(const S &r, const Tf<S> &tS, const V3<S> &he, const Tf<S> &tB, const V3<S> &normal,
                            const PointGrad<S> &g, V3<S> gn, Tf<S> &gS, Tf<S> &gB) {
    const S z = S(0), half = S(0.5f);
    const V3<S> c = rotate(conj(tB.q), tS.p - tB.p);
    const V3<S> cl{clampv(c.x, -he.x, he.x), clampv(c.y, -he.y, he.y), clampv(c.z, -he.z, he.z)};
    const V3<S> dl = cl - c;
    const S distance = length(dl);
    const bool outside = distance > 1e-6f;
    const V3<S> bp = toWorld(cl, tB), sp = tS.p + normal * r;
    const V3<S> w = anchorsReverse((sp + bp) * half, tS, tB, g, gS, gB) * half;
    gn += w * r;
    gS.p += w;
    V3<S> gcl{z, z, z}, gc{z, z, z};
    rotateAdj(tB.q, cl, w, gB.q, gcl);  // bp
    gB.p += w;
    // normal = rotate(qB, nl)
    V3<S> nl, gnl{z, z, z};
    uint32_t region = 6;
    if (outside) {
        nl = dl / distance;
    } else {
        const S d[6] = {he.x - c.x, he.x + c.x, he.y - c.y, he.y + c.y, he.z - c.z, he.z + c.z};
        region = 0;
        S nearest = d[0];
        for (uint32_t k = 1; k < 6; ++k)
            if (d[k] < nearest) {
                nearest = d[k];
                region = k;
            }
        const S s = (region & 1) ? S(1) : -S(1);
        nl = V3<S>{(region >> 1) == 0 ? s : z, (region >> 1) == 1 ? s : z, (region >> 1) == 2 ? s : z};
    }
    rotateAdj(tB.q, nl, gn, gB.q, gnl);
    if (outside) {
        const V3<S> gdl = unitAdj(nl, distance, gnl) - nl * g.depth;  // nl, pen = r - distance
        gcl += gdl;
        gc += -gdl;
    } else {
        // pen = r + he -+ c along the region's axis
        const S s = ((region & 1) ? S(1) : -S(1)) * g.depth;
        gc += V3<S>{(region >> 1) == 0 ? s : z, (region >> 1) == 1 ? s : z, (region >> 1) == 2 ? s : z};
    }
    // clampv passes the derivative strictly by its branches
    if (!(-he.x == he.x) && !(c.x < -he.x) && !(c.x > he.x)) gc.x = gc.x + gcl.x;
    if (!(-he.y == he.y) && !(c.y < -he.y) && !(c.y > he.y)) gc.y = gc.y + gcl.y;
    if (!(-he.z == he.z) && !(c.z < -he.z) && !(c.z > he.z)) gc.z = gc.z + gcl.z;
    V3<S> gw{z, z, z};
    rotateConjAdj(tB.q, tS.p - tB.p, gc, gB.q, gw);
    gS.p += gw;
    gB.p += -gw;
}

// Local corner of the box that boxSupport takes along dir.
template <class S> AD_HD V3<S> supportCorner(const V3<S> &he, const Q<S> &q, const V3<S> &dir) {
    const V3<S> ld = rotate(conj(q), dir);
    return {ld.x >= 0.0f ? he.x : -he.x, ld.y >= 0.0f ? he.y : -he.y, ld.z >= 0.0f ? he.z : -he.z};
}

// A kept face vertex (boxFaceCandidates) of box A (source 0) or B (source 1).
template <class S>
AD_HD void boxFaceReverse(const V3<S> &heA, const Tf<S> &tA, const V3<S> &heB, const Tf<S> &tB, const V3<S> &normal,
                          uint32_t feature, const PointGrad<S> &g, V3<S> &gn, Tf<S> &gA, Tf<S> &gB) {
    const bool fromA = ((feature >> 16) & 1u) == 0;
    const Tf<S> src = fromA ? tA : tB, oth = fromA ? tB : tA;
    const V3<S> srcHe = fromA ? heA : heB, othHe = fromA ? heB : heA;
    const V3<S> dir = fromA ? normal : -normal;
    const uint32_t axis = (feature >> 8) & 3u, vi = feature & 3u;
    const uint32_t fa = axis == 2 ? 0u : axis + 1;
    const S one = S(1), half = S(0.5f);
    // sign of each local coordinate of the vertex
    auto sign = [&](uint32_t k) {
        const bool neg = k == axis ? ((feature >> 4) & 1u) != 0 : k == fa ? (vi & 1u) == 0 : (vi & 2u) == 0;
        return neg ? -one : one;
    };
    const V3<S> lv{sign(0) * srcHe.x, sign(1) * srcHe.y, sign(2) * srcHe.z};
    const V3<S> v = toWorld(lv, src);
    const V3<S> lo = supportCorner(othHe, oth.q, -dir);
    const V3<S> sv = toWorld(lo, oth);
    const S raw = dot(v, dir) - dot(sv, dir);
    const S depth = smax(raw, S(0));
    const V3<S> cand = v - dir * (depth * half);
    const V3<S> gcand = anchorsReverse(cand, tA, tB, g, gA, gB);
    V3<S> gv = gcand, gdir = gcand * (-(depth * half));
    Tf<S> gSrc{{S(0), S(0), S(0)}, {S(0), S(0), S(0), S(0)}}, gOth = gSrc;
    if (!(raw < S(0))) {
        const S gd = g.depth - half * dot(gcand, dir);
        gv += dir * gd;
        gdir += (v - sv) * gd;
        toWorldAdj(lo, oth, dir * -gd, gOth);
    }
    toWorldAdj(lv, src, gv, gSrc);
    gn += fromA ? gdir : -gdir;
    const Tf<S> toA = fromA ? gSrc : gOth, toB = fromA ? gOth : gSrc;
    gA.p += toA.p;
    gB.p += toB.p;
    gA.q = Q<S>{gA.q.x + toA.q.x, gA.q.y + toA.q.y, gA.q.z + toA.q.z, gA.q.w + toA.q.w};
    gB.q = Q<S>{gB.q.x + toB.q.x, gB.q.y + toB.q.y, gB.q.z + toB.q.z, gB.q.w + toB.q.w};
}

// Separating axis `axis` before it is made a unit vector.
template <class S> AD_HD V3<S> boxAxis(const M3<S> &RA, const M3<S> &RB, uint32_t axis) {
    const uint32_t e = axis >= 6 ? axis - 6 : 0u, i = axis < 3 ? axis : e / 3, j = axis < 6 ? axis - 3 : e % 3;
    if (axis < 3) return column(RA, i);
    if (axis < 6) return column(RB, j);
    return cross(column(RA, i), column(RB, j));
}

// r = boxProjectedRadius(he, R, axis)
template <class S>
AD_HD void projectedRadiusAdj(const V3<S> &he, const M3<S> &R, const V3<S> &axis, const S &g, M3<S> &Rb, V3<S> &axisB) {
    for (uint32_t k = 0; k < 3; ++k) {
        const V3<S> a = column(R, k);
        const S h = k == 0 ? he.x : k == 1 ? he.y : he.z;
        const S s = dot(a, axis) < S(0) ? -(h * g) : h * g;
        addColumn(Rb, k, axis * s);
        axisB += a * s;
    }
}

// The one point of two boxes without a kept vertex (boxBox's fallback), and its
// depth, the penetration along the separating axis.
template <class S>
AD_HDN void boxFallbackReverse(const V3<S> &heA, const Tf<S> &tA, const V3<S> &heB, const Tf<S> &tB,
                               const V3<S> &normal, uint32_t axis, const PointGrad<S> &g, V3<S> &gn, Tf<S> &gA,
                               Tf<S> &gB) {
    const S z = S(0), half = S(0.5f);
    const M3<S> RA = toMat3(tA.q), RB = toMat3(tB.q);
    M3<S> bA{z, z, z, z, z, z, z, z, z}, bB = bA;
    const V3<S> cd = tB.p - tA.p;
    const V3<S> tref = sabs(normal.x) < 0.9f ? cst<S>(1.0f, 0.0f, 0.0f) : cst<S>(0.0f, 1.0f, 0.0f);
    const V3<S> c1 = cross(normal, tref);
    const S len = length(c1);
    const V3<S> t1 = normalize(c1), t2 = cross(normal, t1);
    const S nc = (dot(tA.p, normal) + boxProjectedRadius(heA, RA, normal) + dot(tB.p, normal) -
                  boxProjectedRadius(heB, RB, normal)) *
                 half;
    struct Mid {
        S value;
        bool lowerB, upperB;
    };
    auto mid = [&](const V3<S> &ax) {
        const S cA = dot(tA.p, ax), cB = dot(tB.p, ax);
        const S ra = boxProjectedRadius(heA, RA, ax), rb = boxProjectedRadius(heB, RB, ax);
        Mid m;
        m.lowerB = cA - ra < cB - rb;  // smax takes its second operand
        m.upperB = cB + rb < cA + ra;  // smin does
        m.value = ((m.lowerB ? cB - rb : cA - ra) + (m.upperB ? cB + rb : cA + ra)) * half;
        return m;
    };
    auto midAdj = [&](const V3<S> &ax, const Mid &m, const S &gm, V3<S> &axB) {
        const S h = gm * half;
        S ra = z, rb = z;  // adjoints of the two radii
        for (int end = 0; end < 2; ++end) {
            const bool onB = end == 0 ? m.lowerB : m.upperB;
            (onB ? gB : gA).p += ax * h;
            axB += (onB ? tB : tA).p * h;
            S &r = onB ? rb : ra;
            r = end == 0 ? r - h : r + h;
        }
        projectedRadiusAdj(heA, RA, ax, ra, bA, axB);
        projectedRadiusAdj(heB, RB, ax, rb, bB, axB);
    };
    const Mid m1 = mid(t1), m2 = mid(t2);
    const V3<S> point = normal * nc + t1 * m1.value + t2 * m2.value;
    const V3<S> gp = anchorsReverse(point, tA, tB, g, gA, gB);
    V3<S> gt1 = gp * m1.value, gt2 = gp * m2.value;
    midAdj(t1, m1, dot(gp, t1), gt1);
    midAdj(t2, m2, dot(gp, t2), gt2);
    gn += gp * nc;
    const S gnc = dot(gp, normal) * half;
    gn += (tA.p + tB.p) * gnc;
    gA.p += normal * gnc;
    gB.p += normal * gnc;
    projectedRadiusAdj(heA, RA, normal, gnc, bA, gn);
    projectedRadiusAdj(heB, RB, normal, -gnc, bB, gn);
    // t2 = normal x t1, t1 = c1 / |c1|, c1 = normal x tref
    crossAdj(normal, t1, gt2, gn, gt1);
    if (len > 1e-8f) {
        V3<S> trefB{z, z, z};
        crossAdj(normal, tref, unitAdj(t1, len, gt1), gn, trefB);
    }
    // penetration = rA + rB - |cd . u| along the unit axis u = +-normal as it
    // was tested (aligned boxes sit on the kinks of |.|, where the sign counts)
    const bool flipped = dot(boxAxis(RA, RB, axis), normal) < z;
    const V3<S> u = flipped ? -normal : normal;
    V3<S> gu{z, z, z};
    projectedRadiusAdj(heA, RA, u, g.depth, bA, gu);
    projectedRadiusAdj(heB, RB, u, g.depth, bB, gu);
    const S s = dot(cd, u) < z ? g.depth : -g.depth;
    gu += cd * s;
    gB.p += u * s;
    gA.p += u * -s;
    gn += flipped ? -gu : gu;
    toMat3Adj(tA.q, bA, gA.q);
    toMat3Adj(tB.q, bB, gB.q);
}

// Box-box normal: +-unit of the separating axis kept.
template <class S>
AD_HD void boxNormalReverse(const Tf<S> &tA, const Tf<S> &tB, uint32_t axis, const V3<S> &normal, const V3<S> &gn,
                            Tf<S> &gA, Tf<S> &gB) {
    const S z = S(0);
    const M3<S> RA = toMat3(tA.q), RB = toMat3(tB.q);
    M3<S> bA{z, z, z, z, z, z, z, z, z}, bB = bA;
    const uint32_t e = axis >= 6 ? axis - 6 : 0u, i = axis < 3 ? axis : e / 3, j = axis < 6 ? axis - 3 : e % 3;
    const V3<S> raw = boxAxis(RA, RB, axis);
    // the normal is the unit axis or its opposite
    const S len = ssqrt(dot(raw, raw));
    V3<S> graw = unitAdj(normal, len, gn);
    if (dot(raw, normal) < z) graw = -graw;
    if (axis < 3) {
        addColumn(bA, i, graw);
    } else if (axis < 6) {
        addColumn(bB, j, graw);
    } else {
        V3<S> ga{z, z, z}, gb{z, z, z};
        crossAdj(column(RA, i), column(RB, j), graw, ga, gb);
        addColumn(bA, i, ga);
        addColumn(bB, j, gb);
    }
    toMat3Adj(tA.q, bA, gA.q);
    toMat3Adj(tB.q, bB, gB.q);
}

// One point of contactPair's manifold in reverse, with shapes as there.  gn:
// adjoint of the manifold's normal; a one-point manifold of a sphere takes it
// here, the points of two boxes add to it and boxNormalReverse follows them.
template <class S>
AD_HD void contactPointReverse(uint32_t sa, const V3<S> &da, const Tf<S> &tA, uint32_t sb, const V3<S> &db,
                               const Tf<S> &tB, const V3<S> &normal, uint32_t feature, const PointGrad<S> &g,
                               V3<S> &gn, Tf<S> &gA, Tf<S> &gB) {
    if (sa == 0 && sb == 0) {
        sphereSphereReverse(da.x, tA, db.x, tB, normal, g, gn, gA, gB);
    } else if (sa == 0) {
        sphereBoxReverse(da.x, tA, db, tB, normal, g, gn, gA, gB);
    } else if (sb == 0) {
        const PointGrad<S> swapped{g.anchorB, g.anchorA, g.depth};
        sphereBoxReverse(db.x, tB, da, tA, -normal, swapped, -gn, gB, gA);
    } else if ((feature >> 24) == kAdFeatBoxFace) {
        boxFaceReverse(da, tA, db, tB, normal, feature, g, gn, gA, gB);
    } else {
        boxFallbackReverse(da, tA, db, tB, normal, (feature & kAdAxisMask) >> kAdAxisShift, g, gn, gA, gB);
    }
}

// --------------------------------------------------------------- prepare ---
// prepareContactPoints for one point (sequential_impulse_solver.cpp:101-214):
// the constants the velocity iterations use.
template <class S> struct Prepared {
    V3<S> offA, offB, t1, t2;
    S iem, bias, rv, itm00, itm01, itm11;
    V3<S> nrA, nrB, trA1, trB1, trA2, trB2;
    S ntr1, ntr2;
    bool tangentValid;
};
constexpr int kPreparedScalars = 38;

template <class S>
AD_HD void preparePoint(const V3<S> &n, const V3<S> &anchorA, const V3<S> &anchorB, const S &penetration,
                        const Q<S> &qA, const Q<S> &qB, const M3<S> &IA, const M3<S> &IB, const S &imA,
                        const S &imB, const V3<S> &linA, const V3<S> &angA, const V3<S> &linB, const V3<S> &angB,
                        const S &rest, const S &inverseDt, Prepared<S> &o) {
    const S z = ADL(S, 0.0f);
    const V3<S> zv{z, z, z};
    o.offA = rotate(qA, anchorA);
    o.offB = rotate(qB, anchorB);
    o.t1 = o.t2 = o.nrA = o.nrB = o.trA1 = o.trB1 = o.trA2 = o.trB2 = zv;
    o.iem = o.bias = o.rv = o.itm00 = o.itm01 = o.itm11 = o.ntr1 = o.ntr2 = z;
    V3<S> tref = sabs(val(n.x)) < 0.9f ? cst<S>(1.0f, 0.0f, 0.0f) : cst<S>(0.0f, 1.0f, 0.0f);
    V3<S> t1 = cross(n, tref);
    S tl = ssqrt(dot(t1, t1));
    o.tangentValid = val(tl) > 1e-6f;
    if (!o.tangentValid) return;
    t1 = t1 / tl;
    V3<S> t2 = cross(n, t1);
    V3<S> vA = linA + cross(angA, o.offA), vB = linB + cross(angB, o.offB);
    S vin = dot(vB - vA, n);
    V3<S> jA = cross(o.offA, n), jB = cross(o.offB, n);
    V3<S> nrA = mul(IA, jA), nrB = mul(IB, jB);
    S ims = imA + imB;
    S iem = ims + dot(jA, nrA) + dot(jB, nrB);
    V3<S> tjA = cross(o.offA, t1), tjB = cross(o.offB, t1);
    V3<S> trA1 = mul(IA, tjA), trB1 = mul(IB, tjB);
    S tm00 = ims + dot(tjA, trA1) + dot(tjB, trB1);
    S ntr1 = ims * dot(n, t1) + dot(tjA, nrA) + dot(tjB, nrB);
    tjA = cross(o.offA, t2);
    tjB = cross(o.offB, t2);
    V3<S> trA2 = mul(IA, tjA), trB2 = mul(IB, tjB);
    S tm11 = ims + dot(tjA, trA2) + dot(tjB, trB2);
    S ntr2 = ims * dot(n, t2) + dot(tjA, nrA) + dot(tjB, nrB);
    S tm01 = dot(tjA, trA1) + dot(tjB, trB1);
    S det = tm00 * tm11 - tm01 * tm01;
    S itm00 = z, itm01 = z, itm11 = z;
    if (val(det) > 0.0f) {
        S inv = ADL(S, 1.0f) / det;
        itm00 = tm11 * inv;
        itm01 = -tm01 * inv;
        itm11 = tm00 * inv;
    }
    S bias = z, rv = z;
    if (!(val(iem) <= 0.0f)) {
        bias = smax(penetration - ADL(S, 0.005f), z) * (ADL(S, 0.2f) * inverseDt);
        rv = val(vin) < -1.0f ? rest * vin : z;
    }
    o.t1 = t1;
    o.t2 = t2;
    o.iem = iem;
    o.bias = bias;
    o.rv = rv;
    o.itm00 = itm00;
    o.itm01 = itm01;
    o.itm11 = itm11;
    o.nrA = nrA;
    o.nrB = nrB;
    o.trA1 = trA1;
    o.trB1 = trB1;
    o.trA2 = trA2;
    o.trB2 = trB2;
    o.ntr1 = ntr1;
    o.ntr2 = ntr2;
}

// Flat order of the prepared constants (index -> field).
template <class S> AD_HD void preparedPack(const Prepared<S> &o, S *out) {
    const V3<S> *vs[10] = {&o.offA, &o.offB, &o.t1, &o.t2, &o.nrA, &o.nrB, &o.trA1, &o.trB1, &o.trA2, &o.trB2};
    for (int i = 0; i < 10; ++i) {
        out[3 * i] = vs[i]->x;
        out[3 * i + 1] = vs[i]->y;
        out[3 * i + 2] = vs[i]->z;
    }
    out[30] = o.iem;
    out[31] = o.bias;
    out[32] = o.rv;
    out[33] = o.itm00;
    out[34] = o.itm01;
    out[35] = o.itm11;
    out[36] = o.ntr1;
    out[37] = o.ntr2;
}
template <class S> AD_HD V3<S> pv(const S *p, int i) { return {p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
enum : int {
    kPOffA = 0, kPOffB = 1, kPT1 = 2, kPT2 = 3, kPNrA = 4, kPNrB = 5, kPTrA1 = 6, kPTrB1 = 7, kPTrA2 = 8, kPTrB2 = 9,
    kPIem = 30, kPBias = 31, kPRv = 32, kPItm00 = 33, kPItm01 = 34, kPItm11 = 35, kPNtr1 = 36, kPNtr2 = 37
};


// ------------------------------------------------------- reverse: prepare ---
// Inputs of preparePoint that carry an adjoint.
template <class S> struct PrepareGrad {
    V3<S> n, anchorA, anchorB;
    S depth;
    Q<S> qA, qB;
    M3<S> IA, IB;
    S imA, imB;
    V3<S> linA, angA, linB, angB;
    S rest;
};

// Adds to g the adjoints of preparePoint's inputs, given the adjoints ac[] of
// the packed constants c[] it produced (preparedPack's order).
template <class S>
AD_HD void preparePointReverse(const V3<S> &n, const V3<S> &anchorA, const V3<S> &anchorB, const S &penetration,
                               const Q<S> &qA, const Q<S> &qB, const M3<S> &IA, const M3<S> &IB, const S &ims,
                               const V3<S> &linA, const V3<S> &angA, const V3<S> &linB, const V3<S> &angB,
                               const S &rest, const S &inverseDt, const S *c, const S *ac, PrepareGrad<S> &g) {
    const S z = S(0);
    const V3<S> offA = pv(c, kPOffA), offB = pv(c, kPOffB), t1 = pv(c, kPT1), t2 = pv(c, kPT2);
    V3<S> gOffA = pv(ac, kPOffA), gOffB = pv(ac, kPOffB);
    const V3<S> tref = sabs(n.x) < 0.9f ? cst<S>(1.0f, 0.0f, 0.0f) : cst<S>(0.0f, 1.0f, 0.0f);
    const V3<S> c1 = cross(n, tref);
    const S tl = ssqrt(dot(c1, c1));
    if (tl > 1e-6f) {
        const V3<S> nrA = pv(c, kPNrA), nrB = pv(c, kPNrB), trA1 = pv(c, kPTrA1), trB1 = pv(c, kPTrB1),
                    trA2 = pv(c, kPTrA2), trB2 = pv(c, kPTrB2);
        const V3<S> jA = cross(offA, n), jB = cross(offB, n), tjA1 = cross(offA, t1), tjB1 = cross(offB, t1),
                    tjA2 = cross(offA, t2), tjB2 = cross(offB, t2);
        const S tm00 = ims + dot(tjA1, trA1) + dot(tjB1, trB1), tm11 = ims + dot(tjA2, trA2) + dot(tjB2, trB2),
                tm01 = dot(tjA2, trA1) + dot(tjB2, trB1);
        const S det = tm00 * tm11 - tm01 * tm01;
        const V3<S> rel = (linB + cross(angB, offB)) - (linA + cross(angA, offA));
        const S vin = dot(rel, n);
        S gvin = z;
        if (!(c[kPIem] <= z)) {
            if (!(penetration - S(0.005f) < z)) g.depth = g.depth + ac[kPBias] * (S(0.2f) * inverseDt);
            if (vin < -1.0f) {
                g.rest = g.rest + ac[kPRv] * vin;
                gvin = ac[kPRv] * rest;
            }
        }
        S g00 = z, g11 = z, g01 = z;
        if (det > z) {
            const S inv = S(1) / det;
            const S ginv = ac[kPItm00] * tm11 - ac[kPItm01] * tm01 + ac[kPItm11] * tm00;
            const S gdet = -(ginv * inv) * inv;
            g00 = ac[kPItm11] * inv + gdet * tm11;
            g11 = ac[kPItm00] * inv + gdet * tm00;
            g01 = -(ac[kPItm01] * inv) - (gdet + gdet) * tm01;
        }
        const S giem = ac[kPIem], gn1 = ac[kPNtr1], gn2 = ac[kPNtr2];
        const S gims = giem + g00 + g11 + gn1 * dot(n, t1) + gn2 * dot(n, t2);
        g.imA = g.imA + gims;
        g.imB = g.imB + gims;
        V3<S> gt1 = pv(ac, kPT1) + n * (gn1 * ims), gt2 = pv(ac, kPT2) + n * (gn2 * ims);
        V3<S> gn = t1 * (gn1 * ims) + t2 * (gn2 * ims) + rel * gvin;
        // one body's rows: j = off x n, nr = I j, tj = off x t, tr = I tj
        auto side = [&](const V3<S> &off, const M3<S> &I, const V3<S> &j, const V3<S> &tj1, const V3<S> &tj2,
                        const V3<S> &nr, const V3<S> &tr1, const V3<S> &tr2, const V3<S> &acNr, const V3<S> &acTr1,
                        const V3<S> &acTr2, V3<S> &gOff, M3<S> &gI) {
            V3<S> gj = nr * giem, gtj1 = tr1 * g00 + nr * gn1, gtj2 = tr2 * g11 + nr * gn2 + tr1 * g01;
            mulAdj(I, j, acNr + j * giem + tj1 * gn1 + tj2 * gn2, gI, gj);
            mulAdj(I, tj1, acTr1 + tj1 * g00 + tj2 * g01, gI, gtj1);
            mulAdj(I, tj2, acTr2 + tj2 * g11, gI, gtj2);
            crossAdj(off, n, gj, gOff, gn);
            crossAdj(off, t1, gtj1, gOff, gt1);
            crossAdj(off, t2, gtj2, gOff, gt2);
        };
        side(offA, IA, jA, tjA1, tjA2, nrA, trA1, trA2, pv(ac, kPNrA), pv(ac, kPTrA1), pv(ac, kPTrA2), gOffA, g.IA);
        side(offB, IB, jB, tjB1, tjB2, nrB, trB1, trB2, pv(ac, kPNrB), pv(ac, kPTrB1), pv(ac, kPTrB2), gOffB, g.IB);
        // vin = n . (linB + angB x offB - linA - angA x offA)
        const V3<S> gv = n * gvin;
        g.linB += gv;
        g.linA += -gv;
        crossAdj(angB, offB, gv, g.angB, gOffB);
        crossAdj(angA, offA, -gv, g.angA, gOffA);
        // t2 = n x t1, t1 = c1 / tl, c1 = n x tref
        crossAdj(n, t1, gt2, gn, gt1);
        V3<S> trefB{z, z, z};
        crossAdj(n, tref, unitAdj(t1, tl, gt1), gn, trefB);
        g.n += gn;
    }
    rotateAdj(qA, anchorA, gOffA, g.qA, g.anchorA);
    rotateAdj(qB, anchorB, gOffB, g.qB, g.anchorB);
}

} // namespace ad
} // namespace pe
