// Scalar-generic math for the differentiable rollout.  The same formulas as the
// engine's float math (pe_math.cuh), written over a scalar type S so that one
// source serves float (GPU) and double (the FP64 CPU adjoint), and the reverse
// of the pieces that the adjoint runs through.  With S = float the operations
// of the forward functions, their order and their constants are the engine's,
// so values are bit-identical.  Compiles as CUDA and as plain C++.
#pragma once
#include <cmath>
#include <cstdint>

#if defined(__CUDACC__)
#define AD_HD __host__ __device__ __forceinline__
// Large routines are compiled once and called, which keeps the kernels' code
// size and compile time down.
#define AD_HDN __host__ __device__ __noinline__
#else
#define AD_HD inline
#define AD_HDN inline
#endif

namespace pe {
namespace ad {

AD_HD float ssqrt(float v) { return sqrtf(v); }
AD_HD double ssqrt(double v) { return sqrt(v); }
AD_HD float sabs(float v) { return fabsf(v); }
AD_HD double sabs(double v) { return fabs(v); }

AD_HD float val(float v) { return v; }
AD_HD double val(double v) { return v; }

// Scalar S built from a constant of its value type (float constants first
// rounded to float, as the reference writes them).
template <class S> struct Lit {
    template <class C> AD_HD static S make(C c) { return S(c); }
};
#define ADL(S, c) ::pe::ad::Lit<S>::make(c)

// std::max / std::min argument semantics (first operand on ties / NaN).
template <class S> AD_HD S smax(const S &a, const S &b) { return (val(a) < val(b)) ? b : a; }
template <class S> AD_HD S smin(const S &a, const S &b) { return (val(b) < val(a)) ? b : a; }

// ------------------------------------------------------------------ vectors --
template <class S> struct V3 {
    S x, y, z;
};
template <class S> AD_HD V3<S> operator+(const V3<S> &a, const V3<S> &b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <class S> AD_HD V3<S> operator-(const V3<S> &a, const V3<S> &b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <class S> AD_HD V3<S> operator-(const V3<S> &a) { return {-a.x, -a.y, -a.z}; }
template <class S> AD_HD V3<S> operator*(const V3<S> &a, const S &s) { return {a.x * s, a.y * s, a.z * s}; }
template <class S> AD_HD V3<S> operator/(const V3<S> &a, const S &s) { return {a.x / s, a.y / s, a.z / s}; }
template <class S> AD_HD V3<S> &operator+=(V3<S> &a, const V3<S> &b) {
    a.x = a.x + b.x;
    a.y = a.y + b.y;
    a.z = a.z + b.z;
    return a;
}
template <class S> AD_HD S dot(const V3<S> &a, const V3<S> &b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <class S> AD_HD V3<S> cross(const V3<S> &a, const V3<S> &b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <class S> AD_HD S length(const V3<S> &v) { return ssqrt(v.x * v.x + v.y * v.y + v.z * v.z); }
template <class S> AD_HD V3<S> normalize(const V3<S> &v) {
    S len = length(v);
    if (val(len) <= 1e-8f) return {ADL(S, 0.0f), ADL(S, 0.0f), ADL(S, 0.0f)};
    return v * (ADL(S, 1.0f) / len);
}
template <class S> AD_HD S clampv(const S &v, const S &lo, const S &hi) {
    if (val(lo) == val(hi)) return lo;
    if (val(v) < val(lo)) return lo;
    if (val(v) > val(hi)) return hi;
    return v;
}

template <class S> struct Q {
    S x, y, z, w;
};
template <class S> AD_HD Q<S> qidentity() { return {ADL(S, 0.0f), ADL(S, 0.0f), ADL(S, 0.0f), ADL(S, 1.0f)}; }
template <class S> AD_HD Q<S> qmul(const Q<S> &a, const Q<S> &o) {
    return {a.w * o.x + a.x * o.w + a.y * o.z - a.z * o.y, a.w * o.y - a.x * o.z + a.y * o.w + a.z * o.x,
            a.w * o.z + a.x * o.y - a.y * o.x + a.z * o.w, a.w * o.w - a.x * o.x - a.y * o.y - a.z * o.z};
}
template <class S> AD_HD Q<S> conj(const Q<S> &q) { return {-q.x, -q.y, -q.z, q.w}; }
template <class S> AD_HD Q<S> qnormalized(const Q<S> &q) {
    S len = ssqrt(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
    if (val(len) == 0.0f) return qidentity<S>();
    return {q.x / len, q.y / len, q.z / len, q.w / len};
}
template <class S> AD_HD V3<S> rotate(const Q<S> &q, const V3<S> &v) {
    Q<S> p{v.x, v.y, v.z, ADL(S, 0.0f)};
    Q<S> r = qmul(qmul(q, p), conj(q));
    return {r.x, r.y, r.z};
}

template <class S> struct M3 {
    S m00, m01, m02, m10, m11, m12, m20, m21, m22;
};
template <class S> AD_HD M3<S> toMat3(const Q<S> &q) {
    S xx = q.x * q.x, yy = q.y * q.y, zz = q.z * q.z;
    S xy = q.x * q.y, xz = q.x * q.z, yz = q.y * q.z;
    S wx = q.w * q.x, wy = q.w * q.y, wz = q.w * q.z;
    const S one = ADL(S, 1.0f), two = ADL(S, 2.0f);
    return {one - two * (yy + zz), two * (xy - wz), two * (xz + wy),
            two * (xy + wz),       one - two * (xx + zz), two * (yz - wx),
            two * (xz - wy),       two * (yz + wx),       one - two * (xx + yy)};
}
template <class S> AD_HD V3<S> mul(const M3<S> &m, const V3<S> &v) {
    return {m.m00 * v.x + m.m01 * v.y + m.m02 * v.z, m.m10 * v.x + m.m11 * v.y + m.m12 * v.z,
            m.m20 * v.x + m.m21 * v.y + m.m22 * v.z};
}
template <class S> AD_HD M3<S> mul(const M3<S> &l, const M3<S> &r) {
    return {l.m00 * r.m00 + l.m01 * r.m10 + l.m02 * r.m20, l.m00 * r.m01 + l.m01 * r.m11 + l.m02 * r.m21,
            l.m00 * r.m02 + l.m01 * r.m12 + l.m02 * r.m22, l.m10 * r.m00 + l.m11 * r.m10 + l.m12 * r.m20,
            l.m10 * r.m01 + l.m11 * r.m11 + l.m12 * r.m21, l.m10 * r.m02 + l.m11 * r.m12 + l.m12 * r.m22,
            l.m20 * r.m00 + l.m21 * r.m10 + l.m22 * r.m20, l.m20 * r.m01 + l.m21 * r.m11 + l.m22 * r.m21,
            l.m20 * r.m02 + l.m21 * r.m12 + l.m22 * r.m22};
}
template <class S> AD_HD M3<S> transpose(const M3<S> &v) {
    return {v.m00, v.m10, v.m20, v.m01, v.m11, v.m21, v.m02, v.m12, v.m22};
}
// (R * I_local) * R^T with the diagonal local inverse inertia
// (include/phys/dynamics/rigid_body.hpp:97-101).
template <class S> AD_HD M3<S> inverseInertiaWorld(const Q<S> &q, const S &ixx, const S &iyy, const S &izz) {
    M3<S> R = toMat3(q);
    const S z = ADL(S, 0.0f);
    M3<S> I{ixx, z, z, z, iyy, z, z, z, izz};
    return mul(mul(R, I), transpose(R));
}

template <class S> struct Tf {
    V3<S> p;
    Q<S> q;
};
template <class S> AD_HD V3<S> toLocal(const V3<S> &w, const Tf<S> &t) { return rotate(conj(t.q), w - t.p); }
template <class S> AD_HD V3<S> toWorld(const V3<S> &l, const Tf<S> &t) { return t.p + rotate(t.q, l); }

// Plain-scalar reverse helpers.
// c = a x b: abar += b x cbar, bbar += cbar x a.
template <class S> AD_HD void crossAdj(const V3<S> &a, const V3<S> &b, const V3<S> &cbar, V3<S> &abar, V3<S> &bbar) {
    abar += cross(b, cbar);
    bbar += cross(cbar, a);
}
// r = qmul(a, o): adjoints of a and o.
template <class S> AD_HD void qmulAdj(const Q<S> &a, const Q<S> &o, const Q<S> &r, Q<S> &ab, Q<S> &ob) {
    ab.x = ab.x + (r.x * o.w - r.y * o.z + r.z * o.y - r.w * o.x);
    ab.y = ab.y + (r.x * o.z + r.y * o.w - r.z * o.x - r.w * o.y);
    ab.z = ab.z + (-r.x * o.y + r.y * o.x + r.z * o.w - r.w * o.z);
    ab.w = ab.w + (r.x * o.x + r.y * o.y + r.z * o.z + r.w * o.w);
    ob.x = ob.x + (r.x * a.w + r.y * a.z - r.z * a.y - r.w * a.x);
    ob.y = ob.y + (-r.x * a.z + r.y * a.w + r.z * a.x - r.w * a.y);
    ob.z = ob.z + (r.x * a.y - r.y * a.x + r.z * a.w - r.w * a.z);
    ob.w = ob.w + (r.x * a.x + r.y * a.y + r.z * a.z + r.w * a.w);
}

// r = rotate(q, v): for any q the product q v q* is
// (w^2 - u.u) v + 2 (u.v) u + 2 w (u x v), so with the adjoint g of r
template <class S> AD_HD void rotateAdj(const Q<S> &q, const V3<S> &v, const V3<S> &g, Q<S> &qb, V3<S> &vb) {
    const V3<S> u{q.x, q.y, q.z};
    const S two = S(2), ug = dot(u, g), uv = dot(u, v), vg = dot(v, g), ww = q.w * q.w - dot(u, u);
    const V3<S> vxg = cross(v, g), gxu = cross(g, u);
    vb += g * ww + u * (two * ug) + gxu * (two * q.w);
    qb.x = qb.x + two * (ug * v.x + uv * g.x - vg * u.x + q.w * vxg.x);
    qb.y = qb.y + two * (ug * v.y + uv * g.y - vg * u.y + q.w * vxg.y);
    qb.z = qb.z + two * (ug * v.z + uv * g.z - vg * u.z + q.w * vxg.z);
    qb.w = qb.w + two * (q.w * vg + dot(u, vxg));
}
// r = rotate(conj(q), v).
template <class S> AD_HD void rotateConjAdj(const Q<S> &q, const V3<S> &v, const V3<S> &g, Q<S> &qb, V3<S> &vb) {
    Q<S> cb{S(0), S(0), S(0), S(0)};
    rotateAdj(conj(q), v, g, cb, vb);
    qb.x = qb.x - cb.x;
    qb.y = qb.y - cb.y;
    qb.z = qb.z - cb.z;
    qb.w = qb.w + cb.w;
}
// l = toLocal(w, t), w = toWorld(l, t).
template <class S> AD_HD void toLocalAdj(const V3<S> &w, const Tf<S> &t, const V3<S> &g, Tf<S> &tb, V3<S> &wb) {
    V3<S> d{S(0), S(0), S(0)};
    rotateConjAdj(t.q, w - t.p, g, tb.q, d);
    wb += d;
    tb.p += -d;
}
template <class S> AD_HD void toWorldAdj(const V3<S> &l, const Tf<S> &t, const V3<S> &g, Tf<S> &tb) {
    V3<S> lb{S(0), S(0), S(0)};
    rotateAdj(t.q, l, g, tb.q, lb);
    tb.p += g;
}
// m = toMat3(q).
template <class S> AD_HD void toMat3Adj(const Q<S> &q, const M3<S> &b, Q<S> &qb) {
    const S two = S(2), four = S(4);
    const S p01 = b.m01 + b.m10, p02 = b.m02 + b.m20, p12 = b.m12 + b.m21;
    const S d01 = b.m10 - b.m01, d02 = b.m02 - b.m20, d12 = b.m21 - b.m12;
    qb.x = qb.x + two * (q.y * p01 + q.z * p02 + q.w * d12) - four * q.x * (b.m11 + b.m22);
    qb.y = qb.y + two * (q.x * p01 + q.z * p12 + q.w * d02) - four * q.y * (b.m00 + b.m22);
    qb.z = qb.z + two * (q.x * p02 + q.y * p12 + q.w * d01) - four * q.z * (b.m00 + b.m11);
    qb.w = qb.w + two * (q.z * d01 + q.y * d02 + q.x * d12);
}
// r = mul(m, v): adjoint of m (outer product) and of v.
template <class S> AD_HD void mulAdj(const M3<S> &m, const V3<S> &v, const V3<S> &g, M3<S> &mb, V3<S> &vb) {
    mb.m00 = mb.m00 + g.x * v.x;
    mb.m01 = mb.m01 + g.x * v.y;
    mb.m02 = mb.m02 + g.x * v.z;
    mb.m10 = mb.m10 + g.y * v.x;
    mb.m11 = mb.m11 + g.y * v.y;
    mb.m12 = mb.m12 + g.y * v.z;
    mb.m20 = mb.m20 + g.z * v.x;
    mb.m21 = mb.m21 + g.z * v.y;
    mb.m22 = mb.m22 + g.z * v.z;
    vb += mul(transpose(m), g);
}
// I = inverseInertiaWorld(q, d) = R diag(d) R^T: the adjoint of R's column k is
// d_k (Ib + Ib^T) R_k.
template <class S> AD_HD void inverseInertiaAdj(const Q<S> &q, const V3<S> &d, const M3<S> &b, Q<S> &qb) {
    const M3<S> R = toMat3(q);
    const M3<S> s{b.m00 + b.m00, b.m01 + b.m10, b.m02 + b.m20, b.m10 + b.m01, b.m11 + b.m11,
                  b.m12 + b.m21, b.m20 + b.m02, b.m21 + b.m12, b.m22 + b.m22};
    const S z = S(0);
    toMat3Adj(q, mul(mul(s, R), M3<S>{d.x, z, z, z, d.y, z, z, z, d.z}), qb);
}

} // namespace ad
} // namespace pe
