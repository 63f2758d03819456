// The FP32 forms of the term energies and gradients (mmff_terms.cuh) with every rounding step
// written out.
//
// The optimizer's accept / reject tests compare energies of neighbouring points, so a
// conformer's whole run follows from the last bit of each term.  Left to the compiler, whether a
// product is fused with the sum it enters depends on the code around it: the same source line
// gave other bits in an energy-only evaluation than in one with gradients, and in one kernel
// instance than in another.  Here each product, sum and fused step is explicit, so a term's energy
// is the same number whichever evaluation it comes from (a trial's energy may come with or without
// its gradient), and code around the terms can change without changing results.  (A conformer's
// energy is the same number where its terms are also summed in the same order: see eval_terms32.)
//
// Conventions: a b + c d + e f is fma(e, f, fma(a, b, c d)) and a b - c d is fma(a, b, -(c d)).
#pragma once
#include "mmff_terms.cuh"

namespace mmffb {
namespace t32 {

#define M_(a, b) __fmul_rn(a, b)
#define A_(a, b) __fadd_rn(a, b)
#define F_(a, b, c) __fmaf_rn(a, b, c)

// 1 / x and 1 / sqrt(x) of the hardware, for normal x: the bits of __fdividef(1, x) and
// rsqrtf(x) without their steps for denormals (no argument below is one: each is bounded below
// by 1e-30 or is a sum with a constant).
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsq(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct V3 {
    float x, y, z;
};

__device__ __forceinline__ V3 at(const float *p4, int a) {
    const float4 v = reinterpret_cast<const float4 *>(p4)[a];
    return V3{v.x, v.y, v.z};
}
__device__ __forceinline__ V3 sub(const V3 &a, const V3 &b) {
    return V3{A_(a.x, -b.x), A_(a.y, -b.y), A_(a.z, -b.z)};
}
__device__ __forceinline__ V3 neg(const V3 &a) { return V3{-a.x, -a.y, -a.z}; }
__device__ __forceinline__ V3 mul(float s, const V3 &a) { return V3{M_(s, a.x), M_(s, a.y), M_(s, a.z)}; }
// a - c b
__device__ __forceinline__ V3 subm(const V3 &a, float c, const V3 &b) {
    return V3{F_(-c, b.x, a.x), F_(-c, b.y, a.y), F_(-c, b.z, a.z)};
}
__device__ __forceinline__ float dot(const V3 &a, const V3 &b) { return F_(a.z, b.z, F_(a.x, b.x, M_(a.y, b.y))); }
__device__ __forceinline__ float rinv(const V3 &a) { return rsq(fmaxf(dot(a, a), 1e-16f)); }
__device__ __forceinline__ float clamp1(float c) { return c < -1.0f ? -1.0f : (c > 1.0f ? 1.0f : c); }
__device__ __forceinline__ V3 cross(const V3 &a, const V3 &b) {
    return V3{F_(a.y, b.z, -M_(a.z, b.y)), F_(a.z, b.x, -M_(a.x, b.z)), F_(a.x, b.y, -M_(a.y, b.x))};
}
// (-a) x b: the two products change places
__device__ __forceinline__ V3 cross_neg(const V3 &a, const V3 &b) {
    return V3{F_(a.z, b.y, -M_(a.y, b.z)), F_(a.x, b.z, -M_(a.z, b.x)), F_(a.y, b.x, -M_(a.x, b.y))};
}

// The run's term constants in FP32, formed once per conformer.
struct Mode {
    float cb, cb15, kang, kang_deg, ksbg;
    bool lin;
    __device__ explicit Mode(const TermMode &md)
        : cb((float)md.cb), cb15(1.5f * (float)md.cb), kang((float)md.kang),
          kang_deg((float)md.kang * (float)MMFF_RAD2DEG), ksbg((float)md.ksbg), lin(md.lin != 0) {}
};

// dst += v
__device__ __forceinline__ void acc(float *dst, const V3 &v) {
    dst[0] = A_(dst[0], v.x); dst[1] = A_(dst[1], v.y); dst[2] = A_(dst[2], v.z);
}
// dst -= v
__device__ __forceinline__ void dec(float *dst, const V3 &v) {
    dst[0] = A_(dst[0], -v.x); dst[1] = A_(dst[1], -v.y); dst[2] = A_(dst[2], -v.z);
}
// dst += s v, fused
__device__ __forceinline__ void accm(float *dst, float s, const V3 &v) {
    dst[0] = F_(s, v.x, dst[0]); dst[1] = F_(s, v.y, dst[1]); dst[2] = F_(s, v.z, dst[2]);
}

// Three steps of the gradient have two forms.  A run's first gradient has always been rounded
// with the product set apart in them (the stretch-bend's only in the 128-register L-BFGS instance
// with its history in shared memory), the later ones and every other caller's with it fused; both are
// kept, so that runs keep their results bit for bit.  A run's first gradient therefore differs from
// an energy_grad call's at the same point in its last bits.
enum Forms { kFused = 0, kBondApart = 1, kTorsionApart = 2, kStrbendApart = 4 };

// 1 - c^2
__device__ __forceinline__ float one_minus_sq(float c, bool apart) {
    return apart ? A_(1.0f, -M_(c, c)) : F_(-c, c, 1.0f);
}

// ---- bond stretch: gradient +f on a, -f on b ----
template <bool G>
__device__ __forceinline__ float bond(const V3 &a, const V3 &b, float kb, float r0, bool apart, V3 &f) {
    const V3 r = sub(a, b);
    const float x2 = fmaxf(dot(r, r), 1e-16f), rs = rsq(x2);
    const float de = F_(x2, rs, -r0);
    const float ce = F_(M_(7.0f / 3.0f, de), de, F_(-2.0f, de, 1.0f));
    if (G) {
        const float d = M_(x2, rs), dr = apart ? A_(d, -r0) : de;
        const float inv = d > 1e-8f ? rcp(d) : 0.0f;
        const float cg = F_(M_(14.0f / 3.0f, dr), dr, F_(-3.0f, dr, 1.0f));
        f = mul(M_(M_(M_(M_((float)MMFF_MDYNE, kb), dr), cg), inv), r);
    }
    return M_(M_(M_(M_((float)(0.5 * MMFF_MDYNE), kb), de), de), ce);
}

// ---- angle bend: gradient s0 f0 on i, -f1 on j, f2 on k ----
template <bool G>
__device__ __forceinline__ float angle(const V3 &pi, const V3 &pj, const V3 &pk, float ka, float t0, bool linear,
                                       const Mode &md, float &s0, V3 &f0, V3 &f1, V3 &f2) {
    const V3 r1 = sub(pi, pj), r2 = sub(pk, pj);
    const float id1 = rinv(r1), id2 = rinv(r2);
    const float c = clamp1(M_(M_(dot(r1, r2), id1), id2));
    linear = linear && md.lin;
    const float dt = F_((float)MMFF_RAD2DEG, acosf(c), -t0);
    if (G) {
        const float sn2 = F_(-c, c, 1.0f);
        float cf = 0.0f;
        if (sn2 >= 1e-16f) {
            const float rs = rsq(fmaxf(sn2, 1e-16f)), sm = fmaxf(sn2, 0.0f);
            const float de = linear ? M_(M_(-(float)MMFF_MDYNE, ka), M_(sm, rsq(sm)))
                                    : M_(M_(M_(md.kang_deg, ka), dt), F_(md.cb15, dt, 1.0f));
            cf = M_(-de, rs);
        }
        const V3 u1 = mul(id1, r1), u2 = mul(id2, r2);
        s0 = M_(cf, id1);
        f0 = subm(u2, c, u1);
        f2 = mul(M_(cf, id2), subm(u1, c, u2));
        f1 = V3{F_(s0, f0.x, f2.x), F_(s0, f0.y, f2.y), F_(s0, f0.z, f2.z)};
    }
    return linear ? M_(M_((float)MMFF_MDYNE, ka), A_(1.0f, c))
                  : M_(M_(M_(M_(M_(0.5f, md.kang), ka), dt), dt), F_(md.cb, dt, 1.0f));
}

// ---- stretch-bend: gradients f0, f1, f2 on i, j, k ----
template <bool G>
__device__ __forceinline__ float strbend(const V3 &pi, const V3 &pj, const V3 &pk, float r0ij, float r0kj, float t0,
                                         float kij, float kkj, const Mode &md, bool apart, V3 &f0, V3 &f1,
                                         V3 &f2) {
    const V3 r1 = sub(pi, pj), r2 = sub(pk, pj);
    const float id1 = rinv(r1), id2 = rinv(r2);
    const float c = clamp1(M_(M_(dot(r1, r2), id1), id2));
    const float d1 = rcp(fmaxf(id1, 1e-8f)), d2 = rcp(fmaxf(id2, 1e-8f));
    const float dt = F_((float)MMFF_RAD2DEG, acosf(c), -t0);
    const float dr1 = A_(d1, -r0ij), dr2 = A_(d2, -r0kj);
    const float ks = F_(dr1, kij, M_(dr2, kkj));
    if (G) {
        const float sn2 = one_minus_sq(c, apart);
        f0 = f1 = f2 = V3{0.0f, 0.0f, 0.0f};
        if (sn2 >= 1e-16f) {
            const float is = fminf(rsq(fmaxf(sn2, 1e-16f)), 1e8f), pf = md.ksbg;
            const float beis = M_(M_((float)MMFF_RAD2DEG, ks), is);
            const V3 u1 = mul(id1, r1), u2 = mul(id2, r2);
            const V3 i1 = mul(id1, subm(u2, c, u1)), i3 = mul(id2, subm(u1, c, u2));
            auto comp = [&](float a1, float a2, float b1, float b3, float &g0, float &g1, float &g2) {
                g0 = M_(pf, F_(M_(dt, a1), kij, -M_(b1, beis)));
                g2 = M_(pf, F_(M_(dt, a2), kkj, -M_(b3, beis)));
                g1 = M_(pf, F_(A_(b1, b3), beis, M_(-dt, F_(a1, kij, M_(a2, kkj)))));
            };
            comp(u1.x, u2.x, i1.x, i3.x, f0.x, f1.x, f2.x);
            comp(u1.y, u2.y, i1.y, i3.y, f0.y, f1.y, f2.y);
            comp(u1.z, u2.z, i1.z, i3.z, f0.z, f1.z, f2.z);
        }
    }
    return M_(M_(2.51210f, dt), ks);
}

// ---- Wilson out-of-plane: gradient s0 f0 on i, -f1 on j, f2 on k, f3 on l ----
template <bool G>
__device__ __forceinline__ float oop(const V3 &pi, const V3 &pj, const V3 &pk, const V3 &pl, float koop,
                                     const Mode &md, float &s0, V3 &f0, V3 &f1, V3 &f2, V3 &f3) {
    const V3 rI = sub(pi, pj), rK = sub(pk, pj), rL = sub(pl, pj);
    const float iI = rinv(rI), iK = rinv(rK), iL = rinv(rL);
    const V3 uI = mul(iI, rI), uK = mul(iK, rK), uL = mul(iL, rL);
    const V3 nv = cross_neg(uI, uK);
    const float s = clamp1(M_(dot(uL, nv), rinv(nv)));
    const float chi = M_((float)MMFF_RAD2DEG, asinf(s));
    if (G) {
        const float c2 = F_(-s, s, 1.0f);
        const float ic = c2 > 0.0f ? rsq(fmaxf(c2, 1e-16f)) : 1e8f;
        const float ct = clamp1(dot(uI, uK));
        const float ist = rsq(fmaxf(F_(-ct, ct, 1.0f), 1e-8f));
        const float dE = M_(M_(md.kang_deg, koop), chi);
        const float t1 = M_(ic, ist), t2 = M_(M_(M_(s, ic), ist), ist);
        const V3 a1 = cross(uL, uK), a2 = cross(uI, uL), a3 = cross(uK, uI);
        const V3 w1 = subm(uI, ct, uK), w3 = subm(uK, ct, uI);
        s0 = iI;
        f0 = V3{M_(dE, F_(a1.x, t1, -M_(w1.x, t2))), M_(dE, F_(a1.y, t1, -M_(w1.y, t2))),
                M_(dE, F_(a1.z, t1, -M_(w1.z, t2)))};
        f2 = mul(iK, V3{M_(dE, F_(a2.x, t1, -M_(w3.x, t2))), M_(dE, F_(a2.y, t1, -M_(w3.y, t2))),
                        M_(dE, F_(a2.z, t1, -M_(w3.z, t2)))});
        f3 = mul(iL, V3{M_(dE, F_(a3.x, t1, -M_(M_(uL.x, s), ic))), M_(dE, F_(a3.y, t1, -M_(M_(uL.y, s), ic))),
                        M_(dE, F_(a3.z, t1, -M_(M_(uL.z, s), ic)))});
        f1 = V3{A_(F_(f0.x, iI, f2.x), f3.x), A_(F_(f0.y, iI, f2.y), f3.y), A_(F_(f0.z, iI, f2.z), f3.z)};
    }
    return M_(M_(M_(M_(0.5f, md.kang), koop), chi), chi);
}

// ---- torsion: gradients f0 .. f3 on its four atoms ----
template <bool G>
__device__ __forceinline__ float torsion(const V3 &p1, const V3 &p2, const V3 &p3, const V3 &p4, float V1, float V2,
                                         float V3_, bool apart, V3 &f0, V3 &f1, V3 &f2, V3 &f3) {
    const V3 a = sub(p1, p2), b = sub(p3, p2), c = sub(p4, p3);
    const V3 c1 = cross(a, b), c2 = cross_neg(b, c);
    const float n1 = dot(c1, c1), n2 = dot(c2, c2), comb = M_(n1, n2);
    float e = 0.0f;
    if (comb >= 1e-16f) {
        const float cp = clamp1(M_(dot(c1, c2), rsq(comb)));
        const float cos2 = F_(M_(2.0f, cp), cp, -1.0f), cos31 = F_(cp, F_(M_(4.0f, cp), cp, -3.0f), 1.0f);
        e = M_(0.5f, F_(V3_, cos31, F_(V1, A_(1.0f, cp), M_(V2, A_(1.0f, -cos2)))));
    }
    if (G) {
        f0 = f1 = f2 = f3 = V3{0.0f, 0.0f, 0.0f};
        if (n1 >= 1e-30f && n2 >= 1e-30f) {
            const float i1 = fminf(rsq(n1), 1e5f), i2 = fminf(rsq(n2), 1e5f);
            const V3 u1 = mul(i1, c1), u2 = mul(i2, c2);
            const float cp = clamp1(dot(u1, u2));
            const float sp2 = one_minus_sq(cp, apart);
            float st = 0.0f;
            if (sp2 > 0.0f)
                st = M_(0.5f, F_(M_(3.0f, V3_), F_(-4.0f, sp2, 3.0f), F_(-M_(2.0f, V2), M_(2.0f, cp), V1)));
            const V3 d = mul(i1, subm(u2, cp, u1)), g = mul(i2, subm(u1, cp, u2));
            auto four = [](float p, float q, float r, float s, float t, float u, float v, float w) {
                return F_(v, w, F_(t, u, F_(p, q, M_(r, s))));
            };
            f0 = mul(st, V3{F_(d.z, b.y, -M_(d.y, b.z)), F_(d.x, b.z, -M_(d.z, b.x)), F_(d.y, b.x, -M_(d.x, b.y))});
            f3 = mul(st, V3{F_(g.z, b.y, -M_(g.y, b.z)), F_(g.x, b.z, -M_(g.z, b.x)), F_(g.y, b.x, -M_(g.x, b.y))});
            f1 = mul(st, V3{four(d.y, A_(b.z, -a.z), d.z, A_(a.y, -b.y), g.y, -c.z, g.z, c.y),
                            four(d.x, A_(a.z, -b.z), d.z, A_(b.x, -a.x), g.x, c.z, g.z, -c.x),
                            four(d.x, A_(b.y, -a.y), d.y, A_(a.x, -b.x), g.x, -c.y, g.y, c.x)});
            f2 = mul(st, V3{four(d.y, a.z, -d.z, a.y, g.y, A_(c.z, b.z), g.z, A_(-c.y, -b.y)),
                            four(d.z, a.x, -d.x, a.z, g.x, A_(-c.z, -b.z), g.z, A_(c.x, b.x)),
                            four(d.x, a.y, -d.y, a.x, g.x, A_(c.y, b.y), g.y, A_(-c.x, -b.x))});
        }
    }
    return e;
}

// ---- buffered 14-7 vdW and Coulomb of one pair; iR = 1 / R*; s: grad_i = s (p_i - p_j) ----
// DD: distance-dependent dielectric
template <bool G, bool DD>
__device__ __forceinline__ void pair(float dx, float dy, float dz, float iR, float eps, float qq, float &e_vdw,
                                     float &e_ele, float &s) {
    const float x2 = fmaxf(F_(dz, dz, F_(dx, dx, M_(dy, dy))), 1e-16f);
    const float rd = rsq(x2), d = M_(x2, rd);
    const float q = M_(d, iR), q2 = M_(q, q), q6 = M_(M_(q2, q2), q2);
    const float ib = rcp(A_(q, 0.07f));
    const float t = M_(1.07f, ib), t2 = M_(t, t), t7 = M_(M_(M_(t2, t2), t2), t);
    const float iq = rcp(F_(q6, q, 0.12f));
    e_vdw = M_(M_(eps, t7), F_(1.12f, iq, -2.0f));
    const float idp = rcp(A_(d, 0.05f));
    const float cq = M_((float)MMFF_ELEC, qq);
    e_ele = DD ? M_(M_(cq, idp), idp) : M_(cq, idp);
    if (G) {
        const float inv = d > 1e-8f ? rd : 0.0f;
        const float br = F_(F_(-7.84f, iq, 14.0f), ib, M_(M_(M_(-7.84f, q6), iq), iq));
        const float de = DD ? M_(M_(M_(M_(-2.0f, cq), idp), idp), idp) : M_(M_(-cq, idp), idp);
        s = M_(F_(M_(M_(eps, iR), t7), br, de), inv);
    }
}

#undef M_
#undef A_
#undef F_

}  // namespace t32
}  // namespace mmffb
