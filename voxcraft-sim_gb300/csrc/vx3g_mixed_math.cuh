// vx3g_mixed_math.cuh -- the arithmetic of the mixed-precision step, with every rounding spelled
// out: products and sums that the compiler must not contract are __fmul_rn / __fadd_rn /
// __fsub_rn, the contracted ones are fmaf.  A step then has the same bits in whichever kernel it
// is inlined (one pass per launch, or many steps per launch).
//
// The link part restates VX3_Link::orientLink/updateForces (src/VX3/VX3_Link.cu:90-218), the
// voxel part VX3_Voxel::timeStep (src/VX3/VX3_Voxel.cu:162-277), without the cancellations FP32
// would suffer (see vx3g_mixed.cu).
#pragma once

#include <math_constants.h>

#include "vx3g_step.cuh"

namespace vx3g {
namespace mx {

using V = V3<float>;
using Q = Q4<float>;

__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float plus(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float minus(float a, float b) { return __fsub_rn(a, b); }
// a*b + c*d with the first or the second product exact
__device__ __forceinline__ float dot_a(float a, float b, float c, float d) { return fmaf(a, b, mul(c, d)); }
__device__ __forceinline__ float dot_b(float a, float b, float c, float d) { return fmaf(c, d, mul(a, b)); }
__device__ __forceinline__ V scale(V a, float f) { return V{mul(f, a.x), mul(f, a.y), mul(f, a.z)}; }
__device__ __forceinline__ V diff(V a, V b) { return V{minus(a.x, b.x), minus(a.y, b.y), minus(a.z, b.z)}; }
__device__ __forceinline__ V fma3(float f, V a, V b) { return V{fmaf(f, a.x, b.x), fmaf(f, a.y, b.y), fmaf(f, a.z, b.z)}; }

__device__ __forceinline__ void quick_two_sum(float a, float b, float &s, float &e) {
    s = plus(a, b);
    e = minus(b, minus(s, a));
}
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = plus(a, b);
    const float bb = minus(s, a);
    e = plus(minus(a, minus(s, bb)), minus(b, bb));
}
// (hi, lo) += x
__device__ __forceinline__ void df_add(float &hi, float &lo, float x) {
    float s, e;
    two_sum(hi, x, s, e);
    quick_two_sum(s, plus(e, lo), hi, lo);
}
// (hi, lo) += a*b, the product exact in both places of the two-sum
__device__ __forceinline__ void df_fma(float &hi, float &lo, float a, float b) {
    const float s = fmaf(a, b, hi);
    const float bb = minus(s, hi);
    const float e = plus(minus(hi, minus(s, bb)), fmaf(a, b, -bb));
    quick_two_sum(s, plus(e, lo), hi, lo);
}
// (ah + al) - (bh + bl) to FP32 accuracy: the rounding of ah - bh is at most half an ulp of
// the difference itself (and none when ah and bh are within a factor 2), so no two-sum is
// needed when nothing is subtracted from the result afterwards
__device__ __forceinline__ float df_diff(float ah, float al, float bh, float bl) {
    return plus(minus(ah, bh), minus(al, bl));
}
// (ah + al) - (bh + bl) - (ch + cl): the axial deviation of a link (a - b ~= c).  The
// rounding of ah - bh is kept (two-sum): it can be as large as the deviation; s - ch is
// exact (Sterbenz) while the link's strain lies between -50% and +100%, and otherwise
// rounds a deviation as large as the rest length
__device__ __forceinline__ float df_diff3(float ah, float al, float bh, float bl, float ch, float cl) {
    float s, e;
    two_sum(ah, -bh, s, e);
    return plus(minus(s, ch), plus(e, minus(minus(al, bl), cl)));
}

// ToRotationVector (src/VX3/VX3_Quat3D.h:347-359) of a unit quaternion (w, v) in FP32.
// The reference takes 1 - w^2 as the squared sine of the half angle and, below
// 2.4e-3 (rotations under about 0.098 rad), does not evaluate the rotation vector
// 2*acos(w)/sin(theta/2) * v but the approximation 2*sqrt((2 - 2w)/(1 - w^2)) * v =
// 2*sqrt(2/(1 + w)) * v, which is smaller by about theta^2/96 relative: 2.6e-5 at
// 0.05 rad, far above FP32 rounding, in every link's bending and torsion terms.  The
// same two branches are taken here, with 1 - w^2 formed as |v|^2 (no cancellation)
// and acos(w)/sin as atan2(|v|, w)/|v|.
__device__ __forceinline__ V rotvec(float w, V v) {
    const float s2 = fmaf(v.z, v.z, dot_b(v.x, v.x, v.y, v.y));
    if (!(s2 > 0.0f)) return V{0, 0, 0};
    if (s2 < 2.4e-3f) return scale(v, mul(2.82842712f, rsqrtf(plus(1.0f, w))));
    const float is = rsqrtf(s2);  // s2 >= 2.4e-3 here
    return scale(v, mul(mul(2.0f, atan2f(mul(s2, is), w)), is));
}

// FromAngleToPosX (src/VX3/VX3_Quat3D.h:384-432) in FP32: the rotation taking r to
// +x.  The reference forms theta = acos(n.x) for n = r/|r| and returns
// (cos(theta/2), 0, n.z sin(theta/2)/|(n.y, n.z)|, -n.y sin(theta/2)/|(n.y, n.z)|).
// With the half-angle identities cos(theta/2) = sqrt((1 + n.x)/2) and
// sin(theta/2)/|(n.y, n.z)| = sqrt((1 - n.x)/2)/sqrt(1 - n.x^2) = 1/sqrt(2(1 + n.x))
// that is (c/2, 0, n.z/c, -n.y/c) with c = sqrt(2(1 + n.x)): one square root and one
// reciprocal instead of acos, sin and cos.  The small-angle shortcut and the
// turned-around case (theta within 1e-7 of pi, where 1 + n.x underflows in FP32)
// are the reference's.
__device__ __forceinline__ Q from_angle_to_posx(V r) {
    if (r.x == 0 && r.y == 0 && r.z == 0) return Q{1, 0, 0, 0};
    const float yx = __fdividef(r.y, r.x), zx = __fdividef(r.z, r.x);
    const float SA = 1.732e-2f;
    if (yx < SA && yx > -SA && zx < SA && zx > -SA) {
        const float qy = mul(0.5f, zx), qz = mul(-0.5f, yx);
        return Q{fmaf(0.5f, dot_a(-qy, qy, -qz, qz), 1.0f), 0, qy, qz};
    }
    const float il = rsqrtf(fmaf(r.z, r.z, dot_b(r.x, r.x, r.y, r.y)));
    const float ny = mul(r.y, il), nz = mul(r.z, il);
    const float t = mul(2.0f, fmaf(r.x, il, 1.0f));  // 2 (1 + n.x)
    if (!(t > 0.0f)) return Q{0, 0, 1, 0};
    const float ic = rsqrtf(t), c = mul(t, ic);
    return Q{mul(0.5f, c), 0, mul(nz, ic), mul(-ny, ic)};
}

// q v q* of the negative end's conjugate orientation (link pass)
__device__ __forceinline__ V rotate_link(Q q, V f) {
    const float tw = fmaf(f.z, q.z, dot_b(f.x, q.x, f.y, q.y)), tx = fmaf(f.z, q.y, dot_b(f.x, q.w, -f.y, q.z));
    const float ty = fmaf(-f.z, q.x, dot_b(f.x, q.z, f.y, q.w)), tz = fmaf(f.z, q.w, dot_a(-f.x, q.y, f.y, q.x));
    return V{fmaf(-q.z, ty, fmaf(q.y, tz, dot_a(q.w, tx, q.x, tw))), fmaf(q.z, tx, fmaf(q.y, tw, dot_a(q.w, ty, -q.x, tz))),
             fmaf(q.z, tw, fmaf(-q.y, tx, dot_a(q.w, tz, q.x, ty)))};
}
// q v q* of a voxel's orientation (voxel pass)
__device__ __forceinline__ V rotate_voxel(Q q, V f) {
    const float tw = fmaf(f.z, q.z, dot_a(f.x, q.x, f.y, q.y)), tx = fmaf(f.z, q.y, dot_a(f.x, q.w, -f.y, q.z));
    const float ty = fmaf(-f.z, q.x, dot_a(f.x, q.z, f.y, q.w)), tz = fmaf(f.z, q.w, dot_b(-f.x, q.y, f.y, q.x));
    return V{fmaf(-q.z, ty, fmaf(q.y, tz, dot_a(q.w, tx, q.x, tw))), fmaf(q.z, tx, fmaf(q.y, tw, dot_a(q.w, ty, -q.x, tz))),
             fmaf(q.z, tw, fmaf(-q.y, tx, dot_a(q.w, tz, q.x, ty)))};
}
// q* v q
__device__ __forceinline__ V rotate_inv(Q q, V f) {
    const float tw = fmaf(q.z, f.z, dot_b(q.x, f.x, q.y, f.y)), tx = fmaf(q.z, f.y, dot_a(q.w, f.x, -q.y, f.z));
    const float ty = fmaf(-q.z, f.x, dot_b(q.w, f.y, q.x, f.z)), tz = fmaf(q.y, f.x, dot_a(q.w, f.z, -q.x, f.y));
    return V{fmaf(-tz, q.y, fmaf(ty, q.z, dot_a(tw, q.x, tx, q.w))), fmaf(tz, q.x, fmaf(ty, q.w, dot_a(tw, q.y, -tx, q.z))),
             fmaf(tz, q.w, fmaf(-ty, q.x, dot_a(tw, q.z, tx, q.y)))};
}
// the same of a quaternion with x = 0 (FromAngleToPosX)
__device__ __forceinline__ V rotate_inv_x0(Q q, V f) {
    const float tw = fmaf(q.z, f.z, mul(q.y, f.y)), tx = fmaf(q.z, f.y, dot_a(q.w, f.x, -q.y, f.z));
    const float ty = fmaf(-q.z, f.x, mul(q.w, f.y)), tz = fmaf(q.y, f.x, mul(q.w, f.z));
    return V{fmaf(-tz, q.y, fmaf(ty, q.z, mul(tx, q.w))), fmaf(ty, q.w, dot_a(tw, q.y, -tx, q.z)),
             fmaf(tz, q.w, dot_a(tw, q.z, tx, q.y))};
}
__device__ __forceinline__ Q product(Q a, Q f) {
    return Q{fmaf(-a.z, f.z, fmaf(-a.y, f.y, dot_a(a.w, f.w, -a.x, f.x))), fmaf(-a.z, f.y, fmaf(a.y, f.z, dot_a(a.w, f.x, a.x, f.w))),
             fmaf(a.z, f.x, fmaf(a.y, f.w, dot_a(a.w, f.y, -a.x, f.z))), fmaf(a.z, f.w, fmaf(-a.y, f.x, dot_a(a.w, f.z, a.x, f.y)))};
}
__device__ __forceinline__ Q product_x0(Q a, Q f) {  // a.x = 0
    return Q{fmaf(-a.z, f.z, fmaf(-a.y, f.y, mul(a.w, f.w))), fmaf(-a.z, f.y, fmaf(a.y, f.z, mul(a.w, f.x))),
             fmaf(a.z, f.x, fmaf(a.y, f.w, mul(a.w, f.y))), fmaf(a.z, f.w, fmaf(-a.y, f.x, mul(a.w, f.z)))};
}

// ------------------------------------------------------------- material constants
// What a step reads of a link or voxel material, as 16-byte rows (Dev::lrow, Dev::vrow, row k of
// material i at [k * count + i]): a warp's lanes pick among a few materials, so a row costs one or
// two cache lines where the fields of an array of structs cost a line per material and field.
struct LinkC {
    float4 ra;  // b1, b2, b3, a2
    float4 rb;  // sqA1, sqA2xIp, sqB1, sqB2xFMp
    float4 rc;  // sqB3xIp, the ends' damping multipliers / dt, transverse area (negative: non-linear model)
    float4 re;  // stress = e.x * (e.y * strain + e.z) of a linear model; failure strain (-1: none)
    __device__ __forceinline__ float4 a() const { return ra; }
    __device__ __forceinline__ float4 b() const { return rb; }
    __device__ __forceinline__ float4 c() const { return rc; }
    __device__ __forceinline__ float4 e() const { return re; }
};
struct VoxC {
    float4 a;  // 1/mass, 1/inertia (negative: expansion turns on later), global damping of translation, rotation
    float4 c;  // weight, CTE, nominal size hi, lo
    const float4 *rb;  // collision damping, kinetic friction, penetration stiffness, static friction: read in contact only
    __device__ __forceinline__ float4 b() const { return *rb; }
};
__device__ __forceinline__ LinkC link_consts_mx(const LMat &m, float dt) {
    // dampingMultiplier / dt, infinite for a Fixed end (its numerator over a zero time step)
    const float idt = __fdividef(1.0f, dt);
    LinkC c;
    c.ra = make_float4(m.b1, m.b2, m.b3, m.a2);
    c.rb = make_float4(m.sqA1, m.sqA2xIp, m.sqB1, m.sqB2xFMp);
    c.rc = make_float4(m.sqB3xIp, mul(m.dmcN, m.fixN ? CUDART_INF_F : idt), mul(m.dmcP, m.fixP ? CUDART_INF_F : idt),
                      m.lin ? m.area : -m.area);
    c.re = m.nu == 0.0f ? make_float4(m.E, 1.0f, 0.0f, m.eps_fail)
                       : make_float4(m.eHat, minus(1.0f, m.nu), mul(m.nu, m.tss), m.eps_fail);
    return c;
}
__device__ __forceinline__ float4 vox_row_a(const VMat &m) {
    return make_float4(m.mass_inv, m.toa_pos ? -m.mom_inv : m.mom_inv, m.c_glob, m.c_glob_rot);
}
__device__ __forceinline__ float4 vox_row_b(const VMat &m) { return make_float4(m.c_col, m.mu_k, m.pstiff, m.mu_s); }
__device__ __forceinline__ float4 vox_row_c(const VMat &m) { return make_float4(m.grav_force, m.cte, m.nom_hi, m.nom_lo); }
// rows i of a table of n materials; a link's either held in registers from the start (LinkC) or read where
// they are used (LinkRows)
struct LinkRows {
    const float4 *t;
    int n;
    __device__ __forceinline__ float4 a() const { return t[0]; }
    __device__ __forceinline__ float4 b() const { return t[n]; }
    __device__ __forceinline__ float4 c() const { return t[2 * n]; }
    __device__ __forceinline__ float4 e() const { return t[3 * n]; }
};
template <bool HELD> __device__ __forceinline__ auto link_rows(const float4 *t, int n, int i) {
    const LinkRows r{t + i, n};
    if constexpr (HELD) return LinkC{r.a(), r.b(), r.c(), r.e()};
    else return r;
}
__device__ __forceinline__ VoxC vox_rows(const float4 *t, int n, int i) { return VoxC{t[i], t[2 * n + i], t + n + i}; }

// ------------------------------------------------------------- link
struct Ends {  // a voxel's position and orientation pairs, hi and lo; pos.w the base size
    float4 pH, pL, qH, qL;
};
struct LinkState {
    V pos2, a1v, a2v;
    float2 strain;  // {strain, maxStrain}
    uint32_t fl;
};
// One link's update from its ends; l is read for non-linear materials only (their curve and the plastic
// offset).  What it leaves is handed to `out` as soon as it is known, so that it does not sit in registers
// until the end: the local state, the strain (torn: above 100, VX3_VoxelyzeKernel.cu:271-281), the flags,
// and force and moment of the negative and the positive end in the lattice frame.
template <class Rows, class Out>
__device__ __forceinline__ void link_step(const Dev &d, const Rows &m, int l, const Ends &en, const Ends &ep,
                                          const LinkState &s, Out &out) {
    const uint32_t fl = s.fl;
    const int axis = (int)(fl & LF_AXIS);
    // rest length L = 0.5*(bsNeg + bsPos) as a hi/lo pair (VX3_Link::updateRestLength)
    float Lh, Ll;
    two_sum(en.pH.w, ep.pH.w, Lh, Ll);
    Ll = plus(Ll, plus(en.pL.w, ep.pL.w));
    quick_two_sum(mul(0.5f, Lh), mul(0.5f, Ll), Lh, Ll);
    // delta = (pPos - pNeg) - L*e_axis in the global frame
    const float ax = axis == 0 ? Lh : 0.0f, ay = axis == 1 ? Lh : 0.0f, az = axis == 2 ? Lh : 0.0f;
    const float axl = axis == 0 ? Ll : 0.0f, ayl = axis == 1 ? Ll : 0.0f, azl = axis == 2 ? Ll : 0.0f;
    const V delta{df_diff3(ep.pH.x, ep.pL.x, en.pH.x, en.pL.x, ax, axl), df_diff3(ep.pH.y, ep.pL.y, en.pH.y, en.pL.y, ay, ayl),
                  df_diff3(ep.pH.z, ep.pL.z, en.pH.z, en.pL.z, az, azl)};
    const Q a1 = to_axis_xq(axis, Q{en.qH.x, en.qH.y, en.qH.z, en.qH.w});
    const Q dq = to_axis_xq(axis, Q{df_diff(ep.qH.x, ep.qL.x, en.qH.x, en.qL.x), df_diff(ep.qH.y, ep.qL.y, en.qH.y, en.qL.y),
                                    df_diff(ep.qH.z, ep.qL.z, en.qH.z, en.qL.z), df_diff(ep.qH.w, ep.qL.w, en.qH.w, en.qL.w)});
    const Q c = qconj(a1);
    const Q cd = product(c, dq);  // angle2 = conj(q1)*q2 = |q1|^2 + conj(q1)*(q2-q1), |q1| = 1
    const V rd = rotate_link(c, to_axis_x(axis, delta));
    const float L = Lh;
    const float pxm = fmaf(mul(-2.0f, L), dot_a(a1.y, a1.y, a1.z, a1.z), rd.x);  // pos2.x - L
    const float py = fmaf(mul(2.0f, L), dot_a(a1.x, a1.y, -a1.w, a1.z), rd.y);
    const float pz = fmaf(mul(2.0f, L), dot_b(a1.x, a1.z, a1.w, a1.y), rd.z);
    const float px = plus(L, pxm);
    // hysteresis on SmallTurn = (|pz| + |py|)/px and ExtendPerc = |pxm/L| (L > 0),
    // compared without dividing: px < 0 (bent past 90 degrees) gives SmallTurn <= 0,
    // px = 0 gives +inf (or NaN when the numerator is 0 too)
    const float HF = 1.2f, BEND = 0.05f, EXT = 0.50f;
    const float turn = plus(fabsf(pz), fabsf(py)), ext = fabsf(pxm);
    const bool turnBelow = px > 0.0f ? turn < mul(BEND, px) : px < 0.0f;
    const bool turnAbove = px > 0.0f ? turn > mul(HF * BEND, px) : (px == 0.0f && turn > 0.0f);
    bool small = (fl & LF_SMALL) != 0, lvv = (fl & LF_LVV) != 0;
    if (!small && turnBelow && ext < mul(EXT, L)) {
        small = true;
        lvv = false;
    } else if (small && (turnAbove || ext > mul(HF * EXT, L))) {
        small = false;
        lvv = false;
    }
    Q angle1{1, 0, 0, 0};
    Q angle2{plus(1.0f, cd.w), cd.x, cd.y, cd.z};
    V pos2{pxm, py, pz}, a1v{0, 0, 0};
    if (!small) {
        angle1 = from_angle_to_posx(V{px, py, pz});
        angle2 = product_x0(angle1, angle2);
        const float zz = mul(pz, pz);
        const float l2 = plus(dot_a(px, px, py, py), zz);
        const float len2 = l2 > 0.0f ? mul(l2, rsqrtf(l2)) : 0.0f;
        pos2 = V{__fdividef(plus(dot_a(pxm, plus(px, L), py, py), zz), plus(len2, L)), 0, 0};  // |pos2| - L
        a1v = rotvec(angle1.w, V{angle1.x, angle1.y, angle1.z});
    }
    const V a2v = rotvec(angle2.w, V{angle2.x, angle2.y, angle2.z});
    const V dP = scale(diff(pos2, s.pos2), 0.5f), d1 = scale(diff(a1v, s.a1v), 0.5f), d2 = scale(diff(a2v, s.a2v), 0.5f);
    out.local(pos2, a1v, a2v, small);
    // FP32 quotients in the hot paths use the hardware reciprocal (__fdividef: within 2 ulp)
    const float axialStrain = __fdividef(pos2.x, L);
    float2 strain = make_float2(axialStrain, s.strain.y);
    float stress;  // updateStrain (VX3_Link.cu:220-260)
    const float4 mc = m.c(), me = m.e();
    if (mc.w > 0.0f) {
        if (axialStrain > strain.y) strain.y = axialStrain;
        stress = me.w != -1.0f && axialStrain > me.w ? 0.0f : mul(me.x, fmaf(me.y, axialStrain, me.z));
    } else {
        stress = link_stress(d, d.lmat[fl >> 8], l, axialStrain, &strain.y);
    }
    out.strain(strain, axialStrain > 100);
    const uint32_t nfl = (fl & ~(LF_SMALL | LF_LVV)) | (small ? LF_SMALL : 0u);
    if (me.w != -1.0f && strain.y > me.w) {  // isFailed: forces zero
        const V z{0, 0, 0};
        out.neg(z, z);
        out.pos(z, z);
        out.flags(nfl | (lvv ? LF_LVV : 0u), true);
        return;
    }
    const float4 ma = m.a();
    const float b1 = ma.x, b2 = ma.y, b3 = ma.z, a2 = ma.w;
    V fN = V{mul(stress, fabsf(mc.w)), dot_a(b1, pos2.y, -b2, plus(a1v.z, a2v.z)), dot_a(b1, pos2.z, b2, plus(a1v.y, a2v.y))};
    V fP = neg(fN);
    V mN = V{mul(a2, minus(a2v.x, a1v.x)), dot_b(-b2, pos2.z, -b3, fmaf(2.0f, a1v.y, a2v.y)),
             dot_b(b2, pos2.y, -b3, fmaf(2.0f, a1v.z, a2v.z))};
    V mP = V{mul(a2, minus(a1v.x, a2v.x)), dot_b(-b2, pos2.z, -b3, fmaf(2.0f, a2v.y, a1v.y)),
             dot_b(b2, pos2.y, -b3, fmaf(2.0f, a2v.z, a1v.z))};
    if (lvv) {
        const float4 mb = m.b();
        const float sB1 = mb.z, sB2 = mb.w, sB3 = mc.x, dmN = mc.y, dmP = mc.z;
        const V pc{mul(mb.x, dP.x), dot_a(sB1, dP.y, -sB2, plus(d1.z, d2.z)), dot_b(sB1, dP.z, sB2, plus(d1.y, d2.y))};
        const float tw = mul(mb.y, minus(d2.x, d1.x));
        fN = fma3(dmN, pc, fN);
        fP = fma3(-dmP, pc, fP);
        mN = fma3(mul(-0.5f, dmN), V{-tw, dot_a(sB2, dP.z, sB3, fmaf(2.0f, d1.y, d2.y)), dot_b(-sB2, dP.y, sB3, fmaf(2.0f, d1.z, d2.z))}, mN);
        mP = fma3(mul(-0.5f, dmP), V{tw, dot_a(sB2, dP.z, sB3, fmaf(2.0f, d2.y, d1.y)), dot_b(-sB2, dP.y, sB3, fmaf(2.0f, d2.z, d1.z))}, mP);
    }
    if (!small) {
        fN = rotate_inv_x0(angle1, fN);
        mN = rotate_inv_x0(angle1, mN);
    }
    out.neg(to_axis_original(axis, fN), to_axis_original(axis, mN));
    fP = rotate_inv(angle2, fP);
    mP = rotate_inv(angle2, mP);
    out.pos(to_axis_original(axis, fP), to_axis_original(axis, mP));
    out.flags(nfl | LF_LVV, false);
}

// base size nomSize*(1 + T*cte) as a hi/lo pair
__device__ __forceinline__ void base_size(float4 mc, float te, float &hi, float &lo) {  // row c of the material
    const float f = fmaf(te, mc.y, 1.0f);
    const float p = mul(mc.z, f);
    quick_two_sum(p, fmaf(mc.w, f, fmaf(mc.z, f, -p)), hi, lo);
}

// temperature at the end of a step (gpu_update_temperature, VX3_VoxelyzeKernel.cu:625-650)
// from the cycles of the phase 2*3.1415926f*(t/P + phase) / (2 pi): the robot's cycles at
// the step's start tc and the voxel's phase cycles ph, each frac(.) reduced in FP64 once
// (by the writer of the robot's time, and at create) and held as FP32 hi + lo pairs, plus
// the step's dt * cycles per second (about 5e-4 cycles, rounded to 3e-11).  The sum c_hi +
// c_lo is formed with two-sums, and sin(2 pi c) = sin(2 pi c_hi) + 2 pi c_lo cos(2 pi c_hi),
// the second term dropping (2 pi c_lo)^2 / 2 < 1e-13.  The FP32 sine of a rounded c alone
// would carry up to 3.7e-7 rad of phase; with the correction the temperature is within
// about one FP32 rounding of the FP64 step's, and no FP64 arithmetic runs per voxel.
__device__ __forceinline__ float temperature(float2 tc, float2 ph, float dtf, float cyc_rate, float amp, bool expansion) {
    float s, e;
    two_sum(tc.x, ph.x, s, e);
    s = minus(s, floorf(s));  // exact: s lies in [0, 2]
    e = plus(e, fmaf(dtf, cyc_rate, plus(tc.y, ph.y)));
    float ch, cl;
    two_sum(s, e, ch, cl);
    float sn, cs;
    sincospif(mul(2.0f, ch), &sn, &cs);
    float T = mul(amp, fmaf(mul(6.28318531f, cl), cs, sn));
    if (!expansion && T > 0) T = 0;
    return T;
}

// ------------------------------------------------------------- voxel
struct VoxelState {
    float4 pH, pL, qH, qL, lH, lL, aH, aL;  // position (w: base size), orientation, momenta
};

__device__ __forceinline__ V velocity(float4 hi, float4 lo, float k) {
    return V{mul(plus(hi.x, lo.x), k), mul(plus(hi.y, lo.y), k), mul(plus(hi.z, lo.z), k)};
}
__device__ __forceinline__ float penetration(const VoxelState &s, const VoxC &m) {  // (VX3_Voxel.h:185-188)
    return fmaf(0.5f, plus(minus(s.pH.w, m.c.z), minus(s.pL.w, m.c.w)), -plus(s.pH.z, s.pL.z));
}

// floor contact, friction and the translation (VX3_Voxel.cu:186-219, 399-426)
__device__ __forceinline__ void move(VoxelState &s, const VoxC &m, V F, V vel, bool floorOn, float dtf, bool &stat) {
    const float pen = penetration(s, m);
    V fric = F;
    if (floorOn) {
        if (pen >= 0) {
            const float4 mb = m.b();
            const float normal = mul(mb.z, pen);
            F.z = plus(F.z, fmaf(-mb.x, vel.z, normal));
            if (stat) {
                const float lim = mul(mb.w, normal);
                if (dot_a(F.x, F.x, F.y, F.y) > mul(lim, lim)) stat = false;
            } else {
                // the horizontal velocity's direction (normalized(): unchanged when zero)
                const float h2 = dot_a(vel.x, vel.x, vel.y, vel.y);
                const float k = h2 > 0.0f ? rsqrtf(h2) : 1.0f;
                const float mk = mul(mb.y, normal);
                F.x = fmaf(-mk, mul(vel.x, k), F.x);
                F.y = fmaf(-mk, mul(vel.y, k), F.y);
            }
        } else {
            stat = false;
        }
    }
    fric.x = minus(F.x, fric.x);
    fric.y = minus(F.y, fric.y);
    df_fma(s.lH.x, s.lL.x, F.x, dtf);
    df_fma(s.lH.y, s.lL.y, F.y, dtf);
    df_fma(s.lH.z, s.lL.z, F.z, dtf);
    const float km = mul(dtf, m.a.x);
    const float lx = plus(s.lH.x, s.lL.x), ly = plus(s.lH.y, s.lL.y), lz = plus(s.lH.z, s.lL.z);
    float tx = mul(lx, km), ty = mul(ly, km);
    if (floorOn && pen >= 0) {
        const float work = dot_a(fric.x, tx, fric.y, ty);
        if (fmaf(mul(0.5f, m.a.x), dot_a(lx, lx, ly, ly), work) <= 0) stat = true;
        if (stat) {
            s.lH.x = s.lL.x = s.lH.y = s.lL.y = 0;
            tx = ty = 0;
        }
    } else {
        stat = false;
    }
    df_add(s.pH.x, s.pL.x, tx);
    df_add(s.pH.y, s.pL.y, ty);
    df_fma(s.pH.z, s.pL.z, lz, km);
}

// the rotation: L += M dt, q' = Quat(angMom*dt/I)*q = q + (dq - 1)*q (FromRotationVector,
// VX3_Quat3D.h:363-377)
__device__ __forceinline__ void turn(VoxelState &s, const VoxC &m, V M, float dtf) {
    df_fma(s.aH.x, s.aL.x, M.x, dtf);
    df_fma(s.aH.y, s.aL.y, M.y, dtf);
    df_fma(s.aH.z, s.aL.z, M.z, dtf);
    const float ki = mul(dtf, fabsf(m.a.y));
    const V th{mul(mul(0.5f, plus(s.aH.x, s.aL.x)), ki), mul(mul(0.5f, plus(s.aH.y, s.aL.y)), ki),
               mul(mul(0.5f, plus(s.aH.z, s.aL.z)), ki)};
    const float m2 = fmaf(th.z, th.z, dot_a(th.x, th.x, th.y, th.y));
    float dw, sfac;
    if (mul(m2, m2) < 5.328e-15f) {
        dw = mul(-0.5f, m2);
        sfac = fmaf(-m2, 1.0f / 6.0f, 1.0f);
    } else if (m2 < 0.25f) {
        // |theta| < 0.5 rad: cos|theta| - 1 and sin|theta| / |theta| as their Taylor series in
        // m2 = |theta|^2, truncated where the next term is below 3e-10 (no square root,
        // sine or division; the same values to FP32 rounding)
        dw = mul(m2, fmaf(m2, fmaf(m2, fmaf(m2, fmaf(-m2, 1.0f / 3628800, 1.0f / 40320), -1.0f / 720), 1.0f / 24), -0.5f));
        sfac = fmaf(m2, fmaf(m2, fmaf(m2, fmaf(m2, 1.0f / 362880, -1.0f / 5040), 1.0f / 120), -1.0f / 6), 1.0f);
    } else {
        const float im = rsqrtf(m2);  // 1 / |theta|, m2 >= 0.25 here
        float sn, cs;
        sincospif(mul(mul(m2, im), 0.159154943f), &sn, &cs);  // sin, cos of |theta| / 2
        dw = mul(mul(-2.0f, sn), sn);
        sfac = mul(mul(mul(2.0f, sn), cs), im);
    }
    const Q delta = product(Q{dw, mul(th.x, sfac), mul(th.y, sfac), mul(th.z, sfac)}, Q{s.qH.x, s.qH.y, s.qH.z, s.qH.w});
    df_add(s.qH.x, s.qL.x, delta.w);
    df_add(s.qH.y, s.qL.y, delta.x);
    df_add(s.qH.z, s.qL.z, delta.y);
    df_add(s.qH.w, s.qL.w, delta.z);
}

// frac(c) as an FP32 hi + lo pair
__device__ __forceinline__ float2 cycles_df(double c) {
    c -= floor(c);
    const float h = (float)c;
    return make_float2(h, (float)(c - (double)h));
}

}  // namespace mx
}  // namespace vx3g
