// vx3g_step.cuh -- the two per-step passes in the reference's arithmetic (FP64 vectors; float
// wherever the reference uses float) and the math they share with the other units.  Compiled
// with --fmad=false so that the rounding sequence matches the reference step op for op.
//
// Link pass  : VX3_Link::orientLink + updateForces + updateStrain
//              (src/VX3/VX3_Link.cu:90-260), one thread per link.
// Voxel pass : VX3_Voxel::timeStep with force()/moment()/floorForce()
//              (src/VX3/VX3_Voxel.cu:162-277, 350-426), one thread per voxel, plus the
//              next step's temperature (gpu_update_temperature, VX3_VoxelyzeKernel.cu:625-650).
#pragma once

#include <type_traits>

#include "vx3g_internal.h"

namespace vx3g {

template <class R> struct V3 { R x, y, z; };
template <class R> struct Q4 { R w, x, y, z; };

template <class R> __device__ __forceinline__ V3<R> v3(R x, R y, R z) { return V3<R>{x, y, z}; }
template <class R> __device__ __forceinline__ V3<R> add(V3<R> a, V3<R> b) { return V3<R>{a.x + b.x, a.y + b.y, a.z + b.z}; }
template <class R> __device__ __forceinline__ V3<R> sub(V3<R> a, V3<R> b) { return V3<R>{a.x - b.x, a.y - b.y, a.z - b.z}; }
template <class R> __device__ __forceinline__ V3<R> neg(V3<R> a) { return V3<R>{-a.x, -a.y, -a.z}; }
// VX3_Vec3D::operator*(f) -> (f*x, f*y, f*z)   (VX3_Vec3D.h:49,61)
template <class R, class F> __device__ __forceinline__ V3<R> scl(V3<R> a, F f) {
    return V3<R>{(R)(f * a.x), (R)(f * a.y), (R)(f * a.z)};
}
// VX3_Vec3D::operator/(f) -> Inv = 1/f; (Inv*x, ...)   (VX3_Vec3D.h:63)
template <class R> __device__ __forceinline__ V3<R> vdiv(V3<R> a, R f) {
    R inv = (R)1.0 / f;
    return V3<R>{inv * a.x, inv * a.y, inv * a.z};
}
template <class R> __device__ __forceinline__ R len(V3<R> a) { return sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
template <class R> __device__ __forceinline__ V3<R> normalized(V3<R> a) {
    R l = sqrt(a.x * a.x + a.y * a.y + a.z * a.z);
    return l > 0 ? vdiv(a, l) : a;
}

template <class R> __device__ __forceinline__ Q4<R> qconj(Q4<R> q) { return Q4<R>{q.w, -q.x, -q.y, -q.z}; }
// VX3_Quat3D.h:217-222
template <class R> __device__ __forceinline__ Q4<R> qmul(Q4<R> a, Q4<R> f) {
    return Q4<R>{a.w * f.w - a.x * f.x - a.y * f.y - a.z * f.z, a.w * f.x + a.x * f.w + a.y * f.z - a.z * f.y,
                 a.w * f.y - a.x * f.z + a.y * f.w + a.z * f.x, a.w * f.z + a.x * f.y - a.y * f.x + a.z * f.w};
}
// VX3_Quat3D.h:439-447
template <class R> __device__ __forceinline__ V3<R> qrot(Q4<R> q, V3<R> f) {
    R tw = f.x * q.x + f.y * q.y + f.z * q.z;
    R tx = f.x * q.w - f.y * q.z + f.z * q.y;
    R ty = f.x * q.z + f.y * q.w - f.z * q.x;
    R tz = -f.x * q.y + f.y * q.x + f.z * q.w;
    return V3<R>{q.w * tx + q.x * tw + q.y * tz - q.z * ty, q.w * ty - q.x * tz + q.y * tw + q.z * tx,
                 q.w * tz + q.x * ty - q.y * tx + q.z * tw};
}
// VX3_Quat3D.h:465-473
template <class R> __device__ __forceinline__ V3<R> qrotinv(Q4<R> q, V3<R> f) {
    R tw = q.x * f.x + q.y * f.y + q.z * f.z;
    R tx = q.w * f.x - q.y * f.z + q.z * f.y;
    R ty = q.w * f.y + q.x * f.z - q.z * f.x;
    R tz = q.w * f.z - q.x * f.y + q.y * f.x;
    return V3<R>{tw * q.x + tx * q.w + ty * q.z - tz * q.y, tw * q.y - tx * q.z + ty * q.w + tz * q.x,
                 tw * q.z + tx * q.y - ty * q.x + tz * q.w};
}

// ------------------------------------------------------------- FP64 arithmetic that is not FP64
// GB300 starts an FP64 warp instruction every 19 cycles per SM (64 cycles per warp, active lanes
// or not, measured) and a float-to-double conversion every 16, against four FP32 or integer ones
// per cycle: the FP64 passes are bound by the number of FP64 instructions.  What is only compared
// is therefore compared as integers or in FP32 with a margin, falling back to the exact FP64
// expression inside the margin, and FP32 constants come converted (LMatD) or are widened with
// integer operations.  Values keep the reference's rounding, operation for operation.
__device__ __forceinline__ int hi_word(double x) {
#if defined(__CUDA_ARCH__)
    return __double2hiint(x);
#else
    long long b;
    __builtin_memcpy(&b, &x, 8);
    return (int)(b >> 32);
#endif
}
__device__ __forceinline__ int lo_word(double x) {
#if defined(__CUDA_ARCH__)
    return __double2loint(x);
#else
    long long b;
    __builtin_memcpy(&b, &x, 8);
    return (int)b;
#endif
}
__device__ __forceinline__ double from_words(int hi, int lo) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double(hi, lo);
#else
    const long long b = ((long long)hi << 32) | (unsigned)lo;
    double x;
    __builtin_memcpy(&x, &b, 8);
    return x;
#endif
}
__device__ __forceinline__ float int_float(int i) {
#if defined(__CUDA_ARCH__)
    return __int_as_float(i);
#else
    float f;
    __builtin_memcpy(&f, &i, 4);
    return f;
#endif
}
__device__ __forceinline__ int float_int(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_int(f);
#else
    int i;
    __builtin_memcpy(&i, &f, 4);
    return i;
#endif
}
// (double)f, exact
__device__ __forceinline__ double widen(float f) {
    const int b = float_int(f), e = b & 0x7f800000;
    if (e == 0 || e == 0x7f800000) return (double)f;
    return from_words((b & (int)0x80000000) | (((b & 0x7fffffff) >> 3) + 0x38000000), b << 29);
}
// |x| in FP32, truncated: at most 2^-20 relative below |x|; 0 below FP32's range, a huge value or
// NaN above it.  For comparisons with a margin.
__device__ __forceinline__ float mag(double x) {
    const int h = (hi_word(x) & 0x7fffffff) - 0x38000000;
    return int_float(h < 0 ? 0 : h >= 0x0ff00000 ? 0x7fc00000 : h << 3);
}
__device__ __forceinline__ float signed_mag(double x) {
    return int_float(float_int(mag(x)) | (hi_word(x) & (int)0x80000000));
}

// qmul and qrotinv by a quaternion with x = 0 (FromAngleToPosX): the products with it, zeros, left out
__device__ __forceinline__ Q4<double> qmul_x0(Q4<double> a, Q4<double> f) {
    return Q4<double>{a.w * f.w - a.y * f.y - a.z * f.z, a.w * f.x + a.y * f.z - a.z * f.y, a.w * f.y + a.y * f.w + a.z * f.x,
                      a.w * f.z - a.y * f.x + a.z * f.w};
}
__device__ __forceinline__ V3<double> qrotinv_x0(Q4<double> q, V3<double> f) {
    const double tw = q.y * f.y + q.z * f.z, tx = q.w * f.x - q.y * f.z + q.z * f.y;
    const double ty = q.w * f.y - q.z * f.x, tz = q.w * f.z + q.y * f.x;
    return V3<double>{tx * q.w + ty * q.z - tz * q.y, tw * q.y - tx * q.z + ty * q.w, tw * q.z + tx * q.y + tz * q.w};
}

// ToRotationVector (VX3_Quat3D.h:347-359), its comparisons on the bits (|w| >= 1; 1 - w^2 >= 0)
__device__ __forceinline__ V3<double> to_rotvec(Q4<double> q) {
    if ((unsigned)((hi_word(q.w) & 0x7fffffff) - 0x3ff00000) <= 0x40000000u) return V3<double>{0, 0, 0};  // |w| >= 1
    const V3<double> v{q.x, q.y, q.z};
    const double sq = 1.0 - q.w * q.w;
    if (mag(sq) < 2.399e-3f || sq < 2.4e-3) {
        const double g = sqrt(fma(-2.0, q.w, 2.0) / sq);  // 1 to 1.0003
        return scl(v, from_words(hi_word(g) + 0x100000, lo_word(g)));  // 2g
    }
    return vdiv(scl(scl(v, 2.0), acos(q.w)), sqrt(sq));
}

// FromRotationVector (VX3_Quat3D.h:363-377) of the rotation vector 2*th.  sincos gives the bits of
// sin and cos for 27 FP64 instructions instead of 43.
__device__ __forceinline__ Q4<double> from_half_rotvec(V3<double> th) {
    const double m2 = th.x * th.x + th.y * th.y + th.z * th.z;
    double w, s;
    if (m2 * m2 < 5.328e-15) {
        w = fma(-0.5, m2, 1.0);
        s = 1.0 - m2 / 6.0;
    } else {
        const double m = sqrt(m2);
        sincos(m, &s, &w);
        s = s / m;
    }
    return Q4<double>{w, th.x * s, th.y * s, th.z * s};
}
__device__ __forceinline__ Q4<double> from_rotvec(V3<double> in) { return from_half_rotvec(scl(in, 0.5)); }

// FromAngleToPosX (VX3_Quat3D.h:384-432); q unchanged for a zero vector.  l = |r|.
__device__ __forceinline__ Q4<double> from_angle_to_posx(Q4<double> q, V3<double> r, double l) {
    if (r.x == 0 && r.y == 0 && r.z == 0) return q;
    const float sx = 0.0174f * mag(r.x);
    if (!(mag(r.y) > sx || mag(r.z) > sx)) {  // near the shortcut's bound: decide exactly
        const double yx = r.y / r.x, zx = r.z / r.x, SA = 1.732e-2;
        if (yx < SA && yx > -SA && zx < SA && zx > -SA) {
            q.x = 0;
            q.y = 0.5 * zx;
            q.z = -0.5 * yx;
            q.w = 1 + 0.5 * (-q.y * q.y - q.z * q.z);
            return q;
        }
    }
    V3<double> n = r;
    if (l > 0) {
        const double li = 1.0 / l;
        n.x *= li; n.y *= li; n.z *= li;
    }
    const double theta = acos(n.x);
    if (theta > 3.14159265358979 - 1e-7) return Q4<double>{0, 0, 1, 0};
    const double axis_inv = 1.0 / sqrt(n.z * n.z + n.y * n.y);
    double s, c;
    sincos(0.5 * theta, &s, &c);
    return Q4<double>{c, 0, n.z * axis_inv * s, -n.y * axis_inv * s};
}

__device__ __forceinline__ bool is_zero(V3<double> a) {  // on the bits, either sign
    return (((hi_word(a.x) | hi_word(a.y) | hi_word(a.z)) & 0x7fffffff) | lo_word(a.x) | lo_word(a.y) | lo_word(a.z)) == 0;
}

// VX3_Link.h:134-191 (bond-local +X frame and back)
// written as per-component selects (no branches: a warp's links mix the three axes)
template <class R> __device__ __forceinline__ V3<R> to_axis_x(int axis, V3<R> v) {
    const bool a1 = axis == 1, a2 = axis == 2;
    return V3<R>{a1 ? v.y : (a2 ? v.z : v.x), a1 ? -v.x : v.y, a2 ? -v.x : v.z};
}
template <class R> __device__ __forceinline__ Q4<R> to_axis_xq(int axis, Q4<R> q) {
    const bool a1 = axis == 1, a2 = axis == 2;
    return Q4<R>{q.w, a1 ? q.y : (a2 ? q.z : q.x), a1 ? -q.x : q.y, a2 ? -q.x : q.z};
}
template <class R> __device__ __forceinline__ V3<R> to_axis_original(int axis, V3<R> v) {
    const bool a1 = axis == 1, a2 = axis == 2;
    return V3<R>{a1 ? -v.y : (a2 ? -v.z : v.x), a1 ? v.x : v.y, a2 ? v.x : v.z};
}

// The voxel runs VX3_Voxel::force() in its timeStep (VX3_Voxel.cu:162-176): not of a Fixed
// material, not fixed in all DOFs by a boundary condition.  force() clears the voxel's
// contactForce (VX3_Voxel.cu:373-374); on those two kinds of voxel the contacts add up over the
// steps.  (A removed voxel, also flagged VF_FIXED, has no contacts and reports none.)
__device__ __forceinline__ bool runs_force(const Dev &d, int bcs, int v, uint32_t vflags) {
    if ((vflags & VF_FIXED) && d.vmat[vflags >> 8].fixed) return false;
    if (bcs && d.vext[v] >= 0 && d.ext[d.vext[v]].dof == EXT_ALL) return false;
    return true;
}

// Mixed-precision link state, in the 36 bytes per link of nine floats: a 16-byte row
// {pos2.x, pos2.y, pos2.z, angle2v.x} per link, an 8-byte row {angle2v.y, angle2v.z} per
// link, then angle1v's three components, component-major (read and written only for
// links in the large-angle branch)
__device__ __forceinline__ float4 *mixed_lstate_a(const Dev &d) { return reinterpret_cast<float4 *>(d.lstate); }
__device__ __forceinline__ float2 *mixed_lstate_b(const Dev &d) {
    return reinterpret_cast<float2 *>(reinterpret_cast<float4 *>(d.lstate) + d.nl);
}
__device__ __forceinline__ float *mixed_lstate_c(const Dev &d) {
    return reinterpret_cast<float *>(reinterpret_cast<float2 *>(reinterpret_cast<float4 *>(d.lstate) + d.nl) + d.nl);
}

// Mixed-precision slots: the slot of (direction dir, voxel v) is split into a 16-byte row
// {force x, y, z, moment x} and an 8-byte row {moment y, z}: six 16-byte rows per voxel
// direction-major, then six 8-byte rows, in the same 24 bytes per slot as Slot<float>,
// so that the link pass stores and the voxel pass loads each slot with two wide accesses
__device__ __forceinline__ void store_slot_mx(const Dev &d, int dir, int v, V3<float> f, V3<float> m) {
    const size_t i = (size_t)dir * d.nv + v;
    reinterpret_cast<float4 *>(d.slots)[i] = make_float4(f.x, f.y, f.z, m.x);
    reinterpret_cast<float2 *>(reinterpret_cast<float4 *>(d.slots) + 6 * (size_t)d.nv)[i] = make_float2(m.y, m.z);
}
__device__ __forceinline__ void load_slot_mx(const Dev &d, int dir, int v, V3<float> *f, V3<float> *m) {
    const size_t i = (size_t)dir * d.nv + v;
    const float4 a = reinterpret_cast<const float4 *>(d.slots)[i];
    const float2 b = reinterpret_cast<const float2 *>(reinterpret_cast<const float4 *>(d.slots) + 6 * (size_t)d.nv)[i];
    *f = V3<float>{a.x, a.y, a.z};
    *m = V3<float>{a.w, b.x, b.y};
}

template <class R> __device__ __forceinline__ void store_slot(Slot<R> *s, V3<R> f, V3<R> m) {
    Slot<R> o;
    o.f[0] = f.x; o.f[1] = f.y; o.f[2] = f.z;
    o.m[0] = m.x; o.m[1] = m.y; o.m[2] = m.z;
    *s = o;
}

// VX3_MathTree::eval (src/Utils/VX3_MathTree.h:50-191): the token program is read in
// order; each token's result is appended to a value queue and operators consume the
// oldest unconsumed values (binary: values[pc + 1] op values[pc]).  Programs are
// validated when the context is created (known operators, the consumption cursor
// never passes the append cursor, mtEND within VX3G_MAX_MATH_TOKENS with exactly one
// value left), so the queue indices stay in bounds.  Variables hit, angle,
// targetCloseness and numClosePairs are 0 (the validated programs read none but hit,
// which the reference never changes from 0).
constexpr int kMaxMathTokens = 256;
#if !defined(__CUDACC__)
// host builds of this header (the host-compiled adjoint checks): Phi(x) = erfc(-x/sqrt 2)/2
inline double normcdf(double x) { return 0.5 * std::erfc(-x / std::sqrt(2.0)); }
#endif

__device__ inline double math_eval(const MathTok *tok, double x, double y, double z, double t, double num_voxel) {
    double vals[kMaxMathTokens];
    int vc = 0, pc = 0;
    for (int i = 0; i < kMaxMathTokens; i++) {
        const MathTok k = tok[i];
        double r;
        switch (k.op) {
            case 0: return vals[pc < vc ? pc : 0];  // mtEND
            case 1: r = k.value; break;
            case 2: r = 2.71828182845904523536; break;
            case 3: r = 3.14159265358979323846; break;
            case 4: {
                const double w = k.value;
                r = w < 0.5 ? x : w < 1.5 ? y : w < 2.5 ? z : (w >= 3.5 && w < 4.5) ? t : (w >= 7.5 && w < 8.5) ? num_voxel : 0.0;
                break;
            }
            case 5: r = vals[pc + 1] + vals[pc]; pc += 2; break;
            case 6: r = vals[pc + 1] - vals[pc]; pc += 2; break;
            case 7: r = vals[pc + 1] * vals[pc]; pc += 2; break;
            case 8: r = vals[pc + 1] / vals[pc]; pc += 2; break;
            case 9: r = pow(vals[pc + 1], vals[pc]); pc += 2; break;
            case 10: r = sqrt(vals[pc]); pc++; break;
            case 11: r = sin(vals[pc]); pc++; break;
            case 12: r = cos(vals[pc]); pc++; break;
            case 13: r = tan(vals[pc]); pc++; break;
            case 14: r = atan(vals[pc]); pc++; break;
            case 15: r = log(vals[pc]); pc++; break;
            case 16: r = rint(vals[pc]); pc++; break;
            case 17: r = fabs(vals[pc]); pc++; break;
            case 18: r = !vals[pc]; pc++; break;
            case 19: r = vals[pc + 1] > vals[pc]; pc += 2; break;
            case 20: r = vals[pc + 1] < vals[pc]; pc += 2; break;
            case 21: r = vals[pc + 1] && vals[pc]; pc += 2; break;
            case 22: r = vals[pc + 1] || vals[pc]; pc += 2; break;
            case 23: r = normcdf(vals[pc]); pc++; break;
            default: return 0.0;
        }
        vals[vc++] = r;
    }
    return 0.0;
}

// v has a link to u (is_neighbor depth 1, VX3_VoxelyzeKernel.cu:651-680) in the current link
// table: robots whose links can be made at runtime keep each face's partner in Dev::vnb
__device__ __forceinline__ bool linked_to(const Dev &d, int v, int u) {
    const uint32_t m = d.vinfo[v].y & VF_LINKMASK;
    for (int k = 0; k < 6; k++)
        if (((m >> k) & 1u) && d.vnb[6 * (size_t)v + k] == u) return true;
    return false;
}

// the force field of robot rp at position (x, y, z) and time t (VX3_Voxel.cu:178-184)
__device__ inline V3<double> force_field(const Dev &d, const RobotP &rp, double x, double y, double z, double t) {
    const double nv = (double)rp.nv;
    return V3<double>{rp.ff[0] >= 0 ? math_eval(d.ftok + rp.ff[0], x, y, z, t, nv) : 0.0,
                      rp.ff[1] >= 0 ? math_eval(d.ftok + rp.ff[1], x, y, z, t, nv) : 0.0,
                      rp.ff[2] >= 0 ? math_eval(d.ftok + rp.ff[2], x, y, z, t, nv) : 0.0};
}

#if defined(__CUDACC__)
// robot r's lists are rebuilt this step; the first voxel to say so puts a robot of the
// shared-memory path on the work list of coll_list_robots
__device__ __forceinline__ void flag_robot(const Dev &d, int r) {
    if (*(volatile int *)&d.cflag[1 + r]) return;
    if (atomicOr(&d.cflag[1 + r], 1) != 0) return;
    atomicOr(d.cflag, 1);
    const int k = d.rp[r].lchunks;
    if (k) {
        const unsigned long long old = atomicAdd(d.lwork_ctr, (1ull << 32) | (unsigned long long)k);
        if ((old >> 32) < (unsigned long long)d.nr) d.lwork[old >> 32] = make_int2(r, (int)(old & 0xffffffffull));
    }
}

// mixed precision: voxel v's contact record (Dev::crec) from its position pair, momentum (hi) and
// material; each rounding on its own in either unit
__device__ __forceinline__ void contact_record(const Dev &d, int v, float4 h, float4 l, float4 lm, float mass_inv, float pstiff,
                                               float c_col) {
    float4 *R = d.crec + 2 * (size_t)v;
    R[0] = make_float4(h.x, h.y, h.z, __fadd_rn(h.w, l.w));
    R[1] = make_float4(l.x, l.y, l.z, pstiff);
    d.crec[2 * (size_t)d.nv + v] = make_float4(__fmul_rn(lm.x, mass_inv), __fmul_rn(lm.y, mass_inv), __fmul_rn(lm.z, mass_inv), c_col);
}

#endif

// ------------------------------------------------------------- link material models
// VX3_Material::stress (src/VX3/VX3_Material.cu:90-124) of link material m at strain eps:
// zero past failure; the linear law for linear models, in compression and on the first
// segment (or when forced); else the segment of the data points holding eps (the last
// one extrapolated), with the volumetric variant when Poisson's ratio is on.  The data
// points are read only on a non-linear segment.
__device__ __forceinline__ float model_stress(const LMat &m, const float2 *pts, float eps, float tss, bool force_linear) {
    if (m.eps_fail != -1.0f && eps > m.eps_fail) return 0.0f;
    if (m.lin || force_linear || eps <= pts[1].x) {
        if (m.nu == 0.0f) return m.E * eps;
        return m.eHat * ((1 - m.nu) * eps + m.nu * tss);
    }
    for (int i = 2; i < m.ssn; i++) {
        const float2 a = pts[i - 1], b = pts[i];
        if (eps <= b.x || i == m.ssn - 1) {
            const float perc = (eps - a.x) / (b.x - a.x);
            const float basic = a.y + perc * (b.y - a.y);
            if (m.nu == 0.0f) return basic;
            const float modulus = (b.y - a.y) / (b.x - a.x);
            const float mod_hat = modulus / ((1 - 2 * m.nu) * (1 + m.nu));
            const float eff = basic / modulus;  // strain where the segment's line from 0 reaches the stress
            const float eff_tss = tss * (eff / eps);
            return mod_hat * ((1 - m.nu) * eff + m.nu * eff_tss);
        }
    }
    return 0.0f;
}

// VX3_Link::updateStrain (src/VX3/VX3_Link.cu:220-260): the link's stress at axial strain
// eps, with maxStrain (*max_strain) and, for non-linear materials, the plastic
// strainOffset (d.soff[l]): on new ground the curve is followed and the offset of the
// unloading line recorded; below the largest strain reached the material unloads
// linearly from that offset.
__device__ __forceinline__ float link_stress(const Dev &d, const LMat &m, int l, float eps, float *max_strain) {
    if (m.lin) {
        if (eps > *max_strain) *max_strain = eps;
        return model_stress(m, nullptr, eps, m.tss, false);
    }
    const float2 *pts = d.ss + m.sso;
    if (eps > *max_strain) {
        *max_strain = eps;
        const float st = model_stress(m, pts, eps, m.tss, false);
        d.soff[l] = m.nu != 0.0f ? *max_strain - model_stress(m, pts, eps, 0.0f, false) / (m.eHat * (1 - m.nu))
                                 : *max_strain - st / m.E;
        return st;
    }
    const float rel = eps - d.soff[l];
    return m.nu != 0.0f ? model_stress(m, pts, rel, m.tss, true) : m.E * rel;
}

// ------------------------------------------------------------- link pass
// isNewLink (VX3_Link.cu:206-213): a runtime link's forces and moments, just stored, are
// scaled by 0.01 for its first SafetyGuard updates (the product of the stored value is the
// product the reference forms before storing).  The slots are read back through volatile
// pointers, so the common path's values need not stay live across this rare branch.
template <class R> __device__ __forceinline__ void new_link_scale(const Dev &d, int l, Slot<R> *sNeg, Slot<R> *sPos) {
    const int n = d.lnew[l];
    if (n == 0) return;
    const R k = (R)0.01;
    volatile R *a = reinterpret_cast<volatile R *>(sNeg), *b = reinterpret_cast<volatile R *>(sPos);
    for (int c = 0; c < 6; c++) {
        a[c] = a[c] * k;
        b[c] = b[c] * k;
    }
    d.lnew[l] = n - 1;
}

// the same for a runtime link's two mixed-precision slots (negative end: direction dneg)
__device__ __forceinline__ void new_link_scale_mx(const Dev &d, int l, int dneg, int vneg, int vpos) {
    const int n = d.lnew[l];
    if (n == 0) return;
    for (int e = 0; e < 2; e++) {
        const size_t i = (size_t)(dneg + e) * d.nv + (e ? vpos : vneg);
        volatile float *a = reinterpret_cast<volatile float *>(reinterpret_cast<float4 *>(d.slots) + i);
        volatile float *b =
            reinterpret_cast<volatile float *>(reinterpret_cast<float2 *>(reinterpret_cast<float4 *>(d.slots) + 6 * (size_t)d.nv) + i);
        for (int c = 0; c < 4; c++) a[c] = a[c] * 0.01f;
        for (int c = 0; c < 2; c++) b[c] = b[c] * 0.01f;
    }
    d.lnew[l] = n - 1;
}

// the constants of a link in FP64, from the damping numerators of its ends (VX3_Voxel::
// dampingMultiplier, VX3_Voxel.h:206-208: previousDt is the robot's dt once a voxel has stepped,
// 0 for fixed voxels, which never step)
__device__ __forceinline__ LMatD make_lmatd(const LMat &m, float dmcN, float dmcP, bool fixN, bool fixP, float dtf) {
    LMatD c;
    c.b1 = widen(m.b1), c.b2 = widen(m.b2), c.b3 = widen(m.b3), c.a2 = widen(m.a2);
    c.sqA1 = widen(m.sqA1), c.sqB1 = widen(m.sqB1), c.sqA2 = widen(m.sqA2xIp), c.sqB2 = widen(m.sqB2xFMp);
    c.sqB3 = widen(m.sqB3xIp);
    const float dmN = dmcN / (fixN ? 0.0f : dtf), dmP = dmcP / (fixP ? 0.0f : dtf);
    c.kN = 0.5 * widen(dmN), c.kP = 0.5 * widen(dmP);
    c.jN = 0.5 * c.kN, c.jP = 0.5 * c.kP;
    c.same = dmN == dmP ? 1 : 0;
    return c;
}
__device__ __forceinline__ LMatD link_consts(const Dev &d, uint32_t i, int2 e, float dtf) {
    if (d.lmatd) return d.lmatd[i];
    const uint32_t fn = d.vinfo[e.x].y, fp = d.vinfo[e.y].y;
    return make_lmatd(d.lmat[i], d.vmat[fn >> 8].dmc, d.vmat[fp >> 8].dmc, fn & VF_FIXED, fp & VF_FIXED, dtf);
}

// the hysteresis of orientLink (VX3_Link.cu:107-125) on pos2 before the rest length is taken off:
// SmallTurn = (|z| + |y|)/x, ExtendPerc = |1 - x/rest|.  Decided in FP32 on the truncated
// magnitudes where they are clear of the thresholds by more than the truncation (2^-20), else
// with the reference's divisions
__device__ __forceinline__ void turn_state(V3<double> pos2, double rest, bool &small, bool &lvv) {
    const float X = mag(pos2.x), T = mag(pos2.y) + mag(pos2.z), R = mag(rest);
    const bool ahead = hi_word(pos2.x) > 0;
    if (small) {
        if (ahead && T < 0.05999f * X && X > 0.401f * R && X < 1.599f * R) return;  // stays small
    } else if (ahead && T > 0.05001f * X) {
        return;  // stays large
    }
    const float SmallTurn = (float)((fabs(pos2.z) + fabs(pos2.y)) / pos2.x);
    const float ExtendPerc = (float)(fabs(1 - pos2.x / rest));
    const float HF = 1.2f, BEND = 0.05f, EXT = 0.50f;
    if (!small && SmallTurn < BEND && ExtendPerc < EXT) {
        small = true;
        lvv = false;
    } else if (small && (SmallTurn > HF * BEND || ExtendPerc > HF * EXT)) {
        small = false;
        lvv = false;
    }
}

// The elastic and damping forces and moments of a link in its own frame (VX3_Link::updateForces,
// VX3_Link.cu:150-204).  Factors 1/2 and 2 are moved through products, which is exact; a link
// that is and was in the small-angle branch (a1v and oldA1 zero) leaves out the terms that are zero;
// ends with equal damping have opposite forces.
struct LinkForces {
    V3<double> fNeg, fPos, mNeg, mPos;
};
__device__ __forceinline__ LinkForces link_forces(const LMatD &c, float axial, bool lvv, bool bent, V3<double> pos2,
                                                  V3<double> oldPos2, V3<double> a1v, V3<double> oldA1, V3<double> a2v,
                                                  V3<double> oldA2) {
    LinkForces o;
    const double t1 = c.b2 * pos2.z, t3 = c.b2 * pos2.y;
    const V3<double> D = sub(pos2, oldPos2), E2 = sub(a2v, oldA2);  // twice dPos2, dAngle2
    const double fx = widen(axial);
    V3<double> P, U, W;  // twice the reference's posCalc and the moments' damping vectors at the two ends
    if (!bent) {
        const double t2 = c.b3 * a2v.y, t4 = c.b3 * a2v.z, u2 = c.sqB3 * E2.y, u4 = c.sqB3 * E2.z;
        const double u1 = c.sqB2 * D.z, u3 = c.sqB2 * D.y;
        o.fNeg = V3<double>{fx, c.b1 * pos2.y - c.b2 * a2v.z, c.b1 * pos2.z + c.b2 * a2v.y};
        o.mNeg = V3<double>{c.a2 * a2v.x, -t1 - t2, t3 - t4};
        o.mPos = V3<double>{-o.mNeg.x, fma(-2.0, t2, -t1), fma(-2.0, t4, t3)};
        P = V3<double>{c.sqA1 * D.x, c.sqB1 * D.y - c.sqB2 * E2.z, c.sqB1 * D.z + c.sqB2 * E2.y};
        const double ux = c.sqA2 * E2.x;
        U = V3<double>{-ux, u1 + u2, u4 - u3};
        W = V3<double>{ux, fma(2.0, u2, u1), fma(2.0, u4, -u3)};
    } else {
        const V3<double> E1 = sub(a1v, oldA1);
        o.fNeg = V3<double>{fx, c.b1 * pos2.y - c.b2 * (a1v.z + a2v.z), c.b1 * pos2.z + c.b2 * (a1v.y + a2v.y)};
        o.mNeg = V3<double>{c.a2 * (a2v.x - a1v.x), -t1 - c.b3 * (2 * a1v.y + a2v.y), t3 - c.b3 * (2 * a1v.z + a2v.z)};
        o.mPos = V3<double>{-o.mNeg.x, -t1 - c.b3 * (a1v.y + 2 * a2v.y), t3 - c.b3 * (a1v.z + 2 * a2v.z)};
        P = V3<double>{c.sqA1 * D.x, c.sqB1 * D.y - c.sqB2 * (E1.z + E2.z), c.sqB1 * D.z + c.sqB2 * (E1.y + E2.y)};
        const double ux = c.sqA2 * (E2.x - E1.x);
        U = V3<double>{-ux, c.sqB2 * D.z + c.sqB3 * (2 * E1.y + E2.y), c.sqB3 * (2 * E1.z + E2.z) - c.sqB2 * D.y};
        W = V3<double>{ux, c.sqB2 * D.z + c.sqB3 * (E1.y + 2 * E2.y), c.sqB3 * (E1.z + 2 * E2.z) - c.sqB2 * D.y};
    }
    if (!lvv) {
        o.fPos = neg(o.fNeg);
        return o;
    }
    if (c.same) {
        o.fNeg = add(o.fNeg, scl(P, c.kN));
        o.fPos = neg(o.fNeg);
    } else {
        o.fPos = neg(add(o.fNeg, scl(P, c.kP)));
        o.fNeg = add(o.fNeg, scl(P, c.kN));
    }
    o.mNeg = sub(o.mNeg, scl(U, c.jN));
    o.mPos = sub(o.mPos, scl(W, c.jP));
    return o;
}

template <class R> __device__ __forceinline__ void link_update(const Dev &d, int l) {
    static_assert(std::is_same<R, double>::value, "the FP64 step");
    const uint2 li = d.linfo[l];
    const int r = (int)li.x;
    if (d.status[r] != 0) return;
    uint32_t fl = li.y;
    if (fl & (LF_BOTH_FIXED | LF_GONE)) return;  // gpu_update_links skips both-fixed and detached links
    const int axis = fl & LF_AXIS;
    const int2 e = d.ends[l];
    const double4 pn = d.pos[e.x], pp = d.pos[e.y];
    const double4 qn = d.quat[e.x], qp = d.quat[e.y];
    const double rest = 0.5 * (pn.w + pp.w);  // VX3_Link::updateRestLength (VX3_Link.cu:80-83)
    const LMat &m = d.lmat[fl >> 8];
    R *ls = (R *)d.lstate;
    const size_t NL = (size_t)d.nl;
    const V3<R> oldPos2{ls[l], ls[NL + l], ls[2 * NL + l]};
    const V3<R> oldA1{ls[3 * NL + l], ls[4 * NL + l], ls[5 * NL + l]};
    const V3<R> oldA2{ls[6 * NL + l], ls[7 * NL + l], ls[8 * NL + l]};

    // orientLink (VX3_Link.cu:90-133)
    V3<R> pos2 = to_axis_x(axis, V3<R>{pp.x - pn.x, pp.y - pn.y, pp.z - pn.z});
    Q4<R> angle1 = to_axis_xq(axis, Q4<R>{qn.x, qn.y, qn.z, qn.w});
    Q4<R> angle2 = to_axis_xq(axis, Q4<R>{qp.x, qp.y, qp.z, qp.w});
    const Q4<R> tot = qconj(angle1);
    pos2 = qrot(tot, pos2);
    angle2 = qmul(tot, angle2);
    angle1 = Q4<R>{1, 0, 0, 0};
    bool small = (fl & LF_SMALL) != 0, lvv = (fl & LF_LVV) != 0;
    turn_state(pos2, rest, small, lvv);
    V3<R> a1v{0, 0, 0};
    if (small) {
        pos2.x -= rest;
    } else {
        const R l2 = len(pos2);
        angle1 = from_angle_to_posx(angle1, pos2, l2);
        angle2 = qmul_x0(angle1, angle2);
        pos2 = V3<R>{l2 - rest, 0, 0};
        a1v = to_rotvec(angle1);
    }
    const V3<R> a2v = to_rotvec(angle2);
    ls[l] = pos2.x; ls[NL + l] = pos2.y; ls[2 * NL + l] = pos2.z;
    bool bent = !small || !is_zero(oldA1);
    if (bent) {
        ls[3 * NL + l] = a1v.x; ls[4 * NL + l] = a1v.y; ls[5 * NL + l] = a1v.z;
    }
    ls[6 * NL + l] = a2v.x; ls[7 * NL + l] = a2v.y; ls[8 * NL + l] = a2v.z;

#if defined(__CUDA_ARCH__)
    // a warp with a bent link takes the terms of a bent link for all (zeros add nothing): one of the two
    // forms instead of both in turn
    bent = __any_sync(__activemask(), bent);
#endif

    // updateForces (VX3_Link.cu:135-218) + updateStrain (:220-260)
    const float axialStrain = (float)(pos2.x / rest);
    float2 sm = d.strain[l];
    sm.x = axialStrain;
    const float stress = link_stress(d, m, l, axialStrain, &sm.y);
    d.strain[l] = sm;
    if (axialStrain > 100) atomicOr(&d.status[r], 1);  // divergence (VX3_VoxelyzeKernel.cu:271-281)

    Slot<R> *S = (Slot<R> *)d.slots;
    Slot<R> *sNeg = &S[(size_t)(2 * axis) * d.nv + e.x];
    Slot<R> *sPos = &S[(size_t)(2 * axis + 1) * d.nv + e.y];
    uint32_t nfl = (fl & ~(LF_SMALL | LF_LVV)) | (small ? LF_SMALL : 0u);
    if (m.eps_fail != -1.0f && sm.y > m.eps_fail) {  // isFailed: forces zero (lvv unchanged)
        const V3<R> z{0, 0, 0};
        store_slot(sNeg, z, z);
        store_slot(sPos, z, z);
        nfl |= lvv ? LF_LVV : 0u;
        if (nfl != fl) d.linfo[l].y = nfl;
        return;
    }
    LinkForces f = link_forces(link_consts(d, fl >> 8, e, d.dt[r]), stress * m.area, lvv, bent, pos2, oldPos2, a1v, oldA1,
                               a2v, oldA2);
    nfl |= LF_LVV;
    if (!small) {
        f.fNeg = qrotinv_x0(angle1, f.fNeg);
        f.mNeg = qrotinv_x0(angle1, f.mNeg);
    }
    f.fPos = qrotinv(angle2, f.fPos);
    f.mPos = qrotinv(angle2, f.mPos);
    store_slot(sNeg, to_axis_original(axis, f.fNeg), to_axis_original(axis, f.mNeg));
    store_slot(sPos, to_axis_original(axis, f.fPos), to_axis_original(axis, f.mPos));
    if (fl & LF_RUNTIME) new_link_scale(d, l, sNeg, sPos);
    if (nfl != fl) d.linfo[l].y = nfl;
}

// ------------------------------------------------------------ voxel pass
// Temperature of a voxel at time t (gpu_update_temperature, VX3_VoxelyzeKernel.cu:625-650)
// returned as the base size nomSize*(1+T*cte) (VX3_Voxel::baseSize); tempe gets T.
template <bool EXACT = true>
__device__ __forceinline__ double temperature_base_size(const RobotP &rp, const VMat &m, double phase, double t,
                                                        double cur_bs, float *tempe) {
    static_assert(EXACT, "the FP64 step");
    if (!(rp.vary_temp && rp.temp_period > 0)) return cur_bs;
    if (m.thermal_on_after > t || m.fixed) return cur_bs;
    double T = rp.temp_amp * sin(2 * 3.1415926f * (t / rp.temp_period + phase));
    if (!rp.expansion && T > 0) T = 0;
    const float tf = (float)T;
    *tempe = tf;
    return m.nom_size * (1 + tf * m.cte);
}

// sine and cosine of the actuation argument 2*3.1415926f*t/P of a robot at its next step's time,
// with that time and a bound on what the two ways to the temperature differ by: an argument of
// up to 2 pi (t/P + 2) carries six roundings of itself between them
__device__ __forceinline__ void actuation_phase(const Dev &d, int r, int parity, double t) {
    const RobotP &rp = d.rp[r];
    const double c = t / rp.temp_period, a = 2 * 3.1415926f * c;
    double s, k;
    sincos(a, &s, &k);
    d.act[(size_t)parity * d.nr + r] = make_double4(s, k, fabs(rp.temp_amp) * 5e-15 * (fabs(c) + 4.0), t);
}

// The same temperature from the robot's sine and cosine and the voxel's own (of its phase), by
// the addition theorem: 3 FP64 instructions instead of a division and a sine (about 45).  The
// reference keeps T in 32 bits; T here is within act.z of its value, so where no rounding
// boundary of FP32 (nor zero, the clamp) lies that near, the stored float is the reference's.
// Elsewhere (about one voxel in 10^7) the reference's expression decides.
__device__ __forceinline__ double next_base_size(const Dev &d, const RobotP &rp, const VMat &m, int v, int r, int parity,
                                                 double t, double cur_bs, float *tempe) {
    if (m.toa_pos && m.thermal_on_after > t) return cur_bs;
    if (d.act) {
        const double4 a = d.act[(size_t)parity * d.nr + r];
        if (hi_word(a.w) == hi_word(t) && a.w == t) {
            const double2 p = d.actv[v];
            const double T = rp.temp_amp * fma(a.x, p.y, a.y * p.x);
            const float lo = (float)(T - a.z), up = (float)(T + a.z);
            if (!rp.expansion && lo > 0) {
                *tempe = 0;
                return m.nom_size;
            }
            if (lo == up) {
                *tempe = lo;
                return m.nom_size * widen(1 + lo * m.cte);
            }
        }
    }
    return temperature_base_size(rp, m, d.phase[v], t, cur_bs, tempe);
}

// sine and cosine of a voxel's phase term; NaN (the reference's expression decides every step)
// for phases beyond two cycles, outside the bound above
__device__ __forceinline__ double2 actuation_voxel(double phase) {
    double s = NAN, k = NAN;
    if (fabs(phase) <= 2.0) sincos(2 * 3.1415926f * phase, &s, &k);
    return make_double2(s, k);
}

// the voxel is clear of the floor: baseSize/2 - nomSize/2 - z < 0, with a margin of several of the
// FP32 magnitudes' truncations (floorPenetration, VX3_Voxel.h:185-188)
__device__ __forceinline__ bool above_floor(double bs, double nom, double z) {
    const float b = mag(bs), zf = signed_mag(z);
    return zf > 0.5f * (b - mag(nom)) + 4e-6f * (b + fabsf(zf));
}
__device__ __forceinline__ float floor_penetration(double bs, double nom, double z) {
    const double bsa = (bs + bs + bs) / 3.0f;  // baseSizeAverage (VX3_Voxel.h:102-105)
    return (float)(bsa / 2 - nom / 2 - z);
}

template <class R> __device__ __forceinline__ void voxel_update(const Dev &d, int v, int parity) {
    static_assert(std::is_same<R, double>::value, "the FP64 step");
    const uint2 vi = d.vinfo[v];
    const int r = (int)vi.x;
    const RobotP &rp = d.rp[r];
    const double Tcur = d.T[(size_t)parity * d.nr + r];
    const int st = d.status[r];
    const float dtf = d.dt[r];
    const double dt = widen(dtf), tn = Tcur + dt;
    if (v == rp.voff) d.T[(size_t)(parity ^ 1) * d.nr + r] = (st == 0) ? tn : Tcur;  // currentTime += dt
    if (st != 0) {
        // the backward pass's recompute: a robot that stopped in this step did not take it, and has no
        // sums here.  The stored state was copied before; from now on it too says that the robot is stopped.
        if (d.fsum && v == rp.voff) d.fstat[r] = st;
        return;
    }
    uint32_t fl = vi.y;
    if (fl & VF_FIXED) return;
    const VMat &m = d.vmat[fl >> 8];
    double4 p = d.pos[v];

    const bool actuated = rp.vary_temp && rp.temp_period > 0;
    float *tcur = d.tempe + (size_t)parity * d.nv, *tnext = d.tempe + (size_t)(parity ^ 1) * d.nv;
    if (dtf == 0.0f) {  // VX3_Voxel::timeStep returns before moving; temperature still follows time
        if (actuated) {
            float te = tcur[v];
            p.w = temperature_base_size(rp, m, d.phase[v], tn, p.w, &te);
            d.pos[v] = p;
            tnext[v] = te;
        }
        return;
    }

    // boundary-condition external (VX3_External), if any
    const int xi = rp.bcs ? d.vext[v] : -1;
    ExtBC ex{};
    if (xi >= 0) ex = d.ext[xi];
    const int dof = ex.dof;
    if (dof == EXT_ALL) {  // isFixedAll (VX3_Voxel.cu:167-173): at its prescribed pose, motion halted
        const short4 l = d.ijk[v];
        p.x = l.x * m.nom_size + ex.t.x;
        p.y = l.y * m.nom_size + ex.t.y;
        p.z = l.z * m.nom_size + ex.t.z;
        d.quat[v] = ex.q;
        d.linmom[v] = make_double4(0, 0, 0, 0);
        d.angmom[v] = make_double4(0, 0, 0, 0);
        if (actuated) {
            float te = tcur[v];
            p.w = next_base_size(d, rp, m, v, r, parity, tn, p.w, &te);
            tnext[v] = te;
        }
        d.pos[v] = p;
        return;
    }
    const double4 q = d.quat[v];
    const double4 lm = d.linmom[v];
    const double4 am = d.angmom[v];

    // link force/moment sums in direction order 0..5 (VX3_Voxel::force/moment, VX3_Voxel.cu:350-397)
    V3<R> Fs{0, 0, 0}, Ms{0, 0, 0};
    const Slot<R> *S = (const Slot<R> *)d.slots;
#pragma unroll
    for (int dir = 0; dir < 6; dir++) {
        if (fl & (1u << dir)) {
            const Slot<R> s = S[(size_t)dir * d.nv + v];
            const V3<R> f{s.f[0], s.f[1], s.f[2]}, n{s.m[0], s.m[1], s.m[2]};
            Fs = dir ? add(Fs, f) : f;
            Ms = dir ? add(Ms, n) : n;
        }
    }
    if (d.fsum) {  // the backward pass's recompute keeps them (Snap::fsum)
        const size_t nv = d.nv;
        double *f = d.fsum + v;
        f[0] = Fs.x, f[nv] = Fs.y, f[2 * nv] = Fs.z;
        f[3 * nv] = Ms.x, f[4 * nv] = Ms.y, f[5 * nv] = Ms.z;
        if (rp.collision) {
            const double4 c = d.contact[v];
            f[6 * nv] = c.x, f[7 * nv] = c.y, f[8 * nv] = c.z;
        }
    }
    bool stat = (fl & VF_STATIC) != 0;
    const bool floorOn = rp.floor != 0;
    const double bs = p.w;
    V3<double> lmv{lm.x, lm.y, lm.z}, amv{am.x, am.y, am.z};
    const double mass_inv = widen(m.mass_inv), mom_inv = widen(m.mom_inv);
    // the floor is off, or the voxel clear of it: no floor force, and the penetration is not needed
    const bool off = !floorOn || above_floor(bs, m.nom_size, p.z);
    const float pen = off ? -1.0f : floor_penetration(bs, m.nom_size, p.z);  // before the position update

    const Q4<double> o{q.x, q.y, q.z, q.w};
    V3<double> F = qrot(o, Fs);
    if (xi >= 0) F = add(F, V3<double>{ex.f[0], ex.f[1], ex.f[2]});  // external force (:363-364)
    if (m.c_glob != 0.0f) F = sub(F, scl(scl(lmv, mass_inv), m.c_glob));
    F.z += widen(m.grav_force);
    if (rp.collision) {
        const double4 c = d.contact[v];
        F = sub(F, V3<double>{c.x, c.y, c.z});
    }
    if (rp.cilia) {  // CiliaForce * Cilia (VX3_Voxel.cu:376), from k_extra_forces
        const double4 c = d.cfv[v];
        F = add(F, V3<double>{c.x, c.y, c.z});
    }
    if (rp.ff_any) {  // force field (VX3_Voxel.cu:178-184), evaluated by k_extra_forces
        const double4 ff = d.ffv[v];
        F.x += ff.x;
        F.y += ff.y;
        F.z += ff.z;
    }
    V3<double> fric{0, 0, 0};
    if (pen >= 0) {  // floorForce (VX3_Voxel.cu:399-426)
        fric = F;
        const V3<double> vel = scl(lmv, mass_inv);
        const float normal = m.pstiff * pen;
        F.z += normal - m.c_col * vel.z;
        if (stat) {
            const float surf = (float)(F.x * F.x + F.y * F.y);
            const float fr = (m.mu_s * normal) * (m.mu_s * normal);
            if (surf > fr) stat = false;
        } else {
            F = sub(F, scl(normalized(V3<double>{vel.x, vel.y, 0}), m.mu_k * normal));
        }
        fric = sub(F, fric);
    } else if (floorOn) {
        stat = false;
    }
    lmv = add(lmv, scl(F, dt));
    V3<double> tr = scl(lmv, dt * mass_inv);
    if (pen >= 0) {
        const double work = fric.x * tr.x + fric.y * tr.y;
        const double hKe = 0.5 * m.mass_inv * (lmv.x * lmv.x + lmv.y * lmv.y);
        if (hKe + work <= 0) stat = true;
        if (stat) {
            lmv.x = lmv.y = 0;
            tr.x = tr.y = 0;
        }
    } else {
        stat = false;
    }
    p.x += tr.x; p.y += tr.y; p.z += tr.z;
    V3<double> M = qrot(o, Ms);
    if (xi >= 0) M = add(M, V3<double>{ex.m[0], ex.m[1], ex.m[2]});  // external moment (:393-394)
    if (m.c_glob_rot != 0.0f) M = sub(M, scl(scl(amv, mom_inv), m.c_glob_rot));
    amv = add(amv, scl(M, dt));
    Q4<double> on = qmul(from_half_rotvec(scl(amv, 0.5 * (dt * mom_inv))), o);
    if (dof) {  // fixed DOFs (VX3_Voxel.cu:222-257)
        const short4 l = d.ijk[v];
        if (dof & 1) { p.x = l.x * m.nom_size + ex.t.x; lmv.x = 0; }
        if (dof & 2) { p.y = l.y * m.nom_size + ex.t.y; lmv.y = 0; }
        if (dof & 4) { p.z = l.z * m.nom_size + ex.t.z; lmv.z = 0; }
        if (dof & EXT_R) {
            if ((dof & EXT_R) == EXT_R) {  // all rotations: the prescribed orientation
                on = Q4<double>{ex.q.x, ex.q.y, ex.q.z, ex.q.w};
                amv = V3<double>{0, 0, 0};
            } else {  // some: zero those components of the rotation vector
                V3<double> rv = to_rotvec(on);
                if (dof & 8) { rv.x = 0; amv.x = 0; }
                if (dof & 16) { rv.y = 0; amv.y = 0; }
                if (dof & 32) { rv.z = 0; amv.z = 0; }
                on = from_rotvec(rv);
            }
        }
    }
    d.quat[v] = make_double4(on.w, on.x, on.y, on.z);
    // static friction freezes rotation (VX3_Voxel.cu:259-264), penetration after the move
    if (stat && !above_floor(bs, m.nom_size, p.z) && floor_penetration(bs, m.nom_size, p.z) >= 0) amv = V3<double>{0, 0, 0};

    // next step's temperature; tempe is double-buffered by step parity so that the
    // buffer of the step just taken keeps the value that step used (the reference's tempe)
    if (actuated) {
        float te = tcur[v];
        p.w = next_base_size(d, rp, m, v, r, parity, tn, bs, &te);
        tnext[v] = te;
    }
    d.pos[v] = p;
    d.linmom[v] = make_double4(lmv.x, lmv.y, lmv.z, 0.0);
    d.angmom[v] = make_double4(amv.x, amv.y, amv.z, 0.0);
    const uint32_t nfl = stat ? (fl | VF_STATIC) : (fl & ~VF_STATIC);
    if (nfl != fl) d.vinfo[v].y = nfl;
}

}  // namespace vx3g
