// vx3g_mixed.cu -- the mixed-precision step: FP32 link forces and moments,
// compensated FP32 (hi + lo float pairs, two-sum arithmetic) for positions,
// orientations and momenta.  No FP64 arithmetic runs per link or per voxel (the actuation
// phase is reduced in FP64 once per robot and step).  Quotients and square roots on the
// hot paths use the hardware reciprocal and reciprocal square root (__fdividef, rsqrtf:
// within 2 ulp), fixed instructions, so every compiled launch shape computes the same
// values; the FP64 step keeps the reference's correctly rounded operations.
//
// The link pass restates VX3_Link::orientLink/updateForces (src/VX3/VX3_Link.cu:90-218)
// without the cancellations FP32 would suffer:
//  * pos2 = R(conj(q1)) * toAxisX(pPos - pNeg) is formed as
//      L*R(conj(q1))e_x + R(conj(q1)) * toAxisX(delta),  delta = (pPos - pNeg) - L*e_axis,
//    with delta taken from the hi/lo pairs (exact differences of nearby values) and
//    R(q)e_x - e_x = (-2(y^2+z^2), 2(xy-wz), 2(xz+wy)) evaluated directly, so the axial
//    deviation pos2.x - L never subtracts two nearly equal FP32 numbers;
//  * angle2 = conj(q1)*q2 = |q1|^2 + conj(q1)*(q2 - q1), the difference again from the
//    hi/lo pairs; the rotation vector uses 2*atan2(|v|, w)/|v|.
// The voxel pass restates VX3_Voxel::timeStep (src/VX3/VX3_Voxel.cu:162-277) with the
// same sums in FP32 and every accumulation (p += F dt, x += p dt/m, L += M dt,
// q += (dq - 1) q) done as a two-sum into the hi/lo pair.
#include "vx3g_mixed_math.cuh"

namespace vx3g {

using mx::df_diff;

// ------------------------------------------------------------- collision narrow phase
// handle_collision_attachment + VX3_Collision::updateContactForce
// (src/VX3/VX3_VoxelyzeKernel.cu:682-727, src/VX3/VX3_Collision.cu:3-31) on the
// listed pairs, in FP32: the pair offset is taken from the hi/lo pairs (one rounding
// of an exact difference), the envelope test and the force in FP32, contacts summed
// in ascending partner order as the FP64 pass does.
// ATTACH: the batch has robots with EnableAttach (their pairs linked this step have their
// contact added, then taken back); the other instance carries none of that code
// candidates in flight per surface voxel: a 64^3 body's evaluation 11.7 us with one, 10.8 with two,
// 14.7 with four (registers against resident warps); 64 small robots' 7.4, 5.1, 4.9
constexpr int kEvalAhead = 2;
template <bool ATTACH> __global__ void __launch_bounds__(256) k_coll_eval_mixed(Dev d) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) {  // the rebuild (if any) is done; the next check starts clear
        *d.cflag = 0;
        *d.lwork_ctr = 0ull;
    }
    if (s >= d.ns) return;
    const int v = d.csurf[s];
    const int n = d.nnb[s];
    const int *lst = d.nbr + s;  // slot-major: entry k at lst[k*ns]
    const size_t ns = (size_t)d.ns;
    // kEvalAhead candidates at a time: their list entries, read one group ahead, then their
    // 32-byte sectors in flight together, so the chain of dependent loads is a fraction as long
    int un[kEvalAhead];
#pragma unroll
    for (int j = 0; j < kEvalAhead; j++) un[j] = j < n ? lst[j * ns] : v;
    const float4 *R = d.crec;  // contact records of this step (written by the displacement check)
    const uint2 vi = d.vinfo[v];
    const float4 pvH = R[2 * v], pvL = R[2 * v + 1];
    const int r = (int)vi.x;
    if (d.cflag[1 + r]) d.cflag[1 + r] = 0;
    // stopped robots and robots flagged before this step keep their contact forces; the
    // divergence bit is left out because the link pass, which may set it, runs beside
    // this kernel (a diverged robot never steps again, so its contacts feed nothing)
    if (d.status[r] & ~1) return;
    // pairs linked by this step's attachment: contact added, then taken back
    const bool att = ATTACH && d.rp[r].attach && d.acnt[r] > 0;
    V3<float> acc{0, 0, 0};
    if (!runs_force(d, d.rp[r].bcs, v, vi.y)) {  // its contactForce is never cleared: the pairs add to it
        const float4 c = reinterpret_cast<const float4 *>(d.contact)[v];
        acc = V3<float>{c.x, c.y, c.z};
    }
    if (n) {
        const float4 wv = R[2 * d.nv + v];
        const float bv = pvH.w;  // baseSizeAverage = baseSize (isotropic)
        for (int k = 0; k < n; k += kEvalAhead) {
            int uu[kEvalAhead];
            float4 hi[kEvalAhead], lo[kEvalAhead];
#pragma unroll
            for (int j = 0; j < kEvalAhead; j++) uu[j] = un[j];
#pragma unroll
            for (int j = 0; j < kEvalAhead; j++) hi[j] = R[2 * uu[j]], lo[j] = R[2 * uu[j] + 1];
#pragma unroll
            for (int j = 0; j < kEvalAhead; j++) un[j] = k + kEvalAhead + j < n ? lst[(k + kEvalAhead + j) * ns] : v;
#pragma unroll
            for (int j = 0; j < kEvalAhead; j++) {
                if (k + j >= n) break;
                const int u = uu[j];  // partner voxel, ascending
                const float4 puH = hi[j], puL = lo[j];
                // offset from the later surface voxel (voxel1) to the earlier one (voxel2)
                const float sg = u < v ? 1.0f : -1.0f;
                const float ox = mx::mul(sg, df_diff(puH.x, puL.x, pvH.x, pvL.x));
                const float oy = mx::mul(sg, df_diff(puH.y, puL.y, pvH.y, pvL.y));
                const float oz = mx::mul(sg, df_diff(puH.z, puL.z, pvH.z, pvL.z));
                const float bu = puH.w;
                const float wd = mx::mul(mx::plus(bv, bu), 0.625f);
                // |offset| and its reciprocal from one hardware reciprocal square root (coincident
                // voxels, d2 = 0, give dist = NaN and are skipped; the reference's force is NaN there)
                const float d2 = fmaf(oz, oz, mx::dot_a(ox, ox, oy, oy));
                const float inv = rsqrtf(d2);
                const float dist = mx::mul(d2, inv);
                if (!(dist <= wd)) continue;
                const float rel = mx::minus(wd, dist);
                if (!(rel > 0)) continue;
                const float4 wu = R[2 * d.nv + u];
                const float pstiff = __fdividef(mx::mul(mx::mul(2.0f, pvL.w), puL.w), mx::plus(pvL.w, puL.w));  // 2 / (1/a + 1/b)
                const float dampC = mx::mul(0.5f, mx::plus(wv.w, wu.w));
                const float ux = mx::mul(ox, inv), uy = mx::mul(oy, inv), uz = mx::mul(oz, inv);
                // voxel1 = the later one: rv = w1.u - w2.u with (1, 2) = (v, u) when u < v, else (u, v)
                const float rv = mx::mul(sg, mx::minus(fmaf(wv.z, uz, mx::dot_a(wv.x, ux, wv.y, uy)),
                                                       fmaf(wu.z, uz, mx::dot_a(wu.x, ux, wu.y, uy))));
                const float f = mx::dot_a(pstiff, rel, dampC, rv);
                // v.contactForce += force (v is voxel1) or -= force (v is voxel2); force along u
                if (ATTACH && att && linked_to(d, v, u)) {  // (acc + c) - c
                    const float cx = mx::mul(mx::mul(sg, ux), f), cy = mx::mul(mx::mul(sg, uy), f), cz = mx::mul(mx::mul(sg, uz), f);
                    acc = V3<float>{mx::minus(mx::plus(acc.x, cx), cx), mx::minus(mx::plus(acc.y, cy), cy),
                                    mx::minus(mx::plus(acc.z, cz), cz)};
                    continue;
                }
                acc.x = fmaf(mx::mul(sg, ux), f, acc.x);
                acc.y = fmaf(mx::mul(sg, uy), f, acc.y);
                acc.z = fmaf(mx::mul(sg, uz), f, acc.z);
            }
        }
    }
    reinterpret_cast<float4 *>(d.contact)[v] = make_float4(acc.x, acc.y, acc.z, 0.0f);
}

void launch_coll_eval_mixed(const Dev &d, cudaStream_t s) {
    if (!d.ns) return;
    if (d.narob) k_coll_eval_mixed<true><<<(d.ns + 255) / 256, 256, 0, s>>>(d);
    else k_coll_eval_mixed<false><<<(d.ns + 255) / 256, 256, 0, s>>>(d);
}

// ------------------------------------------------------------- programmatic dependent launch
// The link and voxel kernels are launched with programmatic stream serialization:
// a kernel may start while the previous one finishes.  Each first issues the loads
// that do not depend on the previous kernel, then waits for it to complete
// (griddepcontrol.wait: a no-op when launched without the attribute), and only then
// lets the next kernel launch, so a kernel never starts before the one two places
// earlier has finished.  Every store comes after the wait.
__device__ __forceinline__ void pdl_wait_then_release() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ------------------------------------------------------------- link pass
struct LinkOut {  // where the link pass leaves a link's update (mx::link_step)
    const Dev &d;
    int l, axis, r;
    int2 e;
    uint32_t fl;
    __device__ __forceinline__ void local(V3<float> pos2, V3<float> a1v, V3<float> a2v, bool small) {
        mixed_lstate_a(d)[l] = make_float4(pos2.x, pos2.y, pos2.z, a2v.x);
        mixed_lstate_b(d)[l] = make_float2(a2v.y, a2v.z);
        if (!(small && (fl & LF_SMALL))) {
            float *C = mixed_lstate_c(d);
            const size_t NL = (size_t)d.nl;
            C[l] = a1v.x, C[NL + l] = a1v.y, C[2 * NL + l] = a1v.z;
        }
    }
    __device__ __forceinline__ void strain(float2 s, bool torn) {
        d.strain[l] = s;
        if (torn) atomicOr(&d.status[r], 1);
    }
    __device__ __forceinline__ void neg(V3<float> f, V3<float> m) { store_slot_mx(d, 2 * axis, e.x, f, m); }
    __device__ __forceinline__ void pos(V3<float> f, V3<float> m) { store_slot_mx(d, 2 * axis + 1, e.y, f, m); }
    __device__ __forceinline__ void flags(uint32_t nfl, bool failed) {
        if ((fl & LF_RUNTIME) && !failed) new_link_scale_mx(d, l, 2 * axis, e.x, e.y);
        if (nfl != fl) d.linfo[l].y = nfl;
    }
};
template <bool HELD> __device__ __forceinline__ void links_mixed_body(const Dev &d, int l) {
    // every load that depends only on l is issued before the first branch, then the
    // endpoint state: two dependent load levels instead of four (latency-bound kernel)
    const uint2 li = d.linfo[l];
    const int2 e = d.ends[l];
    // link state (mixed precision): a 16-byte row {pos2, angle2v.x} and an 8-byte row
    // {angle2v.y, angle2v.z} per link, then angle1v component-major (mixed_lstate_*)
    const float *lsC = mixed_lstate_c(d);
    const size_t NL = (size_t)d.nl;
    const float4 sa = mixed_lstate_a(d)[l];
    const float2 sb = mixed_lstate_b(d)[l];
    // angle1v is zero while a link is in the small-angle branch (the flag it entered
    // this step with says so); it is read and written only for large-angle links and
    // zeroed once when a link returns to the small branch
    const bool wasSmall = (li.y & LF_SMALL) != 0;
    mx::LinkState s{{sa.x, sa.y, sa.z}, {0, 0, 0}, {sa.w, sb.x, sb.y}, d.strain[l], li.y};
    if (!wasSmall) s.a1v = V3<float>{lsC[l], lsC[NL + l], lsC[2 * NL + l]};
    pdl_wait_then_release();  // the previous voxel pass has moved the endpoints
    const float4 *P = reinterpret_cast<const float4 *>(d.pos);
    const float4 *Q = reinterpret_cast<const float4 *>(d.quat);
    const mx::Ends en{P[2 * e.x], P[2 * e.x + 1], Q[2 * e.x], Q[2 * e.x + 1]};
    const mx::Ends ep{P[2 * e.y], P[2 * e.y + 1], Q[2 * e.y], Q[2 * e.y + 1]};
    const int r = (int)li.x;
    if (d.status[r] != 0) return;
    const uint32_t fl = li.y;
    if (fl & (LF_BOTH_FIXED | LF_GONE)) return;
    LinkOut out{d, l, (int)(fl & LF_AXIS), r, e, fl};
    mx::link_step(d, mx::link_rows<HELD>(d.lrow, d.nlm, (int)(fl >> 8)), l, en, ep, s, out);
}

__global__ void k_init_temperature_mixed(Dev d) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= d.nv) return;
    const uint2 vi = d.vinfo[v];
    const VMat &m = d.vmat[vi.y >> 8];
    const RobotP &rp = d.rp[vi.x];
    float te = d.tempe[v];
    if (rp.vary_temp && rp.temp_period > 0 && !(m.thermal_on_after > 0.0) && !m.fixed)
        te = mx::temperature(make_float2(0.0f, 0.0f), d.phc[v], 0.0f, rp.cyc_rate, rp.amp_f, rp.expansion != 0);
    float4 *P = reinterpret_cast<float4 *>(d.pos);
    mx::base_size(mx::vox_row_c(m), te, P[2 * v].w, P[2 * v + 1].w);
    d.tempe[v] = te;
    d.tempe[d.nv + v] = te;
}

// ------------------------------------------------------------ voxel pass
// The FP64 arithmetic of the mixed voxel pass, kept out of line: if-converted into the
// pass, it would issue in every warp (GB300 runs FP64 at about 1/64 of the FP32 rate).
// The robot's time and actuation cycles of the next step (one thread per robot):
__device__ __noinline__ void advance_time(const Dev &d, const RobotP &rp, int r, int parity, float dtf, int st) {
    const double Tcur = d.T[(size_t)parity * d.nr + r];
    const double Tn = (st == 0) ? Tcur + dtf : Tcur;
    d.T[(size_t)(parity ^ 1) * d.nr + r] = Tn;
    d.tcyc[(size_t)(parity ^ 1) * d.nr + r] = mx::cycles_df(Tn * rp.inv_period * kCycle);
}
// a material with TurnOnThermalExpansionAfterThisManySeconds > 0: is expansion on at the
// end of this step?
__device__ __noinline__ bool thermal_on(const Dev &d, double toa, int r, int parity, float dtf) {
    return !(toa > d.T[(size_t)parity * d.nr + r] + dtf);
}

// a double as an FP32 hi/lo pair
__device__ __forceinline__ void set_df(float &hi, float &lo, double x) {
    hi = (float)x;
    lo = (float)(x - (double)hi);
}

// BC = false: every voxel without a boundary-condition external (the main pass, which
// compiles without the external code).  BC = true: the voxels with one (Dev::xbc), after
// the main pass, with the external force and moment, the fixed DOFs and the fixed-all
// pose (VX3_Voxel.cu:167-173, 222-257, 363-364, 393-394).
// EARLY: with registers for every load at once (the launch shapes of 96 registers and more)
template <bool BC, bool EARLY> __device__ __forceinline__ void voxels_mixed_body(const Dev &d, int v, int parity) {
    // the voxel's own state is loaded together with its info word, before any branch
    // (latency-bound kernel: one dependent level fewer)
    const uint2 vi = d.vinfo[v];
    float4 *P = reinterpret_cast<float4 *>(d.pos);
    float4 *Qa = reinterpret_cast<float4 *>(d.quat);
    float4 *LM = reinterpret_cast<float4 *>(d.linmom);
    float4 *AM = reinterpret_cast<float4 *>(d.angmom);
    mx::VoxelState s{P[2 * v], P[2 * v + 1], Qa[2 * v], Qa[2 * v + 1], LM[2 * v], LM[2 * v + 1], AM[2 * v], AM[2 * v + 1]};
    pdl_wait_then_release();  // the link pass (or the contact evaluation) of this step is done
    float *tcur = d.tempe + (size_t)parity * d.nv, *tnext = d.tempe + (size_t)(parity ^ 1) * d.nv;
    float te = 0;
    float2 ph = make_float2(0, 0);
    float4 ct = make_float4(0, 0, 0, 0);
    int si = -1;
    if (EARLY) {  // what depends on the voxel's number alone, beside the robot's and the materials' loads
        te = tcur[v];
        ph = d.phc[v];
        if (d.ns) ct = reinterpret_cast<const float4 *>(d.contact)[v];
        if (d.vsurf) si = d.vsurf[v];
    }
    const int r = (int)vi.x;
    const RobotP &rp = d.rp[r];
    const int st = d.status[r];
    const float dtf = d.dt[r];
    if (!BC && v == rp.voff) advance_time(d, rp, r, parity, dtf, st);
    uint32_t fl = vi.y;
    // the forces at its faces, with the loads that the checks below wait for
    V3<float> Fs{0, 0, 0}, Ms{0, 0, 0};
#pragma unroll
    for (int dir = 0; dir < 6; dir++) {
        if (fl & (1u << dir)) {
            V3<float> sf, sm;
            load_slot_mx(d, dir, v, &sf, &sm);
            Fs = add(Fs, sf);
            Ms = add(Ms, sm);
        }
    }
    if (st != 0) return;
    if (fl & VF_FIXED) return;
    if (!BC && rp.bcs && d.vext[v] >= 0) return;  // stepped by the BC pass
    const mx::VoxC m = mx::vox_rows(d.vrow, d.nvm, (int)(fl >> 8));
    const bool actuated = rp.vary_temp && rp.temp_period > 0;
    const int xi = BC ? d.vext[v] : -1;  // boundary-condition external
    const int dof = BC ? d.ext[xi].dof : 0;
    const double nom = BC ? d.vmat[fl >> 8].nom_size : 0.0;
    if (BC && dtf != 0.0f && dof == EXT_ALL) {  // isFixedAll (VX3_Voxel.cu:167-173)
        const ExtBC &e = d.ext[xi];
        const short4 l = d.ijk[v];
        set_df(s.pH.x, s.pL.x, l.x * nom + e.t.x);
        set_df(s.pH.y, s.pL.y, l.y * nom + e.t.y);
        set_df(s.pH.z, s.pL.z, l.z * nom + e.t.z);
        set_df(s.qH.x, s.qL.x, e.q.x);
        set_df(s.qH.y, s.qL.y, e.q.y);
        set_df(s.qH.z, s.qL.z, e.q.z);
        set_df(s.qH.w, s.qL.w, e.q.w);
        Qa[2 * v] = s.qH;
        Qa[2 * v + 1] = s.qL;
        const float4 z4 = make_float4(0, 0, 0, 0);
        LM[2 * v] = z4;
        LM[2 * v + 1] = z4;
        AM[2 * v] = z4;
        AM[2 * v + 1] = z4;
    } else if (dtf != 0.0f) {
        bool stat = (fl & VF_STATIC) != 0;
        const bool floorOn = rp.floor != 0;
        const Q4<float> o{s.qH.x, s.qH.y, s.qH.z, s.qH.w};
        V3<float> F = mx::rotate_voxel(o, Fs);
        if (BC) F = add(F, V3<float>{d.ext[xi].f[0], d.ext[xi].f[1], d.ext[xi].f[2]});  // external force
        const V3<float> vel = mx::velocity(s.lH, s.lL, m.a.x);
        F = mx::fma3(-m.a.z, vel, F);
        F.z = mx::plus(F.z, m.c.x);
        if (rp.collision) {
            if (!EARLY && d.ns) ct = reinterpret_cast<const float4 *>(d.contact)[v];
            F = mx::diff(F, V3<float>{ct.x, ct.y, ct.z});
        }
        if (rp.cilia) {  // CiliaForce * Cilia (VX3_Voxel.cu:376), evaluated in FP64 by k_extra_forces
            const double4 c = d.cfv[v];
            F = add(F, V3<float>{(float)c.x, (float)c.y, (float)c.z});
        }
        if (rp.ff_any) {  // force field (VX3_Voxel.cu:178-184), evaluated in FP64 by k_extra_forces
            const double4 ff = d.ffv[v];
            F = add(F, V3<float>{(float)ff.x, (float)ff.y, (float)ff.z});
        }
        mx::move(s, m, F, vel, floorOn, dtf, stat);
        V3<float> M = mx::rotate_voxel(o, Ms);
        if (BC) M = add(M, V3<float>{d.ext[xi].m[0], d.ext[xi].m[1], d.ext[xi].m[2]});  // external moment
        mx::turn(s, m, mx::fma3(-m.a.w, mx::velocity(s.aH, s.aL, fabsf(m.a.y)), M), dtf);
        if (BC && dof) {  // fixed DOFs (VX3_Voxel.cu:222-257), in FP64 on the hi/lo pairs
            const ExtBC &e = d.ext[xi];
            if (dof & EXT_T) {
                const short4 l = d.ijk[v];
                if (dof & 1) { set_df(s.pH.x, s.pL.x, l.x * nom + e.t.x); s.lH.x = s.lL.x = 0; }
                if (dof & 2) { set_df(s.pH.y, s.pL.y, l.y * nom + e.t.y); s.lH.y = s.lL.y = 0; }
                if (dof & 4) { set_df(s.pH.z, s.pL.z, l.z * nom + e.t.z); s.lH.z = s.lL.z = 0; }
            }
            if ((dof & EXT_R) == EXT_R) {  // all rotations: the prescribed orientation
                set_df(s.qH.x, s.qL.x, e.q.x);
                set_df(s.qH.y, s.qL.y, e.q.y);
                set_df(s.qH.z, s.qL.z, e.q.z);
                set_df(s.qH.w, s.qL.w, e.q.w);
                s.aH.x = s.aH.y = s.aH.z = s.aL.x = s.aL.y = s.aL.z = 0;
            } else if (dof & EXT_R) {  // some: those rotation-vector components zeroed
                V3<double> rv = to_rotvec(Q4<double>{(double)s.qH.x + s.qL.x, (double)s.qH.y + s.qL.y,
                                                     (double)s.qH.z + s.qL.z, (double)s.qH.w + s.qL.w});
                if (dof & 8) { rv.x = 0; s.aH.x = s.aL.x = 0; }
                if (dof & 16) { rv.y = 0; s.aH.y = s.aL.y = 0; }
                if (dof & 32) { rv.z = 0; s.aH.z = s.aL.z = 0; }
                const Q4<double> q = from_rotvec(rv);
                set_df(s.qH.x, s.qL.x, q.w);
                set_df(s.qH.y, s.qL.y, q.x);
                set_df(s.qH.z, s.qL.z, q.y);
                set_df(s.qH.w, s.qL.w, q.z);
            }
        }
        if (floorOn && mx::penetration(s, m) >= 0 && stat) s.aH.x = s.aH.y = s.aH.z = s.aL.x = s.aL.y = s.aL.z = 0;
        const uint32_t nfl = stat ? (fl | VF_STATIC) : (fl & ~VF_STATIC);
        if (nfl != fl) d.vinfo[v].y = nfl;
        Qa[2 * v] = s.qH;
        Qa[2 * v + 1] = s.qL;
        LM[2 * v] = s.lH;
        LM[2 * v + 1] = s.lL;
        AM[2 * v] = s.aH;
        AM[2 * v + 1] = s.aL;
    }
    if (actuated) {  // next step's temperature and base size
        if (!EARLY) te = tcur[v], ph = d.phc[v];
        if (m.a.y > 0.0f || thermal_on(d, d.vmat[fl >> 8].thermal_on_after, r, parity, dtf))
            te = mx::temperature(d.tcyc[(size_t)parity * d.nr + r], ph, dtf, rp.cyc_rate, rp.amp_f, rp.expansion != 0);
        mx::base_size(m.c, te, s.pH.w, s.pL.w);
        tnext[v] = te;
    }
    P[2 * v] = s.pH;
    P[2 * v + 1] = s.pL;
    // the next step's displacement check (k_coll_check), while the voxel is at hand: 64 bytes written
    // instead of a kernel that reads 80 and writes 64 (2.3 us of a 64^3 body's step, 9 us of 256
    // colliding robots')
    if (!EARLY && d.vsurf) si = d.vsurf[v];
    if (si >= 0) {
        const float4 q = d.cref[si];
        const float px = mx::plus(s.pH.x, s.pL.x), py = mx::plus(s.pH.y, s.pL.y), pz = mx::plus(s.pH.z, s.pL.z);
        d.cposf[si] = make_float4(px, py, pz, mx::plus(s.pH.w, s.pL.w));
        const float4 mb = m.b();
        contact_record(d, v, s.pH, s.pL, s.lH, m.a.x, mb.z, mb.x);
        const float ex = mx::minus(px, q.x), ey = mx::minus(py, q.y), ez = mx::minus(pz, q.z);
        if (fmaf(ez, ez, mx::dot_a(ex, ex, ey, ey)) > q.w) flag_robot(d, r);
    }
}

// the voxels with a boundary-condition external, after the main voxel pass
__global__ void __launch_bounds__(128) k_voxels_bc_mixed(Dev d, int parity) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.nxbc) voxels_mixed_body<true, false>(d, d.xbc[i], parity);
}

void launch_voxels_bc_mixed(const Dev &d, int parity, cudaStream_t s) {
    if (d.nxbc) k_voxels_bc_mixed<<<(d.nxbc + 127) / 128, 128, 0, s>>>(d, parity);
}

// Launch-shape variants (threads per block, minimum resident blocks): the same body, so every variant
// computes bit-identical results; they trade registers for occupancy (both passes are latency-bound
// gathers), and vx3g_autotune picks one of each per context by timing real steps.  HELD: a link's material
// rows are loaded with its ends and kept; EARLY: see voxels_mixed_body.
// Shape 6 of each is the default: small blocks, so that an SM's places are refilled a few warps at a time,
// and every load of a thread out at once.  Steps of 822,751 voxels / 410,307 / 262,144 / 32,768 / 13,824 without
// collisions, in us: shapes (6, 6) 143.8, 73.9, 45.6, 8.3, 5.8; (1, 0), in blocks of 256, 145.8, 76.5, 47.9, 10.0,
// 7.6; (1, 4), the voxel's loads held back until they are used to fit 72 registers, 151.5, 78.6, 46.0, 10.2, 9.3.
// A link's material rows held or not: 143.8 and 141.6, 73.9 and 74.0, 45.6 and 46.3, 8.3 and 8.7, 5.8 and 6.3.
// With collisions: a 64^3 body 41.1 us a step early in a run with (6, 6), 43.0 with (1, 0); 256 robots 136.7, 146.2.
template <int TPB, int MINB, bool HELD> __global__ void __launch_bounds__(TPB, MINB) k_links_mixed(Dev d) {
    const int l = blockIdx.x * TPB + threadIdx.x;
    if (l < d.nl) links_mixed_body<HELD>(d, l);
}
template <int TPB, int MINB, bool EARLY> __global__ void __launch_bounds__(TPB, MINB) k_voxels_mixed(Dev d, int parity) {
    const int v = blockIdx.x * TPB + threadIdx.x;
    if (v < d.nv) voxels_mixed_body<false, EARLY>(d, v, parity);
}

const LaunchShape kLinkShapes[kMixedShapes] = {{256, 1}, {256, 4}, {128, 9}, {128, 10}, {64, 20}, {256, 5}, {128, 8}, {128, 8}};
const LaunchShape kVoxelShapes[kMixedShapes] = {{256, 1}, {256, 3}, {128, 7}, {128, 8}, {64, 14}, {64, 16}, {64, 8}, {64, 10}};

// launch with programmatic stream serialization (see pdl_wait_then_release)
template <typename... KArgs, typename... Args>
static void launch_pdl(void (*kernel)(KArgs...), int n, int threads, cudaStream_t s, bool pdl, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((n + threads - 1) / threads));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

void launch_links_mixed(const Dev &d, cudaStream_t s, int shape, bool pdl) {
    if (!d.nl) return;
    switch (shape) {
        case 0: launch_pdl(k_links_mixed<256, 1, true>, d.nl, 256, s, pdl, d); break;
        case 1: launch_pdl(k_links_mixed<256, 4, false>, d.nl, 256, s, pdl, d); break;
        case 2: launch_pdl(k_links_mixed<128, 9, false>, d.nl, 128, s, pdl, d); break;
        case 3: launch_pdl(k_links_mixed<128, 10, false>, d.nl, 128, s, pdl, d); break;
        case 4: launch_pdl(k_links_mixed<64, 20, false>, d.nl, 64, s, pdl, d); break;
        case 5: launch_pdl(k_links_mixed<256, 5, false>, d.nl, 256, s, pdl, d); break;
        case 6: launch_pdl(k_links_mixed<128, 8, true>, d.nl, 128, s, pdl, d); break;
        default: launch_pdl(k_links_mixed<128, 8, false>, d.nl, 128, s, pdl, d); break;
    }
}
void launch_voxels_mixed(const Dev &d, int parity, cudaStream_t s, int shape, bool pdl) {
    if (!d.nv) return;
    switch (shape) {
        case 0: launch_pdl(k_voxels_mixed<256, 1, true>, d.nv, 256, s, pdl, d, parity); break;
        case 1: launch_pdl(k_voxels_mixed<256, 3, false>, d.nv, 256, s, pdl, d, parity); break;
        case 2: launch_pdl(k_voxels_mixed<128, 7, false>, d.nv, 128, s, pdl, d, parity); break;
        case 3: launch_pdl(k_voxels_mixed<128, 8, false>, d.nv, 128, s, pdl, d, parity); break;
        case 4: launch_pdl(k_voxels_mixed<64, 14, false>, d.nv, 64, s, pdl, d, parity); break;
        case 5: launch_pdl(k_voxels_mixed<64, 16, false>, d.nv, 64, s, pdl, d, parity); break;
        case 6: launch_pdl(k_voxels_mixed<64, 8, true>, d.nv, 64, s, pdl, d, parity); break;
        default: launch_pdl(k_voxels_mixed<64, 10, true>, d.nv, 64, s, pdl, d, parity); break;
    }
}
// ------------------------------------------------------------ many steps in one launch
// The link and voxel passes are bound by the latency of their dependent loads, and on a batch
// beyond the L2 by HBM (1024 robots, 7.1e5 voxels: 120 us a step, of which 76 us are the bytes at
// the copy rate; issue slots 25% used).  Robots never touch each other, so here a cluster of CTAs
// keeps a bundle of whole robots in its shared memory and takes n steps there: nothing leaves
// the cluster between steps.  A CTA owns a contiguous range of q voxels of the bundle and the
// links whose positive end is among them (links are made in the voxel order of that end); the
// negative end may be in a CTA of lower rank, reached through distributed shared memory.  Two
// barriers per step: after the links (forces written to the six rows of each end) and after the
// voxels.  Bound by those barriers and by instruction issue: 43 to 55% of the issue slots of an SM with
// work, 3.3 to 5.3 stall cycles of an instruction at the barriers; 83 us a step on those 1024 robots, 2.7
// instead of 5.9 on one robot of 104 voxels.
// Two CTAs of 384 threads per SM (113 KB each), so that one's loads overlap the other's
// arithmetic: 1200-voxel robots 80 us a step against 101 with one CTA of 768 threads.
struct ResRobot {
    double T[2];     // time by parity
    float2 tc[2];    // actuation cycles by parity
    double inv_period;
    float dt, cyc_rate, amp;
    int status;  // with kTorn, a link tore in this step: its voxels stay, and at the end of the step it is stopped
    int actuated, expansion, floor;
};
// The link phase takes no notice of kTorn, so that a step in which a robot diverges updates all of its
// links, as the reference does, whichever warp finds the torn one first; and a status without it
// changes between the voxel phase's barriers only.
constexpr int kTorn = 1 << 30;
// A CTA's arrays, all computed from q (voxels) and lc (links), multiples of 16.  Float4 planes of q:
// position hi, lo, orientation hi, lo, six force rows; then the link and material rows and the
// robots; then float2, float and byte planes.
struct ResSmem {
    int q, lc;
    __device__ __forceinline__ static float4 *base() {
        extern __shared__ float4 rsm[];
        return rsm;
    }
    __device__ __forceinline__ float4 &PH(int i) const { return base()[i]; }
    __device__ __forceinline__ float4 &PL(int i) const { return base()[q + i]; }
    __device__ __forceinline__ float4 &QH(int i) const { return base()[2 * q + i]; }
    __device__ __forceinline__ float4 &QL(int i) const { return base()[3 * q + i]; }
    __device__ __forceinline__ float4 &SA(int dir, int i) const { return base()[(4 + dir) * q + i]; }
    __device__ __forceinline__ float4 &LA(int i) const { return base()[10 * q + i]; }
    __device__ __forceinline__ float4 &lrow(int i) const { return base()[10 * q + lc + i]; }
    __device__ __forceinline__ float4 &vrow(int i) const { return base()[10 * q + lc + 4 * kResMats + i]; }
    __device__ __forceinline__ ResRobot &rob(int i) const {
        return reinterpret_cast<ResRobot *>(base() + 10 * q + lc + 7 * kResMats)[i];
    }
    __device__ __forceinline__ float2 *f2() const {
        return reinterpret_cast<float2 *>(base() + 10 * q + lc + 7 * kResMats + kResRobots * sizeof(ResRobot) / 16);
    }
    __device__ __forceinline__ float2 &SB(int dir, int i) const { return f2()[dir * q + i]; }
    __device__ __forceinline__ float2 &ph(int i) const { return f2()[6 * q + i]; }
    __device__ __forceinline__ float2 &LB(int i) const { return f2()[7 * q + i]; }
    __device__ __forceinline__ float2 &ST(int i) const { return f2()[7 * q + lc + i]; }
    __device__ __forceinline__ float *f1() const { return reinterpret_cast<float *>(f2() + 7 * q + 2 * lc); }
    __device__ __forceinline__ float &mom(int k, int i) const { return f1()[k * q + i]; }  // linear hi, lo, angular hi, lo
    __device__ __forceinline__ float &te(int i) const { return f1()[12 * q + i]; }
    __device__ __forceinline__ uint32_t &vi(int i) const { return reinterpret_cast<uint32_t *>(f1())[13 * q + i]; }
    __device__ __forceinline__ float &LC(int k, int i) const { return f1()[14 * q + k * lc + i]; }
    __device__ __forceinline__ uint32_t &fl(int i) const { return reinterpret_cast<uint32_t *>(f1())[14 * q + 3 * lc + i]; }
    __device__ __forceinline__ uint32_t &le(int i) const { return reinterpret_cast<uint32_t *>(f1())[14 * q + 4 * lc + i]; }  // ends in the bundle
    __device__ __forceinline__ unsigned char &rb(int i) const {  // robot in the bundle
        return reinterpret_cast<unsigned char *>(f1() + 14 * q + 5 * lc)[i];
    }
};
static_assert(sizeof(ResRobot) * kResRobots % 16 == 0, "alignment of the arrays after the robots");
static_assert(kResRobots <= 32, "one bit per robot of a bundle");
size_t steps_mixed_bytes(int q, int lc) {
    return (size_t)q * (10 * 16 + 7 * 8 + 14 * 4 + 1) + (size_t)lc * (16 + 2 * 8 + 5 * 4) + kResRobots * sizeof(ResRobot) +
           kResMats * 7 * 16;
}

template <bool CLUSTER> __device__ __forceinline__ void res_sync() {
    if (CLUSTER) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    else __syncthreads();
}
// the address in the shared memory of cluster rank k of what p points to in this CTA's
template <class T> __device__ __forceinline__ T *res_map(T *p, int k) {
    T *q;
    asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(k));
    return q;
}

template <bool CLUSTER> struct ResLinkOut {  // where k_steps_mixed leaves a link's update (mx::link_step)
    const Dev &d;
    const ResSmem &S;
    int i, axis, in, ip, own, rank, K, r0;
    uint32_t fl;
    __device__ __forceinline__ void local(V3<float> pos2, V3<float> a1v, V3<float> a2v, bool small) {
        S.LA(i) = make_float4(pos2.x, pos2.y, pos2.z, a2v.x);
        S.LB(i) = make_float2(a2v.y, a2v.z);
        if (!(small && (fl & LF_SMALL))) S.LC(0, i) = a1v.x, S.LC(1, i) = a1v.y, S.LC(2, i) = a1v.z;
    }
    __device__ __forceinline__ void strain(float2 s, bool torn) {
        S.ST(i) = s;
        if (!torn) return;
        const int k = S.rb(ip);
        atomicOr(&d.status[r0 + k], 1);
        if (!CLUSTER) atomicOr(&S.rob(k).status, kTorn);
        else
            for (int c = 0; c < K; c++) atomicOr(res_map(&S.rob(k).status, c), kTorn);
    }
    __device__ __forceinline__ void neg(V3<float> f, V3<float> m) {
        float4 *a = &S.SA(2 * axis, in);
        float2 *b = &S.SB(2 * axis, in);
        if (CLUSTER && own != rank) a = res_map(a, own), b = res_map(b, own);
        *a = make_float4(f.x, f.y, f.z, m.x);
        *b = make_float2(m.y, m.z);
    }
    __device__ __forceinline__ void pos(V3<float> f, V3<float> m) {
        S.SA(2 * axis + 1, ip) = make_float4(f.x, f.y, f.z, m.x);
        S.SB(2 * axis + 1, ip) = make_float2(m.y, m.z);
    }
    __device__ __forceinline__ void flags(uint32_t nfl, bool) { S.fl(i) = nfl; }
};

template <bool CLUSTER>
__device__ __forceinline__ void res_link(const Dev &d, const ResSmem &S, const ResBundle &B, int i, const int *lid, int rank, int K) {
    const uint32_t fl = S.fl(i);
    if (fl & (LF_BOTH_FIXED | LF_GONE)) return;
    const int q = B.q, vb = rank * q, axis = (int)(fl & LF_AXIS);
    const uint32_t e = S.le(i);
    const int ip = (int)(e >> 16) - vb;
    int in = (int)(e & 0xffffu) - vb, own = rank;
    if (S.rob(S.rb(ip)).status & ~kTorn) return;
    if (CLUSTER && in < 0) {  // the negative end is in a CTA of lower rank
        own = (int)(e & 0xffffu) / q;
        in = (int)(e & 0xffffu) - own * q;
    }
    mx::Ends en;
    if (CLUSTER && own != rank)
        en = mx::Ends{*res_map(&S.PH(in), own), *res_map(&S.PL(in), own), *res_map(&S.QH(in), own), *res_map(&S.QL(in), own)};
    else en = mx::Ends{S.PH(in), S.PL(in), S.QH(in), S.QL(in)};
    const mx::Ends ep{S.PH(ip), S.PL(ip), S.QH(ip), S.QL(ip)};
    const float4 sa = S.LA(i);
    const float2 sb = S.LB(i);
    mx::LinkState st{{sa.x, sa.y, sa.z}, {0, 0, 0}, {sa.w, sb.x, sb.y}, S.ST(i), fl};
    if (!(fl & LF_SMALL)) st.a1v = V3<float>{S.LC(0, i), S.LC(1, i), S.LC(2, i)};
    const int lm = (int)(fl >> 8);
    ResLinkOut<CLUSTER> out{d, S, i, axis, in, ip, own, rank, K, B.r0, fl};
    mx::link_step(d, B.nlm ? mx::link_rows<true>(&S.lrow(0), B.nlm, lm - B.lm0) : mx::link_rows<true>(d.lrow, d.nlm, lm), *lid, en, ep, st, out);
}

__device__ __forceinline__ void res_voxel(const Dev &d, const ResSmem &S, const ResBundle &B, int i, int v, int parity, bool last) {
    const uint32_t fl = S.vi(i);
    const ResRobot &R = S.rob(S.rb(i));
    if (R.status != 0 || (fl & VF_FIXED)) return;
    const float dtf = R.dt;
    const mx::VoxC m = B.nvm ? mx::vox_rows(&S.vrow(0), B.nvm, (int)(fl >> 8) - B.vm0)
                             : mx::vox_rows(d.vrow, d.nvm, (int)(fl >> 8));
    mx::VoxelState s;
    s.pH = S.PH(i), s.pL = S.PL(i);
    if (dtf != 0.0f) {
        s.qH = S.QH(i), s.qL = S.QL(i);
        s.lH = make_float4(S.mom(0, i), S.mom(1, i), S.mom(2, i), 0.0f);
        s.lL = make_float4(S.mom(3, i), S.mom(4, i), S.mom(5, i), 0.0f);
        s.aH = make_float4(S.mom(6, i), S.mom(7, i), S.mom(8, i), 0.0f);
        s.aL = make_float4(S.mom(9, i), S.mom(10, i), S.mom(11, i), 0.0f);
        V3<float> Fs{0, 0, 0}, Ms{0, 0, 0};
#pragma unroll
        for (int k = 0; k < 6; k++)
            if (fl & (1u << k)) {
                const float4 a = S.SA(k, i);
                const float2 b = S.SB(k, i);
                Fs = V3<float>{mx::plus(Fs.x, a.x), mx::plus(Fs.y, a.y), mx::plus(Fs.z, a.z)};
                Ms = V3<float>{mx::plus(Ms.x, a.w), mx::plus(Ms.y, b.x), mx::plus(Ms.z, b.y)};
            }
        bool stat = (fl & VF_STATIC) != 0;
        const Q4<float> o{s.qH.x, s.qH.y, s.qH.z, s.qH.w};
        const V3<float> vel = mx::velocity(s.lH, s.lL, m.a.x);
        V3<float> F = mx::fma3(-m.a.z, vel, mx::rotate_voxel(o, Fs));
        F.z = mx::plus(F.z, m.c.x);
        mx::move(s, m, F, vel, R.floor != 0, dtf, stat);
        mx::turn(s, m, mx::fma3(-m.a.w, mx::velocity(s.aH, s.aL, fabsf(m.a.y)), mx::rotate_voxel(o, Ms)), dtf);
        if (R.floor && mx::penetration(s, m) >= 0 && stat) s.aH = s.aL = make_float4(0, 0, 0, 0);
        const uint32_t nfl = stat ? (fl | VF_STATIC) : (fl & ~VF_STATIC);
        if (nfl != fl) S.vi(i) = nfl;
        S.QH(i) = s.qH, S.QL(i) = s.qL;
        const float w[12] = {s.lH.x, s.lH.y, s.lH.z, s.lL.x, s.lL.y, s.lL.z, s.aH.x, s.aH.y, s.aH.z, s.aL.x, s.aL.y, s.aL.z};
#pragma unroll
        for (int k = 0; k < 12; k++) S.mom(k, i) = w[k];
    }
    if (R.actuated) {  // next step's temperature and base size
        float te = S.te(i);
        if (last) d.tempe[(size_t)parity * d.nv + v] = te;  // the temperature the last step used
        if (m.a.y > 0.0f || !(d.vmat[fl >> 8].thermal_on_after > R.T[parity] + dtf))
            te = mx::temperature(R.tc[parity], S.ph(i), dtf, R.cyc_rate, R.amp, R.expansion != 0);
        mx::base_size(m.c, te, s.pH.w, s.pL.w);
        S.te(i) = te;
    }
    S.PH(i) = s.pH, S.PL(i) = s.pL;
}

// bundles, one per cluster; ctas: the first entry and the entries in `order` of each CTA's links,
// axis by axis, each axis filled up to whole warps with -1
template <bool CLUSTER>
__global__ void __launch_bounds__(kResThreads, 1) k_steps_mixed(Dev d, int parity, int n, const ResBundle *bundles, const int2 *ctas,
                                                                const int *order) {
    int rank = 0, K = 1;
    if (CLUSTER) {
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(K));
    }
    const ResBundle B = bundles[blockIdx.x / K];
    const int q = B.q;
    const ResSmem S{q, B.lc};
    const int tid = threadIdx.x, T = blockDim.x;
    const int vb = rank * q, nv = max(0, min(q, B.nv - vb)), v0 = B.v0 + vb;  // this CTA's voxels
    const int nl = ctas[blockIdx.x].y;
    const int *lid = order + ctas[blockIdx.x].x;
    const float4 *P = reinterpret_cast<const float4 *>(d.pos), *Qa = reinterpret_cast<const float4 *>(d.quat);
    const float4 *LM = reinterpret_cast<const float4 *>(d.linmom), *AM = reinterpret_cast<const float4 *>(d.angmom);
    for (int i = tid; i < nv; i += T) {
        const int v = v0 + i;
        S.PH(i) = P[2 * v], S.PL(i) = P[2 * v + 1], S.QH(i) = Qa[2 * v], S.QL(i) = Qa[2 * v + 1];
        const float4 a = LM[2 * v], b = LM[2 * v + 1], c = AM[2 * v], e = AM[2 * v + 1];
        const float m[12] = {a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z, e.x, e.y, e.z};
#pragma unroll
        for (int k = 0; k < 12; k++) S.mom(k, i) = m[k];
        const uint2 vi = d.vinfo[v];
        S.vi(i) = vi.y;
        S.rb(i) = (unsigned char)((int)vi.x - B.r0);
        S.ph(i) = d.phc[v];
        S.te(i) = d.tempe[(size_t)parity * d.nv + v];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            S.SA(k, i) = make_float4(0, 0, 0, 0);
            S.SB(k, i) = make_float2(0, 0);
        }
    }
    for (int i = tid; i < nl; i += T) {
        const int l = lid[i];
        S.fl(i) = LF_GONE;
        if (l < 0) continue;
        S.LA(i) = mixed_lstate_a(d)[l];
        S.LB(i) = mixed_lstate_b(d)[l];
        S.ST(i) = d.strain[l];
        const uint32_t fl = d.linfo[l].y;
        S.fl(i) = fl;
        const int2 e = d.ends[l];
        S.le(i) = (uint32_t)(e.x - B.v0) | (uint32_t)(e.y - B.v0) << 16;
        if (!(fl & LF_SMALL))
            for (int k = 0; k < 3; k++) S.LC(k, i) = mixed_lstate_c(d)[(size_t)k * d.nl + l];
    }
    for (int i = tid; i < 4 * B.nlm; i += T) S.lrow(i) = d.lrow[(size_t)(i / B.nlm) * d.nlm + B.lm0 + i % B.nlm];
    for (int i = tid; i < 3 * B.nvm; i += T) S.vrow(i) = d.vrow[(size_t)(i / B.nvm) * d.nvm + B.vm0 + i % B.nvm];
    for (int i = tid; i < B.nr; i += T) {
        const int r = B.r0 + i;
        const RobotP &rp = d.rp[r];
        ResRobot R;
        for (int k = 0; k < 2; k++) R.T[k] = d.T[(size_t)k * d.nr + r], R.tc[k] = d.tcyc[(size_t)k * d.nr + r];
        R.inv_period = rp.inv_period;
        R.dt = rp.nv ? d.dt[r] : 0.0f;  // a robot without voxels stays at its time
        R.cyc_rate = rp.cyc_rate, R.amp = rp.amp_f;
        R.status = d.status[r];
        R.actuated = rp.vary_temp && rp.temp_period > 0;
        R.expansion = rp.expansion, R.floor = rp.floor;
        S.rob(i) = R;
    }
    res_sync<CLUSTER>();
    unsigned stopped = 0;  // robots that were not running when the launch began
    for (int i = 0; i < B.nr; i++) stopped |= (unsigned)((S.rob(i).status & ~kTorn) != 0) << i;
    for (int s = 0; s < n; s++, parity ^= 1) {
        for (int i = tid; i < nl; i += T) res_link<CLUSTER>(d, S, B, i, lid + i, rank, K);
        res_sync<CLUSTER>();
        for (int i = tid; i < nv; i += T) res_voxel(d, S, B, i, v0 + i, parity, s == n - 1);
        // the robots' time and actuation cycles
        for (int i = T - 1 - tid; i < B.nr; i += T) {
            ResRobot &R = S.rob(i);
            const double Tn = R.status == 0 ? R.T[parity] + R.dt : R.T[parity];
            R.T[parity ^ 1] = Tn;
            R.tc[parity ^ 1] = mx::cycles_df(Tn * R.inv_period * kCycle);
            if (R.status & kTorn) R.status = (R.status & ~kTorn) | 1;
        }
        res_sync<CLUSTER>();
    }
    float4 *Po = reinterpret_cast<float4 *>(d.pos), *Qo = reinterpret_cast<float4 *>(d.quat);
    float4 *Lo = reinterpret_cast<float4 *>(d.linmom), *Ao = reinterpret_cast<float4 *>(d.angmom);
    float4 *ga = reinterpret_cast<float4 *>(d.slots);
    float2 *gb = reinterpret_cast<float2 *>(ga + 6 * (size_t)d.nv);
    for (int i = tid; i < nv; i += T) {
        const int v = v0 + i, r = S.rb(i);
        const uint32_t fl = S.vi(i);
        if ((stopped >> r) & 1u) continue;
        if (!(fl & VF_FIXED)) {
            Po[2 * v] = S.PH(i), Po[2 * v + 1] = S.PL(i), Qo[2 * v] = S.QH(i), Qo[2 * v + 1] = S.QL(i);
            Lo[2 * v] = make_float4(S.mom(0, i), S.mom(1, i), S.mom(2, i), 0.0f);
            Lo[2 * v + 1] = make_float4(S.mom(3, i), S.mom(4, i), S.mom(5, i), 0.0f);
            Ao[2 * v] = make_float4(S.mom(6, i), S.mom(7, i), S.mom(8, i), 0.0f);
            Ao[2 * v + 1] = make_float4(S.mom(9, i), S.mom(10, i), S.mom(11, i), 0.0f);
            d.vinfo[v].y = fl;
            if (S.rob(r).actuated) {
                d.tempe[(size_t)parity * d.nv + v] = S.te(i);
                if (S.rob(r).status != 0) d.tempe[(size_t)(parity ^ 1) * d.nv + v] = S.te(i);  // diverged on the way
            }
        }
#pragma unroll
        for (int k = 0; k < 6; k++)
            if (fl & (1u << k)) {
                ga[(size_t)k * d.nv + v] = S.SA(k, i);
                gb[(size_t)k * d.nv + v] = S.SB(k, i);
            }
    }
    for (int i = tid; i < nl; i += T) {
        const int l = lid[i];
        if (l < 0) continue;
        const int ip = (int)(S.le(i) >> 16) - vb;
        if ((stopped >> S.rb(ip)) & 1u) continue;
        mixed_lstate_a(d)[l] = S.LA(i);
        mixed_lstate_b(d)[l] = S.LB(i);
        d.strain[l] = S.ST(i);
        const uint32_t fl = S.fl(i);
        for (int k = 0; k < 3; k++) mixed_lstate_c(d)[(size_t)k * d.nl + l] = (fl & LF_SMALL) ? 0.0f : S.LC(k, i);
        d.linfo[l].y = fl;
    }
    if (rank == 0)
        for (int i = tid; i < B.nr; i += T)
            for (int k = 0; k < 2; k++) d.T[(size_t)k * d.nr + B.r0 + i] = S.rob(i).T[k], d.tcyc[(size_t)k * d.nr + B.r0 + i] = S.rob(i).tc[k];
}

// the links of each CTA of k_steps_mixed axis by axis, each axis padded with -1 to whole warps: one warp
// per CTA.  On the host this and its upload took 15 of the 96 ms that a batch of 1024 robots took to create.
__global__ void __launch_bounds__(32) k_res_order(const uint2 *linfo, const int2 *links, const int2 *ctas, int *order) {
    const int lane = threadIdx.x;
    const int2 lk = links[blockIdx.x];
    int at = ctas[blockIdx.x].x;
    for (uint32_t x = 0; x < 3; x++) {
        int n = 0;
        for (int l0 = lk.x; l0 < lk.y; l0 += 32) {
            const int l = l0 + lane;
            const bool hit = l < lk.y && (linfo[l].y & LF_AXIS) == x;
            const unsigned m = __ballot_sync(~0u, hit);
            if (hit) order[at + n + __popc(m & ((1u << lane) - 1))] = l;
            n += __popc(m);
        }
        const int end = (n + 31) / 32 * 32;
        if (n + lane < end) order[at + n + lane] = -1;
        at += end;
    }
}
cudaError_t launch_res_order(const Dev &d, const int2 *links, const int2 *ctas, int n, int *order, cudaStream_t s) {
    k_res_order<<<n, 32, 0, s>>>(d.linfo, links, ctas, order);
    return cudaGetLastError();
}

cudaError_t init_steps_mixed() {
    cudaError_t e = cudaFuncSetAttribute(k_steps_mixed<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_steps_mixed<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem);
    return e;
}

cudaError_t steps_mixed_active(int K, int threads, size_t smem, int *n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)K);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)K;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return K > 1 ? cudaOccupancyMaxActiveClusters(n, k_steps_mixed<true>, &cfg)
                 : cudaOccupancyMaxActiveClusters(n, k_steps_mixed<false>, &cfg);
}

cudaError_t launch_steps_mixed(const Dev &d, int parity, int n, const ResClass &c, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(c.count * c.K));
    cfg.blockDim = dim3((unsigned)c.threads);
    cfg.dynamicSmemBytes = c.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c.K;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = c.K > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, c.K > 1 ? k_steps_mixed<true> : k_steps_mixed<false>, d, parity, n, c.bundles, c.ctas, c.order);
}

// the material rows, once the time step is known
__global__ void k_rows_mixed(Dev d, float4 *lrow, float4 *vrow) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.nlm) {
        const mx::LinkC c = mx::link_consts_mx(d.lmat[i], d.dt[d.lmat[i].robot]);
        lrow[i] = c.ra, lrow[d.nlm + i] = c.rb, lrow[2 * (size_t)d.nlm + i] = c.rc, lrow[3 * (size_t)d.nlm + i] = c.re;
    }
    if (i < d.nvm) {
        const VMat &m = d.vmat[i];
        vrow[i] = mx::vox_row_a(m), vrow[d.nvm + i] = mx::vox_row_b(m), vrow[2 * (size_t)d.nvm + i] = mx::vox_row_c(m);
    }
}
void launch_rows_mixed(const Dev &d, float4 *lrow, float4 *vrow, cudaStream_t s) {
    const int n = d.nlm > d.nvm ? d.nlm : d.nvm;
    if (n) k_rows_mixed<<<(n + 127) / 128, 128, 0, s>>>(d, lrow, vrow);
}
void launch_init_temperature_mixed(const Dev &d, cudaStream_t s) {
    if (d.nv) k_init_temperature_mixed<<<(d.nv + 255) / 256, 256, 0, s>>>(d);
}

}  // namespace vx3g
