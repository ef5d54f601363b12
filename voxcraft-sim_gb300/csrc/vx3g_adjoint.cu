// vx3g_adjoint.cu -- kernels of the FP64 adjoint (per-element math in vx3g_adjoint.cuh)
// and the state-snapshot copy used by the recorded run and its recomputation.
#include "vx3g_adjoint.cuh"

namespace vx3g {

__global__ void __launch_bounds__(256) k_snap_copy(Snap dst, Snap src, int nv, int nl, int nr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nv) {
        dst.pos[i] = src.pos[i];
        dst.quat[i] = src.quat[i];
        dst.linmom[i] = src.linmom[i];
        dst.angmom[i] = src.angmom[i];
        dst.vinfo[i] = src.vinfo[i];
        dst.tempe[i] = src.tempe[i];
        dst.tempe[nv + i] = src.tempe[nv + i];
    }
    if (i < nl) {
        for (int k = 0; k < 9; k++) dst.lstate[(size_t)k * nl + i] = src.lstate[(size_t)k * nl + i];
        dst.strain[i] = src.strain[i];
        dst.linfo[i] = src.linfo[i];
    }
    if (i < nr) {
        dst.T[i] = src.T[i];
        dst.T[nr + i] = src.T[nr + i];
        dst.status[i] = src.status[i];
    }
}

void launch_snap_copy(const Snap &dst, const Snap &src, int nv, int nl, int nr, cudaStream_t st) {
    int n = nv > nl ? nv : nl;
    if (nr > n) n = nr;
    const int t = fp64_threads(n, 256);  // latency-bound when small: spread it
    if (n) k_snap_copy<<<(n + t - 1) / t, t, 0, st>>>(dst, src, nv, nl, nr);
}

static int adj_grid(int n) {
    const int t = fp64_threads(n, 128);
    return (n + t - 1) / t;
}

__global__ void __launch_bounds__(128) k_adj_voxel(Dev d, Snap s, AdjBufs a) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < d.nv) adj::adj_voxel(d, s, a, v);
}
__global__ void __launch_bounds__(128) k_adj_link(Dev d, Snap s, AdjBufs a) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l < d.nl) adj::adj_link(d, s, a, l);
}
// gather of step k+1 (state sg, parity a.parity), then the voxel adjoint of step k (state sv): each
// thread reads of the gather only what it wrote, and no other thread's entries are touched, so the two
// need no launch between them.  The reverse sweep is bound by the FP64 pipe, or, on a body of some 30
// warps, by one warp's chain of FP64 instructions (64 cycles each); the link forces and contacts of a
// step, which it used to compute again (two launches a step, three with collisions), come from the
// recompute store.  Record and backward of 200 steps of a 12x12x6 body: 42.5 -> 34.9 ms with the store,
// the widened constants, shared sines and the kept graphs; 60 of 12 colliding robots: 32.8 -> 25.6 ms.
// No contraction: where friction holds a body its gradient is a sum that cancels to 1e-6 of its terms,
// and rounding that differs shows in it.
__global__ void __launch_bounds__(128) k_adj_gather_voxel(Dev d, Snap sg, Snap sv, AdjBufs a) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= d.nv) return;
    adj::adj_gather(d, sg, a, v);
    a.parity ^= 1;
    adj::adj_voxel(d, sv, a, v);
}
__global__ void __launch_bounds__(128) k_adj_gather(Dev d, Snap s, AdjBufs a) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < d.nv) adj::adj_gather(d, s, a, v);
}
__global__ void __launch_bounds__(128) k_adj_seed(Dev d, AdjBufs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.nv) adj::adj_seed(d, a, i);
    if (i < d.nl)
        for (int k = 0; k < 9; k++) a.lloc[9 * (size_t)i + k] = 0.0;
}

void launch_adj_voxel(const Dev &d, const Snap &s, const AdjBufs &a, cudaStream_t st) {
    if (d.nv) k_adj_voxel<<<adj_grid(d.nv), fp64_threads(d.nv, 128), 0, st>>>(d, s, a);
}
void launch_adj_link(const Dev &d, const Snap &s, const AdjBufs &a, cudaStream_t st) {
    if (d.nl) k_adj_link<<<adj_grid(d.nl), fp64_threads(d.nl, 128), 0, st>>>(d, s, a);
}
void launch_adj_gather_voxel(const Dev &d, const Snap &sg, const Snap *sv, const AdjBufs &a, cudaStream_t st) {
    if (!d.nv) return;
    const int g = adj_grid(d.nv), t = fp64_threads(d.nv, 128);
    if (sv) k_adj_gather_voxel<<<g, t, 0, st>>>(d, sg, *sv, a);
    else k_adj_gather<<<g, t, 0, st>>>(d, sg, a);
}

__global__ void __launch_bounds__(128) k_adj_contact(Dev d, Snap s, AdjBufs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {  // the rebuild flags, cleared for the next check as the narrow phase does
        *d.cflag = 0;
        *d.lwork_ctr = 0ull;
    }
    if (i >= d.ns) return;
    const int r = (int)s.vinfo[d.csurf[i]].x;
    if (d.cflag[1 + r]) d.cflag[1 + r] = 0;
    adj::adj_contact(d, s, a, i);
}

void launch_adj_contact(const Dev &d, const Snap &s, const AdjBufs &a, cudaStream_t st) {
    if (d.ns) k_adj_contact<<<adj_grid(d.ns), fp64_threads(d.ns, 128), 0, st>>>(d, s, a);
}

void launch_adj_seed(const Dev &d, const AdjBufs &a, cudaStream_t st) {
    const int n = d.nv > d.nl ? d.nv : d.nl;
    if (n) k_adj_seed<<<adj_grid(n), fp64_threads(n, 128), 0, st>>>(d, a);
}

}  // namespace vx3g
