// The FP64 step passes (compiled with --fmad=false: every multiply and add rounds
// separately, as in the reference's arithmetic) and the tables they read.
#include "vx3g_step.cuh"

namespace vx3g {

__global__ void __launch_bounds__(256) k_links_fp64(Dev d) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l < d.nl) link_update<double>(d, l);
}

// the blocks past the voxels' advance the robots' actuation phase for the next step: a sine and a
// cosine per robot, on other SMs than a small batch's voxels
__global__ void __launch_bounds__(256) k_voxels_fp64(Dev d, int parity, int vblocks) {
    if ((int)blockIdx.x < vblocks) {
        const int v = blockIdx.x * blockDim.x + threadIdx.x;
        if (v < d.nv) voxel_update<double>(d, v, parity);
        return;
    }
    const int r = (blockIdx.x - vblocks) * blockDim.x + threadIdx.x;
    if (r >= d.nr || d.status[r] != 0) return;
    if (!(d.rp[r].vary_temp && d.rp[r].temp_period > 0)) return;
    const double dt = d.dt[r], tn = d.T[(size_t)parity * d.nr + r] + dt;
    actuation_phase(d, r, parity ^ 1, tn + dt);
}

__global__ void k_actuation(Dev d, int parity) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= d.nr || !(d.rp[r].vary_temp && d.rp[r].temp_period > 0)) return;
    actuation_phase(d, r, parity, d.T[(size_t)parity * d.nr + r] + (double)d.dt[r]);
}

__global__ void k_fp64_tables(Dev d, LMatD *out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const LMat &m = d.lmat[i];
        out[i] = make_lmatd(m, m.dmcN, m.dmcP, m.fixN, m.fixP, d.dt[m.robot]);
    }
    if (d.actv && i < d.nv) d.actv[i] = actuation_voxel(d.phase[i]);
}

void launch_links_fp64(const Dev &d, cudaStream_t s) {
    const int t = fp64_threads(d.nl, 256);
    if (d.nl) k_links_fp64<<<(d.nl + t - 1) / t, t, 0, s>>>(d);
}
void launch_voxels_fp64(const Dev &d, int parity, cudaStream_t s) {
    const int t = fp64_threads(d.nv, 256), vb = (d.nv + t - 1) / t;
    if (d.nv) k_voxels_fp64<<<vb + (d.act ? (d.nr + t - 1) / t : 0), t, 0, s>>>(d, parity, vb);
}
void launch_actuation(const Dev &d, int parity, cudaStream_t s) {
    if (d.act) k_actuation<<<(d.nr + 31) / 32, 32, 0, s>>>(d, parity);
}
void launch_fp64_tables(const Dev &d, LMatD *lmatd, int n, cudaStream_t s) {
    const int k = d.nv > n ? d.nv : n;
    if (k) k_fp64_tables<<<(k + 255) / 256, 256, 0, s>>>(d, lmatd, n);
    launch_actuation(d, 0, s);
}

}  // namespace vx3g
