// Update kernels of one neuron model and integrator, EB_KIND and EB_INTEG (the
// build compiles this file once per pair, so the pairs compile in parallel).
#include "eb_step.cuh"

namespace eb {

template <int KIND, int INTEG>
void launch_update_t(const PopDev &P, const NetDev &N, int rel, int nsteps, double push_inv_dt, cudaStream_t st) {
    if (P.wide) {
        const int blocks = (int)std::min<int64_t>(P.n, 148 * 8);
        const size_t sm = stage_smem_bytes();
        if (P.mon) k_update_wide<KIND, INTEG, 1, -1><<<blocks, kWideThreads, sm, st>>>(P, N, rel, nsteps, push_inv_dt);
        else if (P.en == 1) k_update_wide<KIND, INTEG, 0, 1><<<blocks, kWideThreads, sm, st>>>(P, N, rel, nsteps, push_inv_dt);
        else k_update_wide<KIND, INTEG, 0, -1><<<blocks, kWideThreads, sm, st>>>(P, N, rel, nsteps, push_inv_dt);
    } else {
        // the common conductance sets get kernels with the set compiled in; a
        // monitored population takes the generic kernel with the monitor hooks
        const int blocks = (int)((P.n + 255) / 256);
        if (P.mon) k_update_narrow<KIND, INTEG, -1, 1><<<blocks, 256, 0, st>>>(P, N, rel, nsteps, push_inv_dt);
        else if (P.en == 1) k_update_narrow<KIND, INTEG, 1, 0><<<blocks, 256, 0, st>>>(P, N, rel, nsteps, push_inv_dt);
        else if (P.en == 3) k_update_narrow<KIND, INTEG, 3, 0><<<blocks, 256, 0, st>>>(P, N, rel, nsteps, push_inv_dt);
        else k_update_narrow<KIND, INTEG, -1, 0><<<blocks, 256, 0, st>>>(P, N, rel, nsteps, push_inv_dt);
    }
}

// Opt the wide updates into their staging area (dynamic shared memory above the
// 48 KB default) on the current device.
template <int KIND, int INTEG>
cudaError_t prepare_update_t() {
    const int bytes = (int)stage_smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(k_update_wide<KIND, INTEG, 0, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_update_wide<KIND, INTEG, 0, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_update_wide<KIND, INTEG, 1, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e;
}

template void launch_update_t<EB_KIND, EB_INTEG>(const PopDev &, const NetDev &, int, int, double, cudaStream_t);
template cudaError_t prepare_update_t<EB_KIND, EB_INTEG>();

}  // namespace eb
