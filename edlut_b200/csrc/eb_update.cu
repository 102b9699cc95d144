// Update kernels of one neuron model and integrator, EB_KIND and EB_INTEG (the
// build compiles this file once per pair, so the pairs compile in parallel).
#include "eb_step.cuh"

namespace eb {

// Neurons per warp of the thread-per-neuron update.  A population too small to give
// every SM sub-partition (148 x 4) a full warp is bound by one warp's serial chain,
// which is that of its slowest lane (Newton iterations, arrivals, spikes to fan
// out): fewer neurons a warp shorten it and cost nothing, down to the 4 whose state
// shares 16 bytes.  Stiff HH, us a step: 1,000 neurons 13.4 -> 10.9, 3,001 14.5 ->
// 11.9; from 18,944 neurons on every warp is full.
static int narrow_npw(int64_t n) { return (int)std::min<int64_t>(32, std::max<int64_t>(4, (n + 148 * 4 - 1) / (148 * 4))); }

// Threads per block: nothing is shared in a block, so small ones only spread the
// warps more evenly over the SMs (32 blocks fit one).  One warp while warps are
// scarce, two when all are full (stiff HH, 20,000 neurons: 17.1 us a step, 18.3 with
// blocks of 256; 100,000: 33.4, 32.4).
static int narrow_tile(int npw) { return npw < 32 ? 32 : 64; }

// Populations that fit the SMs at the register count the unbounded update needs
// (16 warps an SM at up to 128 registers, HH 12 at 168).
static int64_t narrow_few(int kind) { return 148 * 32 * (kind == KIND_HH ? 12 : 16); }

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
        const int npw = narrow_npw(P.n), tile = narrow_tile(npw), per = tile / 32 * npw;
        const int blocks = (int)((P.n + per - 1) / per);
        auto launch = [&](auto fn) { fn<<<blocks, tile, 0, st>>>(P, N, rel, nsteps, push_inv_dt, npw); };
        // The staged window is compiled with and without the plastic code; the per-step fold
        // asks at run time: its code is the same.  Of the populations that fit the SMs, the
        // monitored ones and those with the common conductance sets take the staged window,
        // HH at every size.  LIF and AdEx with other sets (NMDA, inhibition alone) keep the
        // per-step fold and its register bound: no workload measured has them.  Large plastic
        // HH with the set compiled in, 100,000 neurons: 30.6 us a step (AMPA; AMPA and GABA
        // 31.6), 32.4 with the set asked at run time.
        const bool small = P.n <= narrow_few(KIND), plastic = P.post_t != nullptr;
        constexpr bool HH = KIND == KIND_HH;
        if (P.mon) plastic ? launch(k_update_narrow<KIND, INTEG, -1, 1, true, true>) : launch(k_update_narrow<KIND, INTEG, -1, 1, true, false>);
        else if (P.en == 1 && small) plastic ? launch(k_update_narrow<KIND, INTEG, 1, 0, true, true>) : launch(k_update_narrow<KIND, INTEG, 1, 0, true, false>);
        else if (P.en == 3 && small) plastic ? launch(k_update_narrow<KIND, INTEG, 3, 0, true, true>) : launch(k_update_narrow<KIND, INTEG, 3, 0, true, false>);
        else if (P.en == 1) plastic ? launch(k_update_narrow<KIND, INTEG, 1, 0, false, HH>) : launch(k_update_narrow<KIND, INTEG, 1, 0, false, false>);
        else if (P.en == 3) plastic ? launch(k_update_narrow<KIND, INTEG, 3, 0, false, HH>) : launch(k_update_narrow<KIND, INTEG, 3, 0, false, false>);
        else plastic ? launch(k_update_narrow<KIND, INTEG, -1, 0, false, HH>) : launch(k_update_narrow<KIND, INTEG, -1, 0, false, false>);
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
