// Launchers of the step kernels, and the kernels that belong to no neuron model:
// input fan-out, Poisson generators, the deferred-STDP flush and the weight transfer.  The update kernels are in eb_step.cuh.
#include "eb_step.cuh"

namespace eb {

// PoissonGeneratorDeviceVector::UpdateState (src/neuron_model/PoissonGeneratorDeviceVector.cpp:56-70):
// a generator with frequency > 0 draws frand() from its own RandomGenerator --
// x <- (x * 1103515245 + 12345) & 0x7fffffff, frand = (float)x / MAX_RAND
// (include/simulation/RandomGenerator.h:91-107) -- and fires when
// frequency * step > frand.  The low 31 bits of the product only depend on its low
// 32 bits, so 32-bit arithmetic gives the reference's sequence.
__global__ void __launch_bounds__(256) k_update_poisson(PopDev P, NetDev N, int rel, int nsteps, double push_inv_dt) {
    const int64_t k0 = cur_step(N, rel);
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const double thr = i < P.n ? P.pthr[i] : 0.0;
    uint32_t x = i < P.n ? P.lcg[i] : 0u;
    for (int s = 0; s < nsteps; ++s) {
        const int64_t k = k0 + s;
        bool sp = false;
        if (thr > 0.0) {
            x = (x * 1103515245u + 12345u) & 0x7fffffffu;
            const float r = (float)x / (float)2147483647;
            sp = thr > (double)r;
        }
        compact_spikes(P, N, k, i, sp, false);
        if (push_inv_dt > 0.0) warp_push(P, N, k, i, sp, push_inv_dt);
    }
    if (i < P.n && thr > 0.0) P.lcg[i] = x;
}

// Input spikes of steps k .. k+nsteps-1.  Their deliveries are independent, so the
// window's inputs -- one contiguous range of the staged list -- are spread over
// the blocks at once; each block finds its spike's step among the window's
// input ranges.
__global__ void __launch_bounds__(256) k_input_push(NetDev N, int rel, int nsteps, double inv_dt) {
    const int64_t k0 = cur_step(N, rel);
    const int64_t q0 = N.in_start[k0], q1 = N.in_start[k0 + nsteps];
    for (int64_t q = q0 + blockIdx.x; q < q1; q += gridDim.x) {
        int64_t k = k0;
        while (k + 1 < k0 + nsteps && N.in_start[k + 1] <= q) ++k;
        input_spike(N, k, q, inv_dt);
    }
}

int persist_class_of(int kind, int integ) {
    if (integ == INTEG_BDF) return 2;
    return kind == KIND_HH ? 1 : 0;
}

template <int CLASS>
const void *persist_fn_t();

static const void *persist_fn(int cls) {
    return cls == 0 ? persist_fn_t<0>() : cls == 1 ? persist_fn_t<1>() : persist_fn_t<2>();
}

int persistent_blocks_per_sm(int cls) {
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, persist_fn(cls), kNarrowTile, 0);
    return nb;
}

cudaError_t launch_persistent(int cls, const PopDev *pops, const PersistInfo &I, const NetDev &N, int K, int grid,
                              cudaStream_t st) {
    void *args[] = {(void *)&pops, (void *)&I, (void *)&N, (void *)&K};
    return cudaLaunchCooperativeKernel(persist_fn(cls), dim3(grid), dim3(kNarrowTile), args, 0, st);
}

// Ends every run segment.  The record count and the error flags go straight to host
// memory, so that a run and a drain need no copies to read them: a closed loop of 10
// steps a call made four of those of 12-18 us each (137 -> 82 us a
// pass with its inputs and read-backs, windows included).
__global__ void k_advance(int64_t *step, int K, const unsigned long long *rec_count, const uint32_t *flags, RunStatus *status) {
    *step += K;
    status->rec_count = *rec_count;
    status->flags = *flags;
}

// ------------------------------------------------------------------ launch --
// Instantiated per model and integrator by eb_update.cu, per register class by eb_persist.cu.
template <int KIND, int INTEG>
void launch_update_t(const PopDev &P, const NetDev &N, int rel, int nsteps, double push_inv_dt, cudaStream_t st);
template <int KIND, int INTEG>
cudaError_t prepare_update_t();

template <int KIND>
static void launch_update_k(const PopDev &P, const NetDev &N, int rel, int nsteps, double push_inv_dt, cudaStream_t st) {
    switch (P.integ) {
    case INTEG_EULER: launch_update_t<KIND, INTEG_EULER>(P, N, rel, nsteps, push_inv_dt, st); break;
    case INTEG_RK2: launch_update_t<KIND, INTEG_RK2>(P, N, rel, nsteps, push_inv_dt, st); break;
    case INTEG_RK4: launch_update_t<KIND, INTEG_RK4>(P, N, rel, nsteps, push_inv_dt, st); break;
    default: launch_update_t<KIND, INTEG_BDF>(P, N, rel, nsteps, push_inv_dt, st); break;
    }
}

template <int KIND>
static cudaError_t prepare_update_k() {
    cudaError_t e = prepare_update_t<KIND, INTEG_EULER>();
    if (e == cudaSuccess) e = prepare_update_t<KIND, INTEG_RK2>();
    if (e == cudaSuccess) e = prepare_update_t<KIND, INTEG_RK4>();
    if (e == cudaSuccess) e = prepare_update_t<KIND, INTEG_BDF>();
    return e;
}

// Kernel attributes of every update; once per device, before any launch.
cudaError_t prepare_update_kernels() {
    cudaError_t e = prepare_update_k<KIND_LIF>();
    if (e == cudaSuccess) e = prepare_update_k<KIND_ADEX>();
    if (e == cudaSuccess) e = prepare_update_k<KIND_HH>();
    return e;
}

void launch_update(const PopDev &P, const NetDev &N, int rel, int nsteps, double push_inv_dt, cudaStream_t st) {
    if (P.n <= 0) return;
    switch (P.kind) {
    case KIND_LIF: launch_update_k<KIND_LIF>(P, N, rel, nsteps, push_inv_dt, st); break;
    case KIND_ADEX: launch_update_k<KIND_ADEX>(P, N, rel, nsteps, push_inv_dt, st); break;
    case KIND_HH: launch_update_k<KIND_HH>(P, N, rel, nsteps, push_inv_dt, st); break;
    case KIND_POISSON:
        k_update_poisson<<<(unsigned)((P.n + 255) / 256), 256, 0, st>>>(P, N, rel, nsteps, push_inv_dt);
        break;
    default: break;
    }
}

void launch_input_push(const NetDev &N, int rel, int nsteps, double inv_dt, int blocks, int threads, cudaStream_t st) {
    k_input_push<<<blocks, threads, 0, st>>>(N, rel, nsteps, inv_dt);
}

// Bring every plastic synapse onto the population up to date with its target's
// deferred post-synaptic spikes: items are (neuron, chunk of kPostThreads plastic
// synapses), neurons without spikes since the last flush skipped.
// Deferred post-synaptic flush in three launches: k_flush_select lists the neurons
// with more than keep pending spikes (P.flush_list, count P.flush_list[P.n]);
// k_flush_post brings their plastic synapses up to date, items (listed neuron,
// chunk of kPostThreads synapses) in contiguous runs per block, so a block reads a
// neuron's count and stages its ring in shared memory once for all its chunks;
// k_flush_mark records the listed neurons as flushed and clears the list.
__global__ void __launch_bounds__(256) k_flush_select(PopDev P, uint32_t keep) {
    uint32_t *list = P.flush_list, *count = P.flush_list + P.n;
    for (int64_t i = threadIdx.x; i < P.n; i += blockDim.x)
        if (P.post_n[i] - P.post_flushed[i] > keep) list[atomicAdd(count, 1u)] = (uint32_t)i;
}

__global__ void __launch_bounds__(kPostThreads) k_flush_post(PopDev P, NetDev N, int max_chunks) {
    __shared__ double ring[kPostRing];
    __shared__ DecayPair fac[kPostRing];
    __shared__ uint32_t s_c;
    const int64_t items = (int64_t)P.flush_list[P.n] * max_chunks;
    const int64_t per = (items + gridDim.x - 1) / gridDim.x;
    const int64_t it0 = (int64_t)blockIdx.x * per, it1 = min(items, it0 + per);
    const int rule = P.post_f ? P.post_rule : -1;
    int64_t cur = -1;
    for (int64_t item = it0; item < it1; ++item) {
        const int64_t li = item / max_chunks, ch = item - li * max_chunks;
        const int64_t i = P.flush_list[li];
        if (li != cur) {
            __syncthreads();  // the block is done with the previous neuron's ring
            if (threadIdx.x == 0) s_c = P.post_n[i];
            for (int q = threadIdx.x; q < kPostRing; q += blockDim.x) {
                ring[q] = P.post_t[i * kPostRing + q];
                if (P.post_f) fac[q] = P.post_f[i * kPostRing + q];
            }
            __syncthreads();
            cur = li;
        }
        const int64_t t = P.first + i;
        const int64_t tp = N.in_ptr[t] + ch * kPostThreads + threadIdx.x;
        if (tp >= N.plastic_end[t]) continue;
        SynRec r = N.syn[tp];
        apply_pending(N, RingSmem{ring, fac}, s_c, rule, r);
        SynRec *o = N.syn + tp;
        o->w = r.w;
        o->pre = r.pre;
        o->post = r.post;
        o->last = r.last;
    }
}

__global__ void __launch_bounds__(256) k_flush_mark(PopDev P) {
    uint32_t *list = P.flush_list, *count = P.flush_list + P.n;
    const uint32_t n = *count;
    for (uint32_t a = threadIdx.x; a < n; a += blockDim.x) {
        const uint32_t i = list[a];
        P.post_flushed[i] = P.post_n[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) *count = 0;
}

void launch_flush_post(const PopDev &P, const NetDev &N, int max_chunks, uint32_t keep, int blocks, cudaStream_t st) {
    k_flush_select<<<1, 256, 0, st>>>(P, keep);
    k_flush_post<<<blocks, kPostThreads, 0, st>>>(P, N, max_chunks);
    k_flush_mark<<<1, 256, 0, st>>>(P);
}

// Weights in network-file order out of and into the synapse records.  Bound by the
// gather: one 32-byte sector per synapse (the record's) and 8 bytes streamed, so a
// thread takes one synapse and the loads of a warp are independent.  A pass of 2,000
// steps, spikes and weights of the 250k-granule layer with 3.0M synapses: 18.7 ms,
// 64.5 ms when the 96 MB of records went to the host and were permuted there.
__global__ void __launch_bounds__(256) k_weights_get(const SynRec *__restrict__ syn, const uint32_t *__restrict__ tpos,
                                                     int64_t c, float *__restrict__ w) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < c) w[k] = syn[tpos[k]].w;
}

__global__ void __launch_bounds__(256) k_weights_set(SynRec *__restrict__ syn, const uint32_t *__restrict__ tpos,
                                                     int64_t c, const float *__restrict__ w) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < c) syn[tpos[k]].w = w[k];
}

void launch_weights_get(const SynRec *syn, const uint32_t *tpos, int64_t c, float *w, cudaStream_t st) {
    k_weights_get<<<(unsigned)((c + 255) / 256), 256, 0, st>>>(syn, tpos, c, w);
}

void launch_weights_set(SynRec *syn, const uint32_t *tpos, int64_t c, const float *w, cudaStream_t st) {
    k_weights_set<<<(unsigned)((c + 255) / 256), 256, 0, st>>>(syn, tpos, c, w);
}

void launch_advance(int64_t *step, int K, const NetDev &N, RunStatus *status, cudaStream_t st) {
    k_advance<<<1, 1, 0, st>>>(step, K, N.rec_count, N.flags, status);
}

}  // namespace eb
