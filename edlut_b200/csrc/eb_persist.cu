// Persistent kernel of one register class, EB_CLASS (the build compiles this file
// once per class).
#include "eb_step.cuh"

namespace eb {

// -------------------------------------------------------- persistent kernel --
// All phases of K consecutive steps in one cooperative launch.  Per step:
//   [inputs]  input-spike fan-out (its own phase only when an input delivery can
//             reach the step being updated)
//   phase A   neuron updates of every population (+ input fan-out when it cannot
//             reach this step): narrow tiles of 256 neurons / one block per
//             wide neuron, items spread over the blocks
//   phase B   post-synaptic STDP chunks and spike fan-out of every population
// separated by grid barriers.  Removes the per-launch cost (about 3 us per
// kernel on this part) and the graph dependency latency of the K x (2..3)
// launches it replaces.  Every barrier wait is bounded: on timeout the block
// records FLAG_BARRIER_TIMEOUT and the kernel ends (I.spin_limit polls).
constexpr int kTlSlots = 6;
constexpr int kBarrierGroup = 16;     // blocks per first-level counter
constexpr int kBarrierStride = 32;    // words between counters (own 128-byte line)

// Two-level grid barrier: blocks arrive on the counter of their group of
// kBarrierGroup; the last of a group arrives on the root counter; the last at
// the root resets the counters and advances the generation word every block
// polls.  Spreads the arrival atomics over many cache lines instead of
// serialising gridDim.x of them on one.  Layout of bar (words):
//   [0] generation, [kBarrierStride] root count, [(g+2)*kBarrierStride] group g.
// I.withhold: block 0 does not arrive, so every block's wait runs out -- the
// failure path, exercised on purpose with a short I.spin_limit.
__device__ __forceinline__ bool grid_sync(const PersistInfo &I, unsigned nblocks, uint32_t *flags) {
    unsigned *bar = I.bar;
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        s_ok = 1;
        volatile unsigned *gen = bar;
        const unsigned g = *gen;
        const unsigned grp = blockIdx.x / kBarrierGroup;
        const unsigned ngroups = (nblocks + kBarrierGroup - 1) / kBarrierGroup;
        const unsigned in_grp = min((unsigned)kBarrierGroup, nblocks - grp * kBarrierGroup);
        unsigned *gc = bar + (grp + 2) * kBarrierStride;
        unsigned *root = bar + kBarrierStride;
        __threadfence();
        bool last = false;
        if (I.withhold && blockIdx.x == 0) {
        } else if (atomicAdd(gc, 1u) == in_grp - 1) {
            *gc = 0;
            __threadfence();
            if (atomicAdd(root, 1u) == ngroups - 1) {
                *root = 0;
                last = true;
            }
        }
        if (last) {
            __threadfence();
            atomicAdd(bar, 1u);
        } else {
            unsigned long long spins = 0;
            while (*gen == g) {
                __nanosleep(32);
                if (++spins > I.spin_limit) {
                    atomicOr(flags, FLAG_BARRIER_TIMEOUT);
                    s_ok = 0;
                    break;
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
    return s_ok != 0;
}

template <int KIND, int INTEG>
__device__ __forceinline__ void update_item(const PopDev &P, const NetDev &N, int64_t k, int64_t local, WideSmem &S) {
    if (P.wide) update_wide_neuron<KIND, INTEG>(P, N, k, local, S);
    else update_narrow_tile<KIND, INTEG>(P, N, k, local);
}

// Register classes of the persistent kernel: the switch below compiles in only
// the model/integrator pairs of its class, so a network without HH or BDF does
// not pay their register pressure.
//   0: LIF, AdEx x Euler, RK2, RK4   1: + HH x Euler, RK2, RK4   2: everything
template <int CLASS, int KIND>
__device__ __forceinline__ void update_item_k(const PopDev &P, const NetDev &N, int64_t k, int64_t local, WideSmem &S) {
    switch (P.integ) {
    case INTEG_EULER: update_item<KIND, INTEG_EULER>(P, N, k, local, S); break;
    case INTEG_RK2: update_item<KIND, INTEG_RK2>(P, N, k, local, S); break;
    case INTEG_RK4: update_item<KIND, INTEG_RK4>(P, N, k, local, S); break;
    default:
        if constexpr (CLASS >= 2) update_item<KIND, INTEG_BDF>(P, N, k, local, S);
        else if (threadIdx.x == 0) atomicOr(N.flags, FLAG_PERSIST_UNSUPPORTED);
        break;
    }
}

__device__ __forceinline__ int64_t update_items(const PopDev &P) {
    return P.wide ? P.n : (P.n + kNarrowTile - 1) / kNarrowTile;
}

// The item code reads its population's parameters many times per neuron; a
// block keeps the descriptor of the population it is working on in shared
// memory (broadcast reads) and reloads it only when it moves to another one.
__device__ __forceinline__ const PopDev &stage_pop(const PopDev *pops, int q, PopDev &sp, int &cur) {
    if (cur != q) {
        __syncthreads();
        const int *src = reinterpret_cast<const int *>(pops + q);
        int *dst = reinterpret_cast<int *>(&sp);
        for (int w = threadIdx.x; w < (int)(sizeof(PopDev) / sizeof(int)); w += blockDim.x) dst[w] = src[w];
        __syncthreads();
        cur = q;
    }
    return sp;
}

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Optional timeline (I.tl): per step r < I.tl_steps and block b, globaltimer at
// phase start, phase-A barrier arrival, phase-A barrier exit, phase-B barrier arrival.
__device__ __forceinline__ void tl_mark(const PersistInfo &I, int r, int slot) {
    if (I.tl && r < I.tl_steps && threadIdx.x == 0) I.tl[((int64_t)r * kTlSlots + slot) * gridDim.x + blockIdx.x] = gtimer();
}
__device__ __forceinline__ void tl_put(const PersistInfo &I, int r, int slot, unsigned long long v) {
    if (I.tl && r < I.tl_steps && threadIdx.x == 0) I.tl[((int64_t)r * kTlSlots + slot) * gridDim.x + blockIdx.x] = v;
}

// Dynamic item queue of one phase: each block starts with item blockIdx.x and
// then takes the next free index from the phase's counter (gridDim.x + n), so a
// block held up by a long item (a wide neuron) does not also receive later items.
// Thread 0 requests the following index as soon as it starts an item, hiding the
// atomic's latency behind the item's work.
struct ItemQueue {
    unsigned long long *ctr;
    int64_t cur, next;
    __device__ __forceinline__ void begin(unsigned long long *c) {
        ctr = c;
        cur = blockIdx.x;
    }
    __device__ __forceinline__ void prefetch() {
        if (threadIdx.x == 0) next = (int64_t)gridDim.x + (int64_t)atomicAdd(ctr, 1ull);
    }
    __device__ __forceinline__ int64_t advance(int64_t *s_next) {
        __syncthreads();
        if (threadIdx.x == 0) *s_next = next;
        __syncthreads();
        cur = *s_next;
        return cur;
    }
};

template <int CLASS>
__global__ void __launch_bounds__(kNarrowTile, CLASS == 0 ? 3 : (CLASS == 1 ? 2 : 1)) k_persistent(const PopDev *__restrict__ pops, PersistInfo I, NetDev N,
                                                            int K) {
    __shared__ WideSmem S;
    __shared__ PopDev sp;
    __shared__ int64_t s_next;
    int cur = -1;
    ItemQueue Q;
    const int64_t base = *N.step;
    const unsigned nb = gridDim.x;
    for (int r = 0; r < K; ++r) {
        const int64_t k = base + r + 1;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            for (int q = 0; q < I.n_pops; ++q) pops[q].spk_count[(k + 1) & 1] = 0;
            I.queue[(((k + 1) & 1) * 2 + 0) * 16] = 0;  // counters of the next step's phases
            I.queue[(((k + 1) & 1) * 2 + 1) * 16] = 0;
        }
        int64_t n_in = 0, q0 = 0;
        if (I.has_inputs) { q0 = N.in_start[k]; n_in = N.in_start[k + 1] - q0; }
        if (I.has_inputs && !I.inputs_concurrent) {
            for (int64_t it = blockIdx.x; it < n_in; it += nb) input_spike(N, k, q0 + it, I.inv_dt);
            if (!grid_sync(I, nb, N.flags)) return;
            n_in = 0;
        }
        // phase A: longest items first -- the populations in I.order (wide ones
        // first), with the input fan-out after the wide populations
        tl_mark(I, r, 0);
        int64_t total = n_in;
        for (int q = 0; q < I.n_pops; ++q) total += update_items(pops[q]);
        int n_items = 0;
        Q.begin(I.queue + ((k & 1) * 2 + 0) * 16);
        for (int64_t it = Q.cur; it < total; it = Q.advance(&s_next)) {
            Q.prefetch();
            if (n_items == 1) tl_mark(I, r, 4);
            ++n_items;
            int64_t local = it;
            int j = 0, q = -1;
            for (; j < I.n_pops; ++j) {
                if (j == I.n_wide) {
                    if (local < n_in) break;
                    local -= n_in;
                }
                const int64_t ni = update_items(pops[I.order[j]]);
                if (local < ni) { q = I.order[j]; break; }
                local -= ni;
            }
            if (q < 0) { input_spike(N, k, q0 + local, I.inv_dt); continue; }  // (advance runs in the for header)
            const PopDev &P = stage_pop(pops, q, sp, cur);
            switch (P.kind) {
            case KIND_LIF: update_item_k<CLASS, KIND_LIF>(P, N, k, local, S); break;
            case KIND_ADEX: update_item_k<CLASS, KIND_ADEX>(P, N, k, local, S); break;
            default:
                if constexpr (CLASS >= 1) update_item_k<CLASS, KIND_HH>(P, N, k, local, S);
                break;
            }
        }
        tl_mark(I, r, 1);
        tl_put(I, r, 5, (unsigned long long)n_items);
        if (!grid_sync(I, nb, N.flags)) return;
        tl_mark(I, r, 2);
        // phase B
        int64_t cnt[kMaxPersistPops];
        total = 0;
        for (int q = 0; q < I.n_pops; ++q) {
            const int64_t ns = min((int64_t)pops[q].spk_count[k & 1], pops[q].n);
            cnt[q] = ns * ((I.has_plastic >> q) & 1 ? I.post_chunks[q] : 0) + ns * ((I.has_out >> q) & 1);
            total += cnt[q];
        }
        Q.begin(I.queue + ((k & 1) * 2 + 1) * 16);
        for (int64_t it = Q.cur; it < total; it = Q.advance(&s_next)) {
            Q.prefetch();
            int64_t local = it;
            int q = 0;
            while (local >= cnt[q]) { local -= cnt[q]; ++q; }
            const PopDev &P = stage_pop(pops, q, sp, cur);
            const int64_t np = ((I.has_plastic >> q) & 1) ? min((int64_t)P.spk_count[k & 1], P.n) * I.post_chunks[q] : 0;
            if (local < np) post_item(P, N, k, local / I.post_chunks[q], local % I.post_chunks[q]);
            else push_spike(P, N, k, local - np, I.inv_dt);
        }
        tl_mark(I, r, 3);
        if (!grid_sync(I, nb, N.flags)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *const_cast<int64_t *>(N.step) += K;
}

template <int CLASS>
const void *persist_fn_t() { return (const void *)k_persistent<CLASS>; }

template const void *persist_fn_t<EB_CLASS>();

}  // namespace eb
