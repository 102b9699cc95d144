// One simulation step of the device-resident network: the update kernels and the
// device code they share with the fan-out and persistent kernels.
//
// Per step k (update time t_k), in stream order:
//   k_input_push   fan out the input-neuron spikes of [t_{k-1}, t_k) into the
//                  arrival buckets of the steps they reach
//   k_update_*     per model population: fold this step's arrivals into the
//                  conductances in the reference's delivery order (arrival time,
//                  then synapse order) with the STDP pre-synaptic update, advance
//                  the neuron one integration step, test the spike condition,
//                  compact the spiking neurons (warp ballot), record them and fan
//                  each spike out into the arrival buckets of its targets (integer
//                  atomics only; the fold sorts, so results do not depend on atomic
//                  order); post-synaptic STDP is deferred (apply_pending)
// The step index is read from device memory (base + offset baked into the
// launch), so one captured CUDA graph of K steps replays for any K steps.
//
// Reference behaviour restated here (paths relative to the reference's Kernel/):
//   delivery g[type] += w then STDP pre hook: src/spike/PropagatedSpikeGroup.cpp:112-149,
//     src/neuron_model/LIFTimeDrivenModel.cpp:77-83
//   STDP: src/learning_rules/STDPWeightChange.cpp:43-76, STDPState.cpp:74-97,
//     include/spike/Interconnection.h:400-407
//   arrival after update at equal time: include/simulation/Event.h:37
//   input-spike delay cascade: src/spike/PropagatedSpike.cpp:60-100
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "eb_device.cuh"
#include "eb_kernels.h"

namespace eb {

__device__ __forceinline__ bool arr_less(const Arrival &x, const Arrival &y) {
    return x.a < y.a || (x.a == y.a && x.spos < y.spos);
}

__device__ __forceinline__ float expt_net(const NetDev &N, float v) {
    if (v >= kExptMin && v <= kExptMax) {
        int pos = (int)((v - kExptMin) * N.expt_aux);
        return __ldg(N.exp_table + pos);
    }
    if (v > kExptMax) return (float)exp((double)v);
    return 0.0f;
}

// STDPWeightChange::ApplyPreSynapticSpike on the record r of a synapse at arrival
// time a (src/learning_rules/STDPWeightChange.cpp:43-56), in place.
__device__ __forceinline__ void stdp_pre_rec(const NetDev &N, SynRec &r, double a) {
    const float *rp = N.rule_par + r.rule * 6;
    float el = (float)(a - r.last);
    float pre = r.pre * expt_net(N, -el * rp[4]);
    float post = r.post * expt_net(N, -el * rp[5]);
    pre += 1.0f;
    float w = r.w;
    w += -rp[2] * post;
    const float mw = r.maxw;
    if (w > mw) w = mw; else if (w < 0.0f) w = 0.0f;
    r.w = w;
    r.pre = pre;
    r.post = post;
    r.last = a;
}

// The same on synapse tp: r is its state as loaded; the updated fields are stored.
__device__ __forceinline__ void stdp_pre(const NetDev &N, uint32_t tp, const SynRec &r, double a) {
    SynRec u = r;
    stdp_pre_rec(N, u, a);
    SynRec *s = N.syn + tp;
    s->w = u.w;
    s->pre = u.pre;
    s->post = u.post;
    s->last = u.last;
}

// STDPWeightChange::ApplyPostSynapticSpike on a synapse record for a spike of its
// target at time t (src/learning_rules/STDPWeightChange.cpp:58-76).
__device__ __forceinline__ void stdp_post(const NetDev &N, SynRec &r, double t) {
    const float *rp = N.rule_par + r.rule * 6;
    const float el = (float)(t - r.last);
    float pre = r.pre * expt_net(N, -el * rp[4]);
    float post = r.post * expt_net(N, -el * rp[5]);
    post += 1.0f;
    float w = r.w + rp[0] * pre;
    if (w > r.maxw) w = r.maxw; else if (w < 0.0f) w = 0.0f;
    r.w = w;
    r.pre = pre;
    r.post = post;
    r.last = t;
}

// Deferred post-synaptic STDP: apply to record r of a plastic synapse onto
// neuron i the target's spikes it has not seen (time > r.last), oldest first --
// the same updates in the same order as at each spike, only later.  Every spike
// of the ring is at most the arrival time being processed (spikes of this step
// are recorded after the fold), and at an equal time the spike came first.
// The ring holds the target's last kPostRing spike times (slot = spike number %
// kPostRing) and, when the population has one plastic rule, the trace decay
// factors of the interval ending at each spike; in global memory (RingGlobal) or
// staged in shared memory (RingSmem).
struct RingGlobal {
    static constexpr bool kLooksAhead = true;
    const double *t;     // the neuron's kPostRing times
    const DecayPair *f;  // and factors
    __device__ double time(uint32_t slot) const { return t[slot]; }
    __device__ DecayPair fac(uint32_t slot) const { return f[slot]; }
};
struct RingSmem {
    static constexpr bool kLooksAhead = false;
    const double *t;
    const DecayPair *f;
    __device__ double time(uint32_t slot) const { return t[slot]; }
    __device__ DecayPair fac(uint32_t slot) const { return f[slot]; }
};

// Apply to r the ring's spikes after r.last, oldest first, as stdp_post would one
// by one.  Spike times increase with the spike number, so the first pending one is
// found by bisection -- after a look at the newest kRingNewest at once when the ring
// is in global memory, where each probe waits for the one before and few spikes are
// pending as a rule.  After the first, r.last is the previous spike, so each
// update's elapsed time -- and its two table lookups -- are the interval's: they
// come from the factor ring when r follows the ring's rule (rule >= 0).
constexpr uint32_t kRingNewest = 4;

template <class Ring>
__device__ __forceinline__ void apply_pending(const NetDev &N, const Ring &ring, uint32_t c, int rule, SynRec &r) {
    const uint32_t lim = c < (uint32_t)kPostRing ? c : (uint32_t)kPostRing;
    uint32_t lo = c - lim, hi = c;  // first spike number in [lo, hi) with time > r.last
    if constexpr (Ring::kLooksAhead) {
        uint32_t n = 0;  // pending among the newest
#pragma unroll
        for (uint32_t q = 1; q <= kRingNewest; ++q)
            if (q <= lim && ring.time((c - q) % kPostRing) > r.last) n = q;
        hi = c - n;
        if (n < kRingNewest) lo = hi;
    }
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (ring.time(mid % kPostRing) > r.last) hi = mid;
        else lo = mid + 1;
    }
    if (lo == c) return;
    stdp_post(N, r, ring.time(lo % kPostRing));
    if (rule >= 0 && r.rule == rule) {
        const float a = N.rule_par[rule * 6];
        float w = r.w, pre = r.pre, post = r.post;
#pragma unroll 4
        for (uint32_t q = lo + 1; q < c; ++q) {
            const DecayPair f = ring.fac(q % kPostRing);
            pre = pre * f.pre;
            post = post * f.post;
            post += 1.0f;
            w = w + a * pre;
            if (w > r.maxw) w = r.maxw; else if (w < 0.0f) w = 0.0f;
        }
        r.w = w;
        r.pre = pre;
        r.post = post;
        r.last = ring.time((c - 1) % kPostRing);
    } else {
        for (uint32_t q = lo + 1; q < c; ++q) stdp_post(N, r, ring.time(q % kPostRing));
    }
}

__device__ __forceinline__ void apply_pending_post(const PopDev &P, const NetDev &N, int64_t i, SynRec &r) {
    const int64_t o = i * kPostRing;
    apply_pending(N, RingGlobal{P.post_t + o, P.post_f ? P.post_f + o : nullptr}, P.post_n[i],
                  P.post_f ? P.post_rule : -1, r);
}

__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// State monitor (the reference's -logp): the state after step k and the spike
// flag of monitored neuron i, at row k % mon_steps.
__device__ __forceinline__ void monitor_state(const PopDev &P, const NetDev &N, int64_t k, int64_t i, const float *x,
                                              int nv, bool sp) {
    const int64_t o = (k % N.mon_steps) * N.mon_n + P.mon_base + i;
    float *d = N.mon_x + o * kMaxVars;
    for (int v = 0; v < nv; ++v) d[v] = x[v];
    N.mon_spk[o] = sp ? 1 : 0;
}

// A delivery of weight w (type ty) into monitored neuron i, folded by step k.
__device__ __forceinline__ void monitor_delivery(const PopDev &P, const NetDev &N, int64_t k, int64_t i,
                                                 const Arrival &v, int ty, float w) {
    const unsigned long long o = atomicAdd(N.mon_count, 1ull);
    if (o < (unsigned long long)N.mon_cap) {
        MonDelivery d;
        d.a = v.a;
        d.spos = v.spos;
        d.cell = (uint32_t)(P.mon_base + i);
        d.w = w;
        d.ty = ty;
        d.k = k;
        N.mon_del[o] = d;
    } else {
        atomicOr(N.flags, FLAG_MONITOR_OVERFLOW);
    }
}

// Monitor hooks: MON 0 compiles them out, 1 keeps them on, 2 asks P.mon at run
// time (the persistent kernel).  The hot kernels are instantiated with 0 and 1:
// a run-time test in the thread-per-neuron update cost the stiff HH network
// 70 % of its step.
template <int MON>
__device__ __forceinline__ bool mon_on(const PopDev &P) { return MON == 1 || (MON == 2 && P.mon != 0); }

template <int ND>
__device__ __forceinline__ void add_conductance(float *x, int ty, float w) {
    if (ty == 0) x[ND] += w;
    else if (ty == 1) x[ND + 1] += w;
    else x[ND + 2] += w;
}

// Apply one arrival at neuron i: g[type] += w (weight before plasticity), then
// STDP pre (after the target's deferred post updates, when it keeps a ring).
template <int ND, int MON = 2>
__device__ __forceinline__ void apply_arrival(const PopDev &P, const NetDev &N, int64_t k, int64_t i, const Arrival &r,
                                              float *x) {
    const uint32_t tp = r.tpos;
    SynRec s = N.syn[tp];
    if (s.rule >= 0 && P.post_t) apply_pending_post(P, N, i, s);
    add_conductance<ND>(x, s.stype, s.w);
    if (mon_on<MON>(P)) monitor_delivery(P, N, k, i, r, s.stype, s.w);
    if (s.rule >= 0) stdp_pre(N, tp, s, r.a);
}

// Record a spike of neuron i at step k for deferred post-synaptic STDP, with the
// decay factors of the interval from its previous spike (stdp_post's lookups for
// a synapse last updated at that spike).
__device__ __forceinline__ void note_post_spike(const PopDev &P, const NetDev &N, int64_t i, int64_t k) {
    const uint32_t c = P.post_n[i];
    const double t = N.tstep[k];
    const int64_t o = i * kPostRing + c % kPostRing;
    if (P.post_f && c > 0) {
        const float *rp = N.rule_par + P.post_rule * 6;
        const float el = (float)(t - P.post_t[i * kPostRing + (c - 1) % kPostRing]);
        P.post_f[o] = DecayPair{expt_net(N, -el * rp[4]), expt_net(N, -el * rp[5])};
    }
    P.post_t[o] = t;
    P.post_n[i] = c + 1;
}

__device__ __forceinline__ int64_t cur_step(const NetDev &N, int rel) { return *N.step + rel + 1; }

// ---------------------------------------------------------------- state io --
template <int KIND>
__device__ __forceinline__ void load_state(const PopDev &P, int64_t i, float *x) {
    constexpr int NV = Model<KIND>::NV;
#pragma unroll
    for (int v = 0; v < NV; ++v) x[v] = P.x[v] ? P.x[v][i] : 0.0f;
}
template <int KIND>
__device__ __forceinline__ void store_state(const PopDev &P, int64_t i, const float *x) {
    constexpr int NV = Model<KIND>::NV;
#pragma unroll
    for (int v = 0; v < NV; ++v) if (P.x[v]) P.x[v][i] = x[v];
}

// Per-neuron integer state next to the variables: LIF updates since the last
// spike, BDF history depth.
struct NeuronAux {
    int refr;
    int bst;
};

template <int KIND, int INTEG>
__device__ __forceinline__ NeuronAux load_aux(const PopDev &P, int64_t i) {
    NeuronAux a;
    a.refr = (KIND == KIND_LIF) ? P.refr[i] : -1;
    a.bst = (INTEG == INTEG_BDF) ? (int)P.bdf_state[i] : 0;
    return a;
}

template <int KIND, int INTEG>
__device__ __forceinline__ void store_aux(const PopDev &P, int64_t i, const NeuronAux &a) {
    if (KIND == KIND_LIF) P.refr[i] = a.refr;
    if (INTEG == INTEG_BDF) P.bdf_state[i] = (int8_t)a.bst;
}

// Advance one neuron (after its arrivals were folded); returns spike flag.  The
// integer state is updated in ax (store_aux writes it back).
template <int KIND, int INTEG, int EN = -1>
__device__ __forceinline__ bool advance_neuron(const PopDev &P, const NetDev &N, int64_t i, float *x, NeuronAux &ax) {
    constexpr int NV = Model<KIND>::NV;
    int refr = ax.refr;
    int bst = ax.bst;
    BdfRef H{P.bdf_D, P.bdf_P, P.n, i};
    const float prevV = x[0];
    if (!integrate<KIND, INTEG, EN>(P, x, refr, bst, H)) atomicOr(N.flags, FLAG_BDF_SINGULAR);
    if (KIND == KIND_LIF && refr >= 0) refr++;  // AddElapsedTime
    bool reset = false;
    const bool sp = spike_condition<KIND>(P, x, prevV, reset);
    if (sp) {
        if (KIND == KIND_LIF) refr = 0;  // NewFiredSpike
        if (reset && INTEG == INTEG_BDF) bst = 0;
    }
    if (__builtin_expect(x[0] != x[0], 0)) {  // CheckValidIntegration: reset a neuron whose V became NaN
#pragma unroll
        for (int v = 0; v < NV; ++v) x[v] = P.init[v];
    }
    ax.refr = refr;
    ax.bst = bst;
    return sp;
}

__device__ __forceinline__ void record_trace(const PopDev &P, const NetDev &N, int64_t k, int64_t gi, const float *x, int nv) {
    if (!N.trace) return;
    int64_t c = gi - N.trace_first, s = k - N.trace_k0;
    if (c < 0 || c >= N.trace_n || s < 0 || s >= N.trace_steps) return;
    float *o = N.trace + (s * N.trace_n + c) * kMaxVars;
    for (int v = 0; v < nv; ++v) o[v] = x[v];
}

// Warp-aggregated append of the spiking lanes to the population spike list (when
// list is set: the persistent kernel, whose eager post-synaptic and
// separate fan-out kernels read) and to the recording buffer.
__device__ __forceinline__ void compact_spikes(const PopDev &P, const NetDev &N, int64_t k, int64_t i, bool sp,
                                               bool list = true) {
    const unsigned full = 0xffffffffu;
    const unsigned m = __ballot_sync(full, sp);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    const unsigned below = m & ((1u << lane) - 1u);
    uint32_t base = 0;
    unsigned long long rbase = 0;
    if (lane == leader) {
        if (list) base = atomicAdd(&P.spk_count[k & 1], (uint32_t)__popc(m));
        if (N.rec_buf) rbase = atomicAdd(N.rec_count, (unsigned long long)__popc(m));
    }
    base = __shfl_sync(full, base, leader);
    rbase = __shfl_sync(full, rbase, leader);
    if (sp) {
        const uint32_t o = base + __popc(below);
        if (!list) {
        } else if (o < (uint32_t)P.n) {
            P.spk[o] = (uint32_t)i;
        } else {
            atomicOr(N.flags, FLAG_SPIKELIST_OVERFLOW);
        }
        if (N.rec_buf) {
            const unsigned long long ro = rbase + __popc(below);
            if (ro < (unsigned long long)N.rec_cap)
                N.rec_buf[ro] = ((unsigned long long)k << 32) | (unsigned long long)(P.first + i);
            else atomicOr(N.flags, FLAG_RECORD_OVERFLOW);
        }
    }
}

// ------------------------------------------------------------ spike fan-out --
// Arrival step of a delivery at time a: the first update time strictly after a
// (never below k_lo).  The guess floor(a/dt)+1 is confirmed by two independent
// table reads in the common case; the loops only run when it is off by rounding.
__device__ __forceinline__ int64_t arrival_step(const NetDev &N, double a, int64_t k_lo, double inv_dt) {
    int64_t ka = (int64_t)(a * inv_dt) + 1;
    if (ka < k_lo) ka = k_lo;
    const double lo = N.tstep[ka - 1], hi = N.tstep[ka];
    if (hi > a && (lo <= a || ka == k_lo)) return ka;
    while (N.tstep[ka] <= a) ++ka;
    while (ka > k_lo && N.tstep[ka - 1] > a) --ka;
    return ka;
}

// Reserve a bucket entry of the target for step ka and store the arrival.
// Loads that do not depend on the reservation are issued before the atomic.
__device__ __forceinline__ void bucket_put(const NetDev &N, int64_t ka, double a, int64_t o) {
    const uint32_t tg = N.out_tgt[o];
    const uint32_t tp = N.out_tpos[o];
    const uint32_t capg = N.cap[tg];
    const int64_t base = N.cap_base[tg];
    const int slot = (int)(ka & (N.R - 1));
    const uint32_t idx = atomicAdd(N.cnt + (int64_t)slot * N.n_neurons + tg, 1u);
    if (idx < capg) {
        Arrival v;
        v.a = a;
        v.spos = (uint32_t)o;
        v.tpos = tp;
        N.rec[(int64_t)slot * N.cap_total + base + idx] = v;
    } else {
        atomicOr(N.flags, FLAG_BUCKET_OVERFLOW);
    }
}

// Fan-out of source neuron src's spike at step k: lanes lane, lane + width, ... of
// the caller's group take its out-synapses (sorted by delay, then target), each
// BATCH at a time: a delivery is a chain of three dependent accesses (synapse, bucket,
// reservation), and a source's deliveries are independent.
template <int BATCH = 1>
__device__ __forceinline__ void push_from(const PopDev &P, const NetDev &N, int64_t k, int64_t src, int lane, int width,
                                          double inv_dt) {
    const double tk = P.kind == KIND_POISSON ? N.tgen[k] : N.tstep[k];  // generators spike on their own grid
    const int64_t o0 = N.out_ptr[src], o1 = N.out_ptr[src + 1];
    for (int64_t o = o0 + lane; o < o1; o += BATCH * width) {
        uint32_t tg[BATCH];
        Arrival v[BATCH];
        int slot[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int64_t q = o + u * width;
            if (q >= o1) continue;
            tg[u] = N.out_tgt[q];
            v[u].a = tk + (double)N.out_units[q] * 0.0001;
            v[u].spos = (uint32_t)q;
            v[u].tpos = N.out_tpos[q];
        }
        uint32_t capg[BATCH];
        int64_t base[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            if (o + u * width >= o1) continue;
            capg[u] = N.cap[tg[u]];
            base[u] = N.cap_base[tg[u]];
            slot[u] = (int)(arrival_step(N, v[u].a, k + 1, inv_dt) & (N.R - 1));
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u)
            if (o + u * width < o1) tg[u] = atomicAdd(N.cnt + (int64_t)slot[u] * N.n_neurons + tg[u], 1u);
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            if (o + u * width >= o1) continue;
            if (tg[u] < capg[u]) N.rec[(int64_t)slot[u] * N.cap_total + base[u] + tg[u]] = v[u];
            else atomicOr(N.flags, FLAG_BUCKET_OVERFLOW);
        }
    }
}

__device__ __forceinline__ void push_spike(const PopDev &P, const NetDev &N, int64_t k, int64_t s, double inv_dt) {
    push_from(P, N, k, P.first + P.spk[s], threadIdx.x, blockDim.x, inv_dt);
}

// Fan-out inside the update kernel (graph path): a spike at step k only reaches
// buckets of steps >= k+1, which no kernel of this step reads, so the spiking
// warp delivers it at once instead of a separate launch after the update.  The
// warp takes its spiking lanes one at a time, lanes over the out-synapses.
template <int BATCH = 1>
__device__ __forceinline__ void warp_push(const PopDev &P, const NetDev &N, int64_t k, int64_t i, bool sp,
                                          double inv_dt) {
    unsigned m = __ballot_sync(0xffffffffu, sp);
    const int lane = threadIdx.x & 31;
    while (m) {
        const int l = __ffs(m) - 1;
        m &= m - 1u;
        const int64_t src = P.first + __shfl_sync(0xffffffffu, i, l);
        push_from<BATCH>(P, N, k, src, lane, 32, inv_dt);
    }
}

// Asynchronous global -> shared copies (cp.async), complete at cp_async_wait_all
// (and a barrier of the threads that read them).
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// ----------------------------------------------------------- narrow update --
// One thread per neuron.  Arrivals of this step are sorted in registers
// (insertion sort; at most 16 in the fast path) and folded in order.
constexpr int kLocalSort = 16;
constexpr int kNarrowTile = 256;   // threads of the persistent kernel's tiles
constexpr int kNarrowBlock = 64;   // most threads of a block of k_update_narrow
// Steps of one launch (the runtime's window length).
constexpr int kMaxWindow = 8;

// The arrivals of step k at neuron i, from its bucket, onto x; returns their number.
template <int ND, int MON>
__device__ __forceinline__ uint32_t narrow_fold(const PopDev &P, const NetDev &N, int64_t k, int64_t i, float *x) {
    const int64_t gi = P.first + i;
    const int slot = (int)(k & (N.R - 1));
    uint32_t *cp = N.cnt + (int64_t)slot * N.n_neurons + gi;
    uint32_t c = *cp;
    if (c) {
        *cp = 0;
        const uint32_t capg = N.cap[gi];
        if (c > capg) { atomicOr(N.flags, FLAG_BUCKET_OVERFLOW); c = capg; }
        Arrival *r = N.rec + (int64_t)slot * N.cap_total + N.cap_base[gi];
        if (c == 1) {
            apply_arrival<ND, MON>(P, N, k, i, r[0], x);
        } else if (c <= kLocalSort) {
            Arrival loc[kLocalSort];
            for (uint32_t a = 0; a < c; ++a) {
                Arrival v = r[a];
                int b = (int)a - 1;
                while (b >= 0 && arr_less(v, loc[b])) { loc[b + 1] = loc[b]; --b; }
                loc[b + 1] = v;
            }
            for (uint32_t a = 0; a < c; ++a) apply_arrival<ND, MON>(P, N, k, i, loc[a], x);
        } else {
            for (uint32_t a = 1; a < c; ++a) {  // in-place insertion sort (rare path)
                Arrival v = r[a];
                int b = (int)a - 1;
                while (b >= 0 && arr_less(v, r[b])) { r[b + 1] = r[b]; --b; }
                r[b + 1] = v;
            }
            for (uint32_t a = 0; a < c; ++a) apply_arrival<ND, MON>(P, N, k, i, r[a], x);
        }
    }
    return c;
}

// Delivered-event counter: one atomic per warp.
__device__ __forceinline__ void count_events(const PopDev &P, uint32_t c) {
    if (__any_sync(0xffffffffu, c != 0)) {
        unsigned long long cw = c;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cw += __shfl_down_sync(0xffffffffu, cw, o);
        if ((threadIdx.x & 31) == 0 && cw) atomicAdd(P.events, cw);
    }
}

// One step of neuron i (lanes with active unset only join the warp collectives);
// x and ax hold its state, loaded and stored by the caller.
template <int KIND, int INTEG, int EN = -1, int MON = 2>
__device__ __forceinline__ void narrow_step(const PopDev &P, const NetDev &N, int64_t k, int64_t i, bool active,
                                            float *x, NeuronAux &ax, bool list, double push_inv_dt) {
    bool sp = false;
    uint32_t c = 0;
    if (active) {
        c = narrow_fold<Model<KIND>::ND, MON>(P, N, k, i, x);
        sp = advance_neuron<KIND, INTEG, EN>(P, N, i, x, ax);
        record_trace(P, N, k, P.first + i, x, Model<KIND>::NV);
        if (mon_on<MON>(P)) monitor_state(P, N, k, i, x, Model<KIND>::NV, sp);
        if (sp && P.post_t) note_post_spike(P, N, i, k);
    }
    count_events(P, c);
    compact_spikes(P, N, k, i, sp, list);
    if (push_inv_dt > 0.0) warp_push(P, N, k, i, sp, push_inv_dt);
}

template <int KIND, int INTEG>
__device__ __forceinline__ void update_narrow_tile(const PopDev &P, const NetDev &N, int64_t k, int64_t tile,
                                                   double push_inv_dt = 0.0) {
    const int64_t i = tile * kNarrowTile + threadIdx.x;
    const bool active = i < P.n;
    float x[kMaxVars];
    NeuronAux ax{-1, 0};
    if (active) {
        load_state<KIND>(P, i, x);
        ax = load_aux<KIND, INTEG>(P, i);
    }
    narrow_step<KIND, INTEG>(P, N, k, i, active, x, ax, true, push_inv_dt);
    if (active) {
        store_state<KIND>(P, i, x);
        store_aux<KIND, INTEG>(P, i, ax);
    }
}

// ------------------------------------------------------ staged narrow window --
// The steps of one launch for the neurons of one warp, with the window's arrivals
// taken in at once.  Every bucket of the window is final when the launch starts, so
// the warp reads the counts of all its steps, copies the arrivals of as many
// consecutive steps as its stage holds into shared memory, each lane its neuron's,
// step by step, and sorts each step's few in delivery order.  That leaves three
// dependent global accesses (count, arrival, synapse) a window where the per-step
// fold waited for them at every step, one arrival after the other.
//   Populations without plastic inputs: all staged arrivals' weights are fetched
// together, a step's fold only reads shared memory.
//   With plastic inputs: a step's arrivals are dealt out to the lanes, whoever's
// neuron they reach, and every lane catches its synapse up on the target's
// post-synaptic spikes, takes the weight and applies the pre-synaptic update;
// the owner then adds the weights in order.  Synapses are independent unless one
// delivers twice in the step (input neurons only): then the step folds serially.
// A step with more arrivals than the stage holds runs on the per-step path.
//   Bound by the latency of the warp's chain: 1,000 LIF neurons, 3,000 steps 4.37 ->
// 3.32 ms; 2,501 AdEx neurons with STDP, 500 steps 3.62 -> 2.42 ms; HH, 3,001 neurons
// 12.9 -> 11.8 us a step, 100,000 29.7 -> 28.2.  Large LIF and AdEx populations are
// bound by issue, and the staging spills 250 bytes at their registers: they keep the
// per-step fold (250,000 granule cells at 40 registers: 5.98 us a step, 6.16 staged).
template <int CAP>
struct NarrowStage {
    Arrival arr[CAP];
    float w[CAP];
    uint16_t list[CAP];  // a step's arrivals: owner lane << 8 | position
    uint8_t ty[CAP];
};
// Arrivals of a warp's stage: HH under BDF runs few, long-lived warps of neurons with
// many inputs; the others keep the shared memory of 48 warps an SM below half of it.
__host__ __device__ constexpr int narrow_stage(int kind) { return kind == KIND_HH ? 128 : 64; }
static_assert(kMaxWindow <= 8, "a lane packs a window's counts into 8 bytes");

template <int KIND, int INTEG, int EN, int MON, bool SMALL, bool PLASTIC, int CAP>
__device__ __forceinline__ void narrow_window(const PopDev &P, const NetDev &N, int64_t k, int64_t i, bool active,
                                              float *x, NeuronAux &ax, int nsteps, double push_inv_dt,
                                              NarrowStage<CAP> &S) {
    constexpr int ND = Model<KIND>::ND;
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t gi = P.first + i;
    constexpr bool plastic = PLASTIC;
    const bool fan_out = push_inv_dt > 0.0;
    const bool traced = N.trace && gi >= N.trace_first && gi < N.trace_first + N.trace_n;
    // counts of the steps not yet run, a byte each (255: that many or more), next step lowest
    unsigned long long pk = 0;
    uint32_t capg = 0;
    const Arrival *rec = nullptr;
    if (active) {
#pragma unroll
        for (int s = 0; s < kMaxWindow; ++s)
            if (s < nsteps) {
                const uint32_t c = N.cnt[(int64_t)((k + s) & (N.R - 1)) * N.n_neurons + gi];
                pk |= (unsigned long long)(c < 255u ? c : 255u) << (8 * s);
            }
        if (pk) {
            capg = N.cap[gi];
            rec = N.rec + N.cap_base[gi];
        }
    }
    int staged = 0;      // steps left of the staged chunk
    uint32_t pos = 0;    // this lane's next staged arrival
    for (int s = 0; s < nsteps; ++s) {
        const int64_t ks = k + s;
        if (staged == 0) {

            if (__any_sync(full, pk != 0)) {
                int len = nsteps - s;
                uint32_t tot, incl, T;
                for (;;) {
                    tot = 0;
                    for (int q = 0; q < len; ++q) {
                        const uint32_t c = (uint32_t)(pk >> (8 * q)) & 255u;
                        tot += c == 255u || c > capg ? CAP + 1 : c;
                    }
                    incl = tot;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t u = __shfl_up_sync(full, incl, o);
                        if (lane >= o) incl += u;
                    }
                    T = __shfl_sync(full, incl, 31);
                    if (T <= (uint32_t)CAP || len == 1) break;
                    len >>= 1;
                }
                staged = len;
                pos = incl - tot;
                const bool direct = T > (uint32_t)CAP;  // this step alone overflows the stage (or a bucket)
                if (direct) {
                    count_events(P, active ? narrow_fold<ND, MON>(P, N, ks, i, x) : 0u);
                    pk &= ~255ull;
                } else if (T) {
                    __syncwarp();  // every lane is done with the last chunk
                    uint32_t j = pos;
                    if (tot)
                        for (int q = 0; q < len; ++q) {
                            const uint32_t c = (uint32_t)(pk >> (8 * q)) & 255u;
                            if (!c) continue;
                            const int slot = (int)((ks + q) & (N.R - 1));
                            const Arrival *r = rec + (int64_t)slot * N.cap_total;
                            for (uint32_t a = 0; a < c; ++a) cp_async16(&S.arr[j++], r + a);
                            N.cnt[(int64_t)slot * N.n_neurons + gi] = 0;
                        }
                    cp_async_commit();
                    if (lane == 0) atomicAdd(P.events, (unsigned long long)T);
                    cp_async_wait_all();
                    j = pos;
                    if (tot)
                        for (int q = 0; q < len; ++q) {  // each step's arrivals in delivery order
                            const uint32_t c = (uint32_t)(pk >> (8 * q)) & 255u;
                            for (uint32_t a = 1; a < c; ++a) {
                                const Arrival v = S.arr[j + a];
                                uint32_t b = a;
                                while (b > 0 && arr_less(v, S.arr[j + b - 1])) { S.arr[j + b] = S.arr[j + b - 1]; --b; }
                                if (b != a) S.arr[j + b] = v;
                            }
                            j += c;
                        }
                    __syncwarp();
                    for (uint32_t e = lane; e < T; e += 32) {
                        const SynRec *r = N.syn + S.arr[e].tpos;
                        if (plastic) {
                            prefetch_l1(r);
                        } else {
                            S.w[e] = r->w;
                            S.ty[e] = r->stype;
                        }
                    }
                    __syncwarp();
                }
            } else {
                staged = nsteps - s;  // no arrival in the rest of the window
            }
        }
        --staged;
        const uint32_t c = (uint32_t)pk & 255u;
        pk >>= 8;
        bool serial = false;  // a synapse delivers twice in this step
        if (plastic && __any_sync(full, c != 0)) {
            if (P.may_repeat) {
                bool twice = false;
                for (uint32_t a = 1; a < c; ++a)
                    for (uint32_t b = 0; b < a; ++b) twice = twice || S.arr[pos + a].spos == S.arr[pos + b].spos;
                serial = __any_sync(full, twice);
            }
            if (!serial) {
                uint32_t incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t u = __shfl_up_sync(full, incl, o);
                    if (lane >= o) incl += u;
                }
                const uint32_t T = __shfl_sync(full, incl, 31);
                for (uint32_t a = 0; a < c; ++a) S.list[incl - c + a] = (uint16_t)(lane << 8 | (pos + a));
                __syncwarp();
                for (uint32_t e = lane; e < T; e += 32) {
                    const uint32_t at = S.list[e];
                    const Arrival v = S.arr[at & 255u];
                    SynRec r = N.syn[v.tpos];
                    if (r.rule >= 0) apply_pending_post(P, N, i - lane + (at >> 8), r);
                    S.w[at & 255u] = r.w;
                    S.ty[at & 255u] = r.stype;
                    if (r.rule >= 0) stdp_pre(N, v.tpos, r, v.a);
                }
                __syncwarp();
            }
        }
        bool sp = false;
        if (active) {
            if (serial) {
                for (uint32_t a = 0; a < c; ++a) apply_arrival<ND, MON>(P, N, ks, i, S.arr[pos + a], x);
            } else {
                for (uint32_t a = 0; a < c; ++a) {
                    add_conductance<ND>(x, S.ty[pos + a], S.w[pos + a]);
                    if (mon_on<MON>(P)) monitor_delivery(P, N, ks, i, S.arr[pos + a], S.ty[pos + a], S.w[pos + a]);
                }
            }
            pos += c;
            sp = advance_neuron<KIND, INTEG, EN>(P, N, i, x, ax);
            if (traced) record_trace(P, N, ks, gi, x, Model<KIND>::NV);
            if (mon_on<MON>(P)) monitor_state(P, N, ks, i, x, Model<KIND>::NV, sp);
            if (sp && plastic) note_post_spike(P, N, i, ks);
        }
        if (__any_sync(full, sp)) {
            compact_spikes(P, N, ks, i, sp, false);
            if (fan_out) warp_push<SMALL ? 4 : 1>(P, N, ks, i, sp, push_inv_dt);
        }
    }
}

// Steps k .. k+nsteps-1 of one tile, the state in registers between them.
// push_inv_dt > 0: also fan out the spikes (1 / step, for arrival_step).
// PLASTIC: the population keeps a post-synaptic spike ring; the staged window of one that
// does not is half the code, and a warp alone on its sub-partition waits for code.
// SMALL: registers are not bounded and a warp keeps more accesses of a fan-out in
// flight (populations that fit the SMs all the same, see eb_update.cu).
// HH under BDF holds the Newton state (Jacobian, inverse, history) in about 120
// registers, which leaves 2 blocks per SM; bounded to 3 blocks (80 registers, a
// 44-byte spill) a 100k-neuron population fits one wave and its steps take a
// quarter less time.  LIF and AdEx under the explicit methods are bounded to 5
// blocks of 256 (48 registers): they are bound by issue, and at 40 registers a fifth
// of the instructions re-read parameters (250,000 granule cells beside 40 Purkinje
// cells: 5.96 us a step at 40 registers, 5.38 at 48, 5.46 at 54).
// EN >= 0: the population's enabled conductance types fixed at compile time.
constexpr int narrow_min_blocks(int kind, int integ) {
    return (kind == KIND_HH && integ == INTEG_BDF) ? 3 : (kind != KIND_HH && integ != INTEG_BDF) ? 5 : 0;
}

template <int KIND, int INTEG, int EN, int MON, bool SMALL, bool PLASTIC>
__global__ void __launch_bounds__(kNarrowBlock, SMALL ? 1 : narrow_min_blocks(KIND, INTEG) * (kNarrowTile / kNarrowBlock)) k_update_narrow(PopDev P, NetDev N, int rel, int nsteps,
                                                                double push_inv_dt, int npw) {
    const int64_t k = cur_step(N, rel);
    __shared__ NarrowStage<SMALL || KIND == KIND_HH ? narrow_stage(KIND) : 1> stage[kNarrowBlock / 32];
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * npw + lane;
    const bool active = lane < npw && i < P.n;
    float x[kMaxVars];
    NeuronAux ax{-1, 0};
    if (active) {
        load_state<KIND>(P, i, x);
        ax = load_aux<KIND, INTEG>(P, i);
    }
    if constexpr (SMALL || KIND == KIND_HH) {
        narrow_window<KIND, INTEG, EN, MON, SMALL, PLASTIC>(P, N, k, i, active, x, ax, nsteps, push_inv_dt, stage[threadIdx.x >> 5]);
    } else {
        for (int s = 0; s < nsteps; ++s)
            narrow_step<KIND, INTEG, EN, MON>(P, N, k + s, i, active, x, ax, false, push_inv_dt);
    }
    if (active) {
        store_state<KIND>(P, i, x);
        store_aux<KIND, INTEG>(P, i, ax);
    }
}

// ------------------------------------------------------------- wide update --
// One block per neuron, for populations whose neurons receive many arrivals per
// step (e.g. Purkinje-like cells with 10^4-10^5 inputs).
//
// Up to kRankSort arrivals, every arrival finds its delivery position by counting
// the arrivals ordered before it -- (time, synapse order) compared as integers,
// since the bits of a non-negative double order like its value -- with all the
// block's threads sharing the comparisons.  Each arrival's synapse record is
// fetched while the positions are counted, its STDP pre-synaptic update applied
// in parallel (synapses are independent; a synapse that can arrive twice in one
// step -- only from input neurons -- forces the serial path) and its weight stored
// at its position; one thread per conductance then adds the weights in delivery
// order.  Up to kWideSmem arrivals: bitonic sort in shared memory; beyond, a
// serial insertion sort in global memory.
// A 512-arrival stage keeps a block at about 70 KB of shared memory, so three
// fit an SM (85 registers a thread): the wide population packs onto fewer SMs
// and leaves the others whole to the thread-per-neuron populations.
constexpr int kWideThreads = 256;
constexpr int kWideSmem = 1024;
constexpr int kRankSort = 256;
static_assert(kRankSort <= kWideThreads && kWideThreads <= kNarrowTile, "wide blocks rank with one thread per arrival");

struct WideSmem {
    int spiked;                         // the block's neuron spiked this step (fused fan-out)
    int ring_ok;                        // ring, ring_f and ring_n hold the neuron's ring
    uint32_t ring_n;                    // post-synaptic spikes noted so far (deferred STDP)
    uint32_t next_c;                    // next step's arrival count (copied ahead)
    float g[3];                         // conductances handed to the per-type adders
    uint32_t wcnt[kMaxWindow];          // staged window: arrivals of each step
    uint32_t woff[kMaxWindow + 1];      // and their offsets (exclusive scan)
    unsigned long long kmin[kMaxWindow];  // smallest and largest time key of each step's arrivals
    unsigned long long kmax[kMaxWindow];
    int dup;                            // a synapse of the staged chunk delivers twice
    int next_s;                         // first step of the chunk's next round
    unsigned long long khi[kRankSort];  // arrival time keys
    uint32_t klo[kRankSort];            // synapse order
    uint32_t rank[kRankSort];           // delivery position
    double ring[kPostRing];             // the neuron's deferred post-synaptic spike times
    DecayPair ring_f[kPostRing];           // and the decay factors of their intervals
    Arrival next_rec[kRankSort];        // next step's first arrivals (copied ahead)
    Arrival sbuf[kWideSmem];
    float sw[kWideSmem];
    uint8_t sty[kWideSmem];
};

// Copy step k's arrival count and its first n records (n <= the neuron's bucket
// capacity) of neuron gi into S.next_c / S.next_rec.  Only for a step whose
// bucket is final: a later step of the same launch (every delivery into it comes
// from steps before the launch, or from input fan-out that precedes it).
__device__ __forceinline__ void wide_prefetch(const NetDev &N, WideSmem &S, int64_t k, int64_t gi, int64_t rbase,
                                              int n) {
    const int slot = (int)(k & (N.R - 1));
    const Arrival *r = N.rec + (int64_t)slot * N.cap_total + rbase;
    for (int a = threadIdx.x; a < n; a += blockDim.x) cp_async16(&S.next_rec[a], r + a);
    if (threadIdx.x == 0) cp_async4(&S.next_c, N.cnt + (int64_t)slot * N.n_neurons + gi);
    cp_async_commit();
}

// Order-preserving integer key of an arrival time (-0 folded into +0).
__device__ __forceinline__ unsigned long long time_key(double a) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(a + 0.0);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// STDP pre hook for one arrival with every synapse load issued up front (they
// only depend on tp); returns the weight before the update through w_old.
__device__ __forceinline__ void stdp_pre_gather(const PopDev &P, const NetDev &N, int64_t i, uint32_t tp, double a,
                                                float &w_old, int &ty) {
    SynRec r = N.syn[tp];
    if (r.rule >= 0 && P.post_t) apply_pending_post(P, N, i, r);
    w_old = r.w;
    ty = r.stype;
    if (r.rule < 0) return;
    stdp_pre(N, tp, r, a);
}

// Add the c weights sw[] (types sty[]) to the conductances x[ND..ND+2] in order.
// Each conductance only sees its own type's weights, in order, so one thread per
// type (lane 0 of warps 0-2) adding its type's weights reproduces the interleaved
// sequential sum.  Thread 0 owns x; block-wide, with barriers.
template <int ND>
__device__ __forceinline__ void wide_fold(WideSmem &S, float *x, uint32_t c) {
    const int tid = threadIdx.x;
    if (tid == 0) { S.g[0] = x[ND]; S.g[1] = x[ND + 1]; S.g[2] = x[ND + 2]; }
    __syncthreads();
    const int T = tid >> 5;
    if ((tid & 31) == 0 && T < 3) {
        float g = S.g[T];
        uint32_t a = 0;
        for (; a + 8 <= c; a += 8) {
            float w[8];
            int t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) { w[u] = S.sw[a + u]; t[u] = S.sty[a + u]; }
#pragma unroll
            for (int u = 0; u < 8; ++u) g = ((t[u] < 2 ? t[u] : 2) == T) ? g + w[u] : g;
        }
        for (; a < c; ++a) {
            const int t = S.sty[a];
            g = ((t < 2 ? t : 2) == T) ? g + S.sw[a] : g;
        }
        S.g[T] = g;
    }
    __syncthreads();
    if (tid == 0) { x[ND] = S.g[0]; x[ND + 1] = S.g[1]; x[ND + 2] = S.g[2]; }
}

// One step of wide neuron i by the whole block; thread 0 holds its state in x and
// ax (loaded and stored by the caller).
template <int KIND, int INTEG, int MON = 2, int EN = -1>
// pf_n: records of this step already copied to S.next_rec (with the count in
// S.next_c; 0: none), updated for the next step when has_next (the next step is
// in the same launch).
__device__ __forceinline__ void wide_step(const PopDev &P, const NetDev &N, int64_t k, int64_t i, WideSmem &S,
                                          float *x, NeuronAux &ax, bool list, double push_inv_dt, int &pf_n,
                                          bool has_next) {
    constexpr int ND = Model<KIND>::ND;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int slot = (int)(k & (N.R - 1));
    const int64_t gi = P.first + i;
    if (pf_n > 0) cp_async_wait_all();
    __syncthreads();  // the block's previous step is done with S; copied arrivals visible
    // every load that does not depend on another goes out first
    uint32_t *cp = N.cnt + (int64_t)slot * N.n_neurons + gi;
    uint32_t c = pf_n > 0 ? S.next_c : *cp;
    const uint32_t capg = N.cap[gi];
    const int64_t rbase = N.cap_base[gi];
    int next_n = 0;
    // after a barrier that follows every thread's read of S.next_*: copy the next
    // step's count and about as many records as this step had
    auto issue_next = [&]() {
        if (!has_next) return;
        const uint32_t guess = ((c + c / 2 + 32) + 31) / 32 * 32;
        next_n = (int)min(min(guess, capg), (uint32_t)kRankSort);
        wide_prefetch(N, S, k + 1, gi, rbase, next_n);
    };
    if (c) {
        if (c > capg) { if (tid == 0) atomicOr(N.flags, FLAG_BUCKET_OVERFLOW); c = capg; }
        Arrival *r = N.rec + (int64_t)slot * N.cap_total + rbase;
        if (c <= (uint32_t)kRankSort) {
            const bool own = tid < (int)c;
            const bool ring = P.post_t != nullptr && !P.may_repeat;
            Arrival v;
            SynRec rec;
            if (own) {
                v = tid < pf_n ? S.next_rec[tid] : r[tid];
                if (!P.may_repeat) rec = N.syn[v.tpos];  // in flight while the positions are counted
                S.khi[tid] = time_key(v.a);
                S.klo[tid] = v.spos;
                S.rank[tid] = 0;
            }
            if (ring && !S.ring_ok) {  // the neuron's deferred post-synaptic spikes (slots past the count are unused)
                for (int q = tid; q < kPostRing; q += nt) {
                    S.ring[q] = P.post_t[i * kPostRing + q];
                    if (P.post_f) S.ring_f[q] = P.post_f[i * kPostRing + q];
                }
                if (tid == nt - 1) S.ring_n = P.post_n[i];
            }
            if (tid == 32) prefetch_l1(N.rule_par);
            __syncthreads();
            if (tid == 0) {
                *cp = 0;
                if (ring) S.ring_ok = 1;
            }
            issue_next();
            // position = arrivals before this one in (time, synapse order, bucket index)
            // order; per threads share each arrival's comparisons
            const int per = nt / (int)c;
            if (tid < per * (int)c) {
                const int e = tid % (int)c, s = tid / (int)c;
                const int b0 = s * (int)c / per, b1 = (s + 1) * (int)c / per;
                const unsigned long long kh = S.khi[e];
                const uint32_t kl = S.klo[e];
                uint32_t n = 0;
#pragma unroll 4
                for (int b = b0; b < b1; ++b) {
                    const unsigned long long uh = S.khi[b];
                    const uint32_t ul = S.klo[b];
                    n += (uh < kh || (uh == kh && (ul < kl || (ul == kl && b < e)))) ? 1u : 0u;
                }
                if (per == 1) S.rank[e] = n;
                else if (n) atomicAdd(&S.rank[e], n);
            }
            __syncthreads();
            if (P.may_repeat) {
                if (own) S.sbuf[S.rank[tid]] = v;
                __syncthreads();
                if (tid == 0)
                    for (uint32_t a = 0; a < c; ++a) apply_arrival<ND, MON>(P, N, k, i, S.sbuf[a], x);
            } else {
                if (own) {
                    if (rec.rule >= 0) {
                        if (ring) apply_pending(N, RingSmem{S.ring, S.ring_f}, S.ring_n, P.post_f ? P.post_rule : -1, rec);
                        S.sw[S.rank[tid]] = rec.w;
                        stdp_pre(N, v.tpos, rec, v.a);
                    } else {
                        S.sw[S.rank[tid]] = rec.w;
                    }
                    S.sty[S.rank[tid]] = rec.stype;
                    if (mon_on<MON>(P)) monitor_delivery(P, N, k, i, v, rec.stype, S.sw[S.rank[tid]]);
                }
                wide_fold<ND>(S, x, c);
            }
        } else if (c <= (uint32_t)kWideSmem) {
            int n2 = 1;
            while (n2 < (int)c) n2 <<= 1;
            for (int a = tid; a < n2; a += nt) {
                if (a < (int)c) S.sbuf[a] = r[a];
                else { S.sbuf[a].a = __longlong_as_double(0x7ff0000000000000LL); S.sbuf[a].spos = 0xffffffffu; S.sbuf[a].tpos = 0; }
            }
            __syncthreads();
            if (tid == 0) *cp = 0;
            issue_next();
            for (int size = 2; size <= n2; size <<= 1)
                for (int stride = size >> 1; stride > 0; stride >>= 1) {
                    for (int a = tid; a < n2; a += nt) {
                        const int b = a ^ stride;
                        if (b > a) {
                            const bool up = ((a & size) == 0);
                            const Arrival ea = S.sbuf[a], eb = S.sbuf[b];
                            if (up ? arr_less(eb, ea) : arr_less(ea, eb)) { S.sbuf[a] = eb; S.sbuf[b] = ea; }
                        }
                    }
                    __syncthreads();
                }
            if (P.may_repeat) {
                if (tid == 0)
                    for (uint32_t a = 0; a < c; ++a) apply_arrival<ND, MON>(P, N, k, i, S.sbuf[a], x);
            } else {
                for (int a = tid; a < (int)c; a += nt) {
                    const Arrival v = S.sbuf[a];
                    float w_old;
                    int ty;
                    stdp_pre_gather(P, N, i, v.tpos, v.a, w_old, ty);
                    S.sw[a] = w_old;
                    S.sty[a] = (uint8_t)ty;
                    if (mon_on<MON>(P)) monitor_delivery(P, N, k, i, v, ty, w_old);
                }
                __syncthreads();
                wide_fold<ND>(S, x, c);
            }
        } else {
            __syncthreads();  // every thread has read the count before it is cleared
            issue_next();
            if (tid == 0) {
                *cp = 0;
                for (uint32_t a = 1; a < c; ++a) {  // rare: insertion sort in global memory
                    Arrival v = r[a];
                    int b = (int)a - 1;
                    while (b >= 0 && arr_less(v, r[b])) { r[b + 1] = r[b]; --b; }
                    r[b + 1] = v;
                }
                for (uint32_t a = 0; a < c; ++a) apply_arrival<ND, MON>(P, N, k, i, r[a], x);
            }
        }
        if (tid == 0) atomicAdd(P.events, (unsigned long long)c);
    } else if (has_next) {
        __syncthreads();  // every thread has read S.next_c
        issue_next();
    }
    if (tid == 0) {
        const bool sp = advance_neuron<KIND, INTEG, EN>(P, N, i, x, ax);
        S.spiked = sp ? 1 : 0;
        if (sp && P.post_t) {
            note_post_spike(P, N, i, k);
            if (S.ring_ok) {  // keep the staged ring current
                const uint32_t n1 = P.post_n[i], q = (n1 - 1) % kPostRing;
                S.ring_n = n1;
                S.ring[q] = P.post_t[i * kPostRing + q];
                if (P.post_f) S.ring_f[q] = P.post_f[i * kPostRing + q];
            }
        }
        record_trace(P, N, k, gi, x, Model<KIND>::NV);
        if (mon_on<MON>(P)) monitor_state(P, N, k, i, x, Model<KIND>::NV, sp);
        if (sp) {
            if (list) {
                const uint32_t o = atomicAdd(&P.spk_count[k & 1], 1u);
                if (o < (uint32_t)P.n) P.spk[o] = (uint32_t)i;
                else atomicOr(N.flags, FLAG_SPIKELIST_OVERFLOW);
            }
            if (N.rec_buf) {
                const unsigned long long ro = atomicAdd(N.rec_count, 1ull);
                if (ro < (unsigned long long)N.rec_cap)
                    N.rec_buf[ro] = ((unsigned long long)k << 32) | (unsigned long long)gi;
                else atomicOr(N.flags, FLAG_RECORD_OVERFLOW);
            }
        }
    }
    __syncthreads();
    if (push_inv_dt > 0.0 && S.spiked) push_from(P, N, k, gi, tid, blockDim.x, push_inv_dt);
    pf_n = next_n;
}

template <int KIND, int INTEG>
__device__ __forceinline__ void update_wide_neuron(const PopDev &P, const NetDev &N, int64_t k, int64_t i, WideSmem &S,
                                                   double push_inv_dt = 0.0) {
    float x[kMaxVars];
    NeuronAux ax{-1, 0};
    if (threadIdx.x == 0) {
        load_state<KIND>(P, i, x);
        ax = load_aux<KIND, INTEG>(P, i);
        S.ring_ok = 0;
    }
    int pf_n = 0;
    wide_step<KIND, INTEG>(P, N, k, i, S, x, ax, true, push_inv_dt, pf_n, false);
    if (threadIdx.x == 0) {
        store_state<KIND>(P, i, x);
        store_aux<KIND, INTEG>(P, i, ax);
    }
}

// ------------------------------------------------------ staged wide window --
// A launch's window of steps for one wide neuron with every delivery of the
// window taken in at once.  All buckets of the window's steps are final when the
// launch starts, so the block stages the arrivals of as many consecutive steps as
// fit in shared memory (a chunk) and every arrival's delivery position within its
// step, in parallel: a few dependent global round trips per chunk instead of per
// step.  When every synapse of the chunk delivers once (the usual case), the
// chunk's steps run in rounds: the whole block computes, in parallel, every
// remaining arrival's synapse update -- deferred post-synaptic catch-up on the
// target's spikes so far and the delivered weight at its position -- then warp 0
// runs the steps in order (ordered sums, integration, spike, fan-out) until the
// neuron spikes.  A spike adds one update to the catch-up of the later arrivals:
// the next round applies it to their staged records.  The STDP pre updates are
// applied as the chunk writes its records back.  A chunk in which a synapse
// delivers on two steps runs its steps serially on warp 0 over one staged record
// per synapse; a step with more arrivals than the stage holds runs on the
// per-step path (wide_step).
constexpr int kStage = 512;           // arrivals of one chunk
constexpr int kStageHashBits = 10;    // open-addressing table of the chunk's synapses
constexpr int kStageHash = 1 << kStageHashBits;
constexpr uint32_t kHashEmpty = 0xffffffffu;
static_assert(kStage <= kWideSmem, "a staged chunk's weights fit the fold buffer");

struct StageSmem {
    Arrival arr[kStage];               // the chunk's arrivals, step by step in bucket order
    SynRec rec[kStage];                // updated synapse records (serial path: at the owning arrival)
    unsigned long long key[kStage];    // order-preserving integer key of each arrival time
    uint32_t hkey[kStageHash];         // tpos of the synapse claiming a slot
    uint16_t hval[kStageHash];         // its owning arrival
    uint16_t own[kStage];              // per arrival: the arrival whose staged record it uses
    uint16_t rank[kStage];             // per arrival: delivery position within its step
};

__host__ __device__ constexpr size_t stage_smem_bytes() { return sizeof(StageSmem); }

__device__ __forceinline__ int stage_step_of(const WideSmem &S, int s0, uint32_t g) {
    int s = s0;
    while (S.woff[s + 1] <= g) ++s;
    return s;
}

// Sum of the c weights sw[o0..o0+c) onto g in order, loads issued 8 at a time.
__device__ __forceinline__ float ordered_sum1(const WideSmem &S, uint32_t o0, uint32_t c, float g) {
    uint32_t q = 0;
    for (; q + 8 <= c; q += 8) {
        float w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) w[u] = S.sw[o0 + q + u];
#pragma unroll
        for (int u = 0; u < 8; ++u) g += w[u];
    }
    for (; q < c; ++q) g += S.sw[o0 + q];
    return g;
}

// Add the c weights sw[o0..o0+c) (types sty[]) to the conductances x[ND..ND+2] in
// order: each conductance sees its own type's weights in delivery order, as the
// reference's successive additions.  A population with one enabled conductance
// receives weights of that type only.
template <int ND>
__device__ __forceinline__ void ordered_sum(const WideSmem &S, uint32_t o0, uint32_t c, float *x, int en) {
    if (en == 1) { x[ND] = ordered_sum1(S, o0, c, x[ND]); return; }
    if (en == 2) { x[ND + 1] = ordered_sum1(S, o0, c, x[ND + 1]); return; }
    if (en == 4) { x[ND + 2] = ordered_sum1(S, o0, c, x[ND + 2]); return; }
    float g0 = x[ND], g1 = x[ND + 1], g2 = x[ND + 2];
    uint32_t q = 0;
    for (; q + 8 <= c; q += 8) {
        float w[8];
        int t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) { w[u] = S.sw[o0 + q + u]; t[u] = S.sty[o0 + q + u]; }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (t[u] == 0) g0 += w[u];
            else if (t[u] == 1) g1 += w[u];
            else g2 += w[u];
        }
    }
    for (; q < c; ++q) {
        const int t = S.sty[o0 + q];
        const float w = S.sw[o0 + q];
        if (t == 0) g0 += w;
        else if (t == 1) g1 += w;
        else g2 += w;
    }
    x[ND] = g0;
    x[ND + 1] = g1;
    x[ND + 2] = g2;
}

// Lane 0 of warp 0, after step ks's conductances are in x: integrate, test the
// spike, note it for deferred post-synaptic STDP (global ring and its staged
// copy), trace and recording.  Returns the spike flag.
template <int KIND, int INTEG, int MON = 2, int EN = -1>
__device__ __forceinline__ int wide_advance(const PopDev &P, const NetDev &N, int64_t ks, int64_t i, WideSmem &S,
                                            float *x, NeuronAux &ax, bool ring) {
    const int64_t gi = P.first + i;
    const int sp = advance_neuron<KIND, INTEG, EN>(P, N, i, x, ax) ? 1 : 0;
    if (sp && ring) {
        note_post_spike(P, N, i, ks);
        const uint32_t n1 = P.post_n[i], q = (n1 - 1) % kPostRing;
        S.ring_n = n1;
        S.ring[q] = P.post_t[i * kPostRing + q];
        if (P.post_f) S.ring_f[q] = P.post_f[i * kPostRing + q];
    }
    record_trace(P, N, ks, gi, x, Model<KIND>::NV);
    if (mon_on<MON>(P)) monitor_state(P, N, ks, i, x, Model<KIND>::NV, sp != 0);
    if (sp) {
        if (N.rec_buf) {
            const unsigned long long ro = atomicAdd(N.rec_count, 1ull);
            if (ro < (unsigned long long)N.rec_cap)
                N.rec_buf[ro] = ((unsigned long long)ks << 32) | (unsigned long long)gi;
            else atomicOr(N.flags, FLAG_RECORD_OVERFLOW);
        }
    }
    return sp;
}

template <int KIND, int INTEG, int MON = 2, int EN = -1>
__device__ __forceinline__ void wide_window(const PopDev &P, const NetDev &N, int64_t k, int64_t i, WideSmem &S,
                                            StageSmem &G, float *x, NeuronAux &ax, int nsteps,
                                            double push_inv_dt) {
    constexpr int ND = Model<KIND>::ND;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    const int64_t gi = P.first + i;
    const uint32_t capg = N.cap[gi];
    const int64_t rbase = N.cap_base[gi];
    const bool ring = P.post_t != nullptr;
    const int prule = P.post_f ? P.post_rule : -1;
    if (tid < nsteps) {
        uint32_t c = N.cnt[(int64_t)((k + tid) & (N.R - 1)) * N.n_neurons + gi];
        if (c > capg) { atomicOr(N.flags, FLAG_BUCKET_OVERFLOW); c = capg; }
        S.wcnt[tid] = c;
    }
    if (ring && !S.ring_ok) {
        for (int q = tid; q < kPostRing; q += nt) {
            S.ring[q] = P.post_t[i * kPostRing + q];
            if (P.post_f) S.ring_f[q] = P.post_f[i * kPostRing + q];
        }
        if (tid == nt - 1) S.ring_n = P.post_n[i];
    }
    __syncthreads();
    if (tid == 0) {
        S.woff[0] = 0;
        for (int s = 0; s < nsteps; ++s) S.woff[s + 1] = S.woff[s] + S.wcnt[s];
        if (ring) S.ring_ok = 1;
    }
    if (tid < nsteps) {
        S.kmin[tid] = ~0ull;
        S.kmax[tid] = 0ull;
    }
    __syncthreads();
    int s0 = 0;
    while (s0 < nsteps) {
        int s1 = s0;
        while (s1 < nsteps && S.woff[s1 + 1] - S.woff[s0] <= (uint32_t)kStage) ++s1;
        if (s1 == s0) {  // this step alone overflows the stage
            int pf_n = 0;
            wide_step<KIND, INTEG, MON, EN>(P, N, k + s0, i, S, x, ax, false, push_inv_dt, pf_n, false);
            __syncthreads();
            ++s0;
            continue;
        }
        const uint32_t a0 = S.woff[s0], T = S.woff[s1] - a0;
        for (uint32_t a = tid; a < T; a += nt) {
            const int s = stage_step_of(S, s0, a0 + a);
            const int slot = (int)((k + s) & (N.R - 1));
            const Arrival v = N.rec[(int64_t)slot * N.cap_total + rbase + (a0 + a - S.woff[s])];
            G.arr[a] = v;
            const unsigned long long key = time_key(v.a);
            G.key[a] = key;
            atomicMin(&S.kmin[s], key);
            atomicMax(&S.kmax[s], key);
            // the synapse record, copied while the chunk is hashed and ranked
            const SynRec *src = N.syn + v.tpos;
            cp_async16(&G.rec[a], src);
            cp_async16(reinterpret_cast<unsigned char *>(&G.rec[a]) + 16, reinterpret_cast<const unsigned char *>(src) + 16);
        }
        cp_async_commit();
        for (int h = tid; h < kStageHash; h += nt) G.hkey[h] = kHashEmpty;
        if (tid == 0) S.dup = 0;
        __syncthreads();
        if (tid >= s0 && tid < s1) N.cnt[(int64_t)((k + tid) & (N.R - 1)) * N.n_neurons + gi] = 0;
        if (tid == 0 && T) atomicAdd(P.events, (unsigned long long)T);
        // synapses of the chunk: the arrival that claims a synapse's slot owns it
        for (uint32_t a = tid; a < T; a += nt) {
            const uint32_t tp = G.arr[a].tpos;
            uint32_t h = (tp * 2654435761u) >> (32 - kStageHashBits);
            for (;;) {
                const uint32_t prev = atomicCAS(&G.hkey[h], kHashEmpty, tp);
                if (prev == kHashEmpty) { G.hval[h] = (uint16_t)a; break; }
                if (prev == tp) { S.dup = 1; break; }
                h = (h + 1) & (kStageHash - 1);
            }
            G.own[a] = (uint16_t)h;
            // a step whose arrival times span less than 2^32 key units ranks on
            // one 64-bit key: (time key - the step's smallest) << 32 | synapse order
            const int s = stage_step_of(S, s0, a0 + a);
            const unsigned long long k0 = S.kmin[s];
            if (S.kmax[s] - k0 <= 0xffffffffull) G.key[a] = ((G.key[a] - k0) << 32) | G.arr[a].spos;
        }
        __syncthreads();
        const bool dup = S.dup != 0;
        if (dup) cp_async_wait_all();  // the serial path below rewrites staged records
        for (uint32_t a = tid; a < T; a += nt) {
            const uint32_t o = G.hval[G.own[a]];
            G.own[a] = (uint16_t)o;
            if (dup && o == a) {  // serial path: one staged record per synapse, caught up to the chunk
                SynRec r = N.syn[G.arr[a].tpos];
                if (r.rule >= 0 && ring) apply_pending(N, RingSmem{S.ring, S.ring_f}, S.ring_n, prule, r);
                G.rec[a] = r;
            }
            // delivery position: arrivals of the same step before it in (time,
            // synapse order) order -- a step's synapses are distinct here -- on the
            // integer keys of the times
            const int s = stage_step_of(S, s0, a0 + a);
            const uint32_t b0 = S.woff[s] - a0, b1 = S.woff[s + 1] - a0;
            const unsigned long long ka = G.key[a];
            uint32_t r = 0;
            if (S.kmax[s] - S.kmin[s] <= 0xffffffffull) {
#pragma unroll 8
                for (uint32_t b = b0; b < b1; ++b) r += G.key[b] < ka ? 1u : 0u;
            } else {
                const uint32_t pa = G.arr[a].spos;
#pragma unroll 4
                for (uint32_t b = b0; b < b1; ++b) {
                    const unsigned long long kb = G.key[b];
                    r += (kb < ka || (kb == ka && G.arr[b].spos < pa)) ? 1u : 0u;
                }
            }
            G.rank[a] = (uint16_t)r;
        }
        cp_async_wait_all();
        __syncthreads();
        if (!dup) {
            int s = s0;
            while (s < s1) {
                for (uint32_t a = S.woff[s] - a0 + tid; a < T; a += nt) {
                    // the staged record, caught up to the spikes of the earlier rounds:
                    // this round adds the spike that ended the last one (the same
                    // updates in the same order as one catch-up from the original);
                    // the pre-synaptic update is applied at the write-back
                    SynRec r = G.rec[a];
                    if (r.rule >= 0 && ring) apply_pending(N, RingSmem{S.ring, S.ring_f}, S.ring_n, prule, r);
                    const uint32_t pos = S.woff[stage_step_of(S, s0, a0 + a)] - a0 + G.rank[a];
                    S.sw[pos] = r.w;
                    S.sty[pos] = r.stype;
                    if (mon_on<MON>(P)) monitor_delivery(P, N, k + stage_step_of(S, s0, a0 + a), i, G.arr[a], r.stype, r.w);
                    G.rec[a] = r;
                }
                __syncthreads();
                if (tid < 32) {
                    int next = s1;
                    for (int j = s; j < s1; ++j) {
                        int sp = 0;
                        if (lane == 0) {
                            ordered_sum<ND>(S, S.woff[j] - a0, S.wcnt[j], x, en_mask<EN>(P));
                            sp = wide_advance<KIND, INTEG, MON, EN>(P, N, k + j, i, S, x, ax, ring);
                        }
                        sp = __shfl_sync(0xffffffffu, sp, 0);
                        if (sp && push_inv_dt > 0.0) push_from(P, N, k + j, gi, lane, 32, push_inv_dt);
                        if (sp && ring) { next = j + 1; break; }
                    }
                    if (lane == 0) S.next_s = next;
                }
                __syncthreads();
                s = S.next_s;
            }
        } else if (tid < 32) {
            for (int s = s0; s < s1; ++s) {
                const int64_t ks = k + s;
                const uint32_t o0 = S.woff[s] - a0, c = S.wcnt[s];
                for (uint32_t a = o0 + lane; a < o0 + c; a += 32) {
                    SynRec &sr = G.rec[G.own[a]];
                    SynRec r = sr;
                    if (r.rule >= 0 && ring) apply_pending(N, RingSmem{S.ring, S.ring_f}, S.ring_n, prule, r);
                    S.sw[o0 + G.rank[a]] = r.w;
                    S.sty[o0 + G.rank[a]] = r.stype;
                    if (mon_on<MON>(P)) monitor_delivery(P, N, ks, i, G.arr[a], r.stype, r.w);
                    if (r.rule >= 0) {
                        stdp_pre_rec(N, r, G.arr[a].a);
                        sr = r;
                    }
                }
                __syncwarp();
                int sp = 0;
                if (lane == 0) {
                    ordered_sum<ND>(S, o0, c, x, en_mask<EN>(P));
                    sp = wide_advance<KIND, INTEG, MON, EN>(P, N, ks, i, S, x, ax, ring);
                }
                sp = __shfl_sync(0xffffffffu, sp, 0);
                if (sp && push_inv_dt > 0.0) push_from(P, N, ks, gi, lane, 32, push_inv_dt);
                __syncwarp();
            }
        }
        __syncthreads();
        for (uint32_t a = tid; a < T; a += nt) {
            if (G.own[a] != a || G.rec[a].rule < 0) continue;
            SynRec r = G.rec[a];
            if (!dup) stdp_pre_rec(N, r, G.arr[a].a);  // the serial path applied it already
            SynRec *d = N.syn + G.arr[a].tpos;
            d->w = r.w;
            d->pre = r.pre;
            d->post = r.post;
            d->last = r.last;
        }
        __syncthreads();
        s0 = s1;
    }
}

// Steps k .. k+nsteps-1 of the block's neurons.
// Populations whose synapses cannot deliver twice in one step take the staged
// window; the others run step by step.  At most 72 registers a thread: blocks of
// this kernel share an SM with the thread-per-neuron blocks of 256 (48 registers).
template <int KIND, int INTEG, int MON, int EN>
__global__ void __maxnreg__(72) k_update_wide(PopDev P, NetDev N, int rel, int nsteps,
                                                                 double push_inv_dt) {
    __shared__ WideSmem S;
    extern __shared__ __align__(32) unsigned char stage_raw[];
    StageSmem &G = *reinterpret_cast<StageSmem *>(stage_raw);
    const int64_t k = cur_step(N, rel);
    for (int64_t i = blockIdx.x; i < P.n; i += gridDim.x) {
        float x[kMaxVars];
        NeuronAux ax{-1, 0};
        if (threadIdx.x == 0) {
            load_state<KIND>(P, i, x);
            ax = load_aux<KIND, INTEG>(P, i);
            S.ring_ok = 0;
        }
        __syncthreads();  // S.ring_ok reset before any thread reads it
        if (!P.may_repeat && nsteps <= kMaxWindow) {
            wide_window<KIND, INTEG, MON, EN>(P, N, k, i, S, G, x, ax, nsteps, push_inv_dt);
        } else {
            int pf_n = 0;
            for (int s = 0; s < nsteps; ++s)
                wide_step<KIND, INTEG, MON, EN>(P, N, k + s, i, S, x, ax, false, push_inv_dt, pf_n, s + 1 < nsteps);
        }
        if (threadIdx.x == 0) {
            store_state<KIND>(P, i, x);
            store_aux<KIND, INTEG>(P, i, ax);
        }
        __syncthreads();  // the next neuron's staging reuses S
    }
}

// ------------------------------------------------------------ spike fan-out --
// One input-neuron spike q emitted in [t_{k-1}, t_k).  A source with several
// distinct delays delivers group j+1 at (a_j - d_j) + d_{j+1}, as the reference's
// PropagatedSpike chain does.
__device__ __forceinline__ void input_spike(const NetDev &N, int64_t k, int64_t q, double inv_dt) {
    const int64_t src = N.in_cell[q];
    const double tin = N.in_time[q];
    const int64_t o0 = N.out_ptr[src], o1 = N.out_ptr[src + 1];
    const int64_t g0 = N.grp_ptr[src], g1 = N.grp_ptr[src + 1];
    for (int64_t o = o0 + threadIdx.x; o < o1; o += blockDim.x) {
        const uint16_t u = N.out_units[o];
        double a = tin + (double)N.grp_units[g0] * 0.0001;
        for (int64_t g = g0 + 1; g < g1 && N.grp_units[g - 1] != u; ++g)
            a = a - (double)N.grp_units[g - 1] * 0.0001 + (double)N.grp_units[g] * 0.0001;
        bucket_put(N, arrival_step(N, a, k, inv_dt), a, o);
    }
}

// Post-synaptic STDP (STDPWeightChange::ApplyPostSynapticSpike) for work item
// (spike s, chunk ch of blockDim plastic inputs): one synapse per thread.
__device__ __forceinline__ void post_item(const PopDev &P, const NetDev &N, int64_t k, int64_t s, int64_t ch) {
    const double tk = N.tstep[k];
    const int64_t t = P.first + P.spk[s];
    const int64_t tp = N.in_ptr[t] + ch * blockDim.x + threadIdx.x;
    if (tp >= N.plastic_end[t]) return;
    const SynRec r = N.syn[tp];
    const float *rp = N.rule_par + r.rule * 6;
    float pre = r.pre, post = r.post, w = r.w;
    const float el = (float)(tk - r.last);
    pre *= expt_net(N, -el * rp[4]);
    post *= expt_net(N, -el * rp[5]);
    post += 1.0f;
    w += rp[0] * pre;
    if (w > r.maxw) w = r.maxw; else if (w < 0.0f) w = 0.0f;
    SynRec *o = N.syn + tp;
    o->w = w;
    o->pre = pre;
    o->post = post;
    o->last = tk;
}

}  // namespace eb
