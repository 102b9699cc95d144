// Batched parameter sweep: many independent conductance-LIF networks of uneven
// size advanced together by one persistent kernel -- the sweep use of EDLUT
// (many simulations of small networks with varied parameters).
//
// A network is one LIF population (sources [0, n_exc) excitatory, [n_exc, n)
// inhibitory) plus n_in input neurons (sources n .. n+n_in-1, excitatory) whose
// spikes are given as times.  Connectivity is Bernoulli(p) from every source to
// every neuron with one delay and static weights; Euler, RK2 or RK4.
//
// One CTA owns one network for a chunk of steps (a persistent grid takes networks
// from an atomic queue, largest first, so uneven sizes balance).  When there are
// fewer networks than half the SMs, a cluster of 2, 4 or 8 CTAs owns one, each CTA a
// tile of its neurons.  Per step k:
//   1. deliveries: the source steps j whose spikes arrive at step k (one or two;
//      a host table, because the arrival step of t_j + d flips with the rounding
//      of the double step times) and the input spikes arriving in the step, listed
//      in the reference's delivery order -- arrival time, then synapse order (source,
//      target) -- by one warp from the spike bitmasks of the delay ring in shared
//      memory.  A spike is needed `lag` steps later, so the steps of a window of up to
//      8 are listed at its start, a warp each, and the listed rows prefetched into L2.
//      Every thread loads a batch of the listed sources' synapses (target, weight) at
//      once, then the batch is applied one source at a time, or in rounds of bids when
//      there are many (deliver_batch), so that each target receives its additions in
//      list order without float atomics (src/spike/PropagatedSpikeGroup.cpp:112-149);
//   2. update: each thread advances neurons tid, tid + blockDim, ... of its tile (the
//      state -- V, refractory counter, gE, gI -- lives in shared memory for the chunk)
//      with the model/integrator arithmetic of the plain path, with the refractory
//      test precomputed per network as step counts
//      (src/neuron_model/LIFTimeDrivenModel.cpp:160-242);
//      (steps without deliveries follow the one before in registers, without a barrier);
//   3. spikes: one warp ballot per 32 neurons is the bitmask word of the step's ring
//      slot, stored into the ring of every CTA of the network.  The CTAs of a cluster
//      meet once per window; the first one then appends the window's spikes to the
//      network's record.
// So each network's spikes equal a solo run of the same network on the plain
// path.  Connectivity and weights come from a counter-based hash of (seed,
// network, source, target), generated on the device at build time.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "eb_sweep.h"
#include "eb_tables.h"

using namespace eb;
using namespace ebsw;

namespace {

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    uint64_t z = x + 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t net_key(uint64_t seed, int net) {
    return splitmix64(seed ^ ((uint64_t)(net + 1) * 0xD1B54A32D192ED03ull));
}

// Bernoulli(p) draw of synapse (src, tgt) of a network; returns the hash for the weight.
__device__ __forceinline__ bool syn_draw(uint64_t key, int src, int tgt, double p, uint64_t &h) {
    h = splitmix64(key ^ (((uint64_t)(uint32_t)src << 32) | (uint32_t)tgt));
    return (double)(h >> 11) * (1.0 / 9007199254740992.0) < p;
}

// ------------------------------------------------------- connectivity build --
// Synapse counts per source: blockIdx.y = network.
__global__ void k_sweep_count(const SweepNet *nets, uint64_t seed, uint32_t *counts) {
    const SweepNet &S = nets[blockIdx.y];
    if (S.explicit_syn) return;
    const uint64_t key = net_key(seed, blockIdx.y);
    const int nsrc = S.n + S.n_in;
    __shared__ int sc[32];
    for (int s = blockIdx.x; s < nsrc; s += gridDim.x) {
        int c = 0;
        for (int t = threadIdx.x; t < S.n; t += blockDim.x) {
            uint64_t h;
            c += syn_draw(key, s, t, (double)S.p, h) ? 1 : 0;
        }
        for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
        if ((threadIdx.x & 31) == 0) sc[threadIdx.x >> 5] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += sc[w];
            counts[S.src_off + s] = (uint32_t)tot;
        }
        __syncthreads();
    }
}

// One warp per source writes its targets in increasing order with their weights.
__global__ void k_sweep_fill(const SweepNet *nets, const uint32_t *optr, uint64_t seed, uint16_t *tgt, float *w) {
    const SweepNet &S = nets[blockIdx.y];
    if (S.explicit_syn) return;
    const uint64_t key = net_key(seed, blockIdx.y);
    const int nsrc = S.n + S.n_in;
    const int lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    for (int s = blockIdx.x * warps + (threadIdx.x >> 5); s < nsrc; s += gridDim.x * warps) {
        int64_t pos = S.syn_off + optr[S.src_off + s];
        const float wmax = s < S.n_exc ? S.w_max[0] : (s < S.n ? S.w_max[1] : S.w_max[2]);
        for (int t0 = 0; t0 < S.n; t0 += 32) {
            const int t = t0 + lane;
            bool hit = false;
            uint64_t h = 0;
            if (t < S.n) hit = syn_draw(key, s, t, (double)S.p, h);
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                const int64_t o = pos + __popc(m & ((1u << lane) - 1u));
                const float u = (float)(splitmix64(h) >> 40) * (1.0f / 16777216.0f);
                tgt[o] = (uint16_t)t;
                w[o] = u * wmax;
            }
            pos += __popc(m);
        }
    }
}

// --------------------------------------------------------------- neuron update --
// One integration step, operation for operation the plain path's integrate<LIF, INTEG>.
template <int INTEG, int EN>
__device__ __forceinline__ void sw_integrate(const SweepLif &L, float dt, float &V, float &gE, float &gI, int cls, float f) {
    if (INTEG == INTEG_EULER) {
        const float k1 = sw_deriv<EN>(L, V, gE, gI, cls, f);
        V += dt * k1;
        sw_decay<EN>(L, gE, gI);
    } else if (INTEG == INTEG_RK2) {
        const float k1 = sw_deriv<EN>(L, V, gE, gI, cls, f);
        V += k1 * dt;
        sw_decay<EN>(L, gE, gI);
        const float k2 = sw_deriv<EN>(L, V, gE, gI, cls, f);
        V += (-k1 + k2) * dt * 0.5f;
    } else {
        const float h05 = dt * 0.5f;
        const float h016 = dt * 0.166666666667f;
        const float k1 = sw_deriv<EN>(L, V, gE, gI, cls, f);
        float a = V + k1 * h05;
        float aE = gE, aI = gI;
        sw_decay<EN>(L, aE, aI);
        const float k2 = sw_deriv<EN>(L, a, aE, aI, cls, f);
        a = V + k2 * h05;
        const float k3 = sw_deriv<EN>(L, a, aE, aI, cls, f);
        a = V + k3 * dt;
        sw_decay<EN>(L, aE, aI);
        const float k4 = sw_deriv<EN>(L, a, aE, aI, cls, f);
        V += (k1 + 2.0f * (k2 + k3) + k4) * h016;
        gE = aE;
        gI = aI;
    }
}

// Largest a in [0, S) with off[a] <= e (off[0] = 0 <= e < off[S]).
__device__ __forceinline__ int list_rank(const int32_t *off, int S, int e) {
    int lo = 0, hi = S;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= e) lo = mid; else hi = mid;
    }
    return lo;
}

// First synapse of every source in each of `ctas` tiles of its network's neurons (one
// thread per source and tile boundary, bisection in the source's ascending targets).
__global__ void k_sweep_tiles(SweepDev G, int ctas, uint32_t *tptr) {
    const SweepNet &S = G.nets[blockIdx.y];
    const int tile = (S.wn + ctas - 1) / ctas * 32;
    const int64_t items = (int64_t)(S.n + S.n_in) * (ctas + 1);
    const uint16_t *tg = G.tgt + S.syn_off;
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < items; x += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = x / (ctas + 1);
        const int first = (int)(x - s * (ctas + 1)) * tile;
        uint32_t lo = G.optr[S.src_off + s], hi = G.optr[S.src_off + s + 1];
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if ((int)tg[mid] < first) lo = mid + 1; else hi = mid;
        }
        tptr[S.src_off * (ctas + 1) + x] = lo;
    }
}

// One step's sources in delivery order, with the synapses they have in the CTA's tile.
struct SweepList {
    int32_t *src, *off;     // [cap], [cap + 1]: source, running total of synapses
    uint32_t *base;         // [cap]: its first synapse
};

struct SweepSmem {
    float4 *x;              // [tile] V, gE, gI, refractory counter (integer bits)
    uint32_t *ring;         // [R][wc] spike bitmasks of the whole network
    uint32_t *bid;          // [kBidSlots] lowest source rank bidding for a target (kNoBid between batches)
    int32_t *lists;         // the lists of a window's steps
    int cap;
    __device__ SweepList list(int s) const {
        int32_t *p = lists + s * (3 * cap + 1);
        return SweepList{p, p + cap, reinterpret_cast<uint32_t *>(p + 2 * cap + 1)};
    }
};

size_t sweep_smem_bytes(int tile, int R, int wc, int window, int cap) {
    return 16 * (size_t)tile + sizeof(uint32_t) * ((size_t)R * wc + kBidSlots) + window * sizeof(int32_t) * (3 * (size_t)cap + 1);
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Barrier of every thread of the cluster, ordering shared-memory stores across it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Store v at the place of p in the shared memory of the cluster's CTA `rank`.
__device__ __forceinline__ void cluster_store(uint32_t *p, uint32_t rank, uint32_t v) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// First input spike at or after `cur` whose key reaches `key` (one warp, 32 at a time).
__device__ __forceinline__ int64_t seek_input(const SweepDev &G, const SweepNet &S, int64_t cur, int32_t key, int lane) {
    for (;;) {
        const bool below = cur + lane < S.n_in_spikes && G.in_key[S.in_off + cur + lane] < key;
        const int c = __popc(__ballot_sync(0xffffffffu, below));
        cur += c;
        if (c < 32) return cur;
    }
}

// One warp lists step k's sources, positions [p0, p0 + cap) of the delivery order, into
// B: per phase the inputs of its key (from input `cur` on), then the spikes of the
// next arriving source step in neuron order; then their synapse ranges and running
// totals, and their rows on the way into L2.  Returns the sources of the whole step.
__device__ __forceinline__ int list_step(const SweepDev &G, const SweepSmem &M, const SweepNet &S, const SweepList &B,
                                         int64_t cur, int64_t k, int p0, int wc, int tile, int lane) {
    constexpr unsigned full = 0xffffffffu;
    const int lo = G.grp_lo[k], groups = G.grp_n[k], cap = M.cap;
    int pos = 0;
    for (int g = 0; g <= groups; ++g) {
        for (;;) {  // inputs of phase g
            const int64_t q = cur + lane;
            const bool mine = q < S.n_in_spikes && G.in_key[S.in_off + q] == (int32_t)(k * 4) + g;
            const int c = __popc(__ballot_sync(full, mine));
            const int p = pos + lane - p0;
            if (mine && p >= 0 && p < cap) B.src[p] = S.n + G.in_src[S.in_off + q];
            pos += c;
            cur += c;
            if (c < 32) break;
        }
        if (g == groups) break;
        const uint32_t *row = M.ring + (int)((uint32_t)(lo + g) % (uint32_t)G.R) * wc;
        for (int a = 0; a < S.wn; a += 32) {
            if (a % 256 == 0) {  // 8,192 neurons at once: most steps have few spikes or none
                uint32_t any = 0;
#pragma unroll
                for (int u = 0; u < 256; u += 32) any |= a + u + lane < S.wn ? row[a + u + lane] : 0u;
                if (!__any_sync(full, any != 0)) { a += 256 - 32; continue; }
            }
            uint32_t w = a + lane < S.wn ? row[a + lane] : 0u;
            if (!__any_sync(full, w != 0)) continue;
            const int c = __popc(w);
            const int incl = warp_incl_scan(c, lane);
            int p = pos + incl - c - p0;
            while (w) {
                const int b = __ffs(w) - 1;
                w &= w - 1u;
                if (p >= 0 && p < cap) B.src[p] = (a + lane) * 32 + b;
                ++p;
            }
            pos += __shfl_sync(full, incl, 31);
        }
    }
    __syncwarp();
    const int cnt = min(pos - p0, cap);
    int carry = 0;
    for (int b = 0; b < cnt; b += 32) {
        const int x = b + lane;
        uint32_t first = 0;
        int fan = 0;
        if (x < cnt) {
            const uint32_t *t = G.tptr + (S.src_off + B.src[x]) * G.tstride + tile;
            first = __ldg(t);
            fan = (int)(__ldg(t + 1) - first);
        }
        const int incl = warp_incl_scan(fan, lane);
        if (x < cnt) {
            B.off[x] = carry + incl - fan;
            B.base[x] = first;
            if (fan > 0) {  // whole 16-byte units around the row
                const uint64_t t = (uint64_t)(G.tgt + S.syn_off + first), w = (uint64_t)(G.w + S.syn_off + first);
                const uint64_t t0 = t & ~15ull, w0 = w & ~15ull;
                const uint32_t nt = (uint32_t)((t + 2ull * fan - t0 + 15) & ~15ull);
                const uint32_t nw = (uint32_t)((w + 4ull * fan - w0 + 15) & ~15ull);
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(t0), "r"(nt) : "memory");
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w0), "r"(nw) : "memory");
            }
        }
        carry += __shfl_sync(full, incl, 31);
    }
    if (lane == 0 && cnt > 0) B.off[cnt] = carry;
    return pos;
}

// Deliver entries e0 .. of the listed sources' flattened synapses, NB a thread, by the
// whole block.  A target receives its additions in list order without atomics on
// floats: a few sources go one at a time with a barrier in between (one source's
// targets are distinct).  Many sources -- the bursts of a large network, whose rows in
// a tile are short -- go in rounds instead: every pending entry bids its source's rank
// for its target's slot, the lowest rank of a slot is added, the others bid again.  A
// batch takes as many rounds as its most frequent target has entries, not one per
// source (slots shared by several targets only make an entry wait).  A fitting step of
// 8 networks of up to 10,000 neurons: 9.2 -> 7.4 ms; 600 networks: 6.5 -> 6.3 ms.
template <int NB>
__device__ __forceinline__ void deliver_batch(const SweepSmem &M, const SweepList &B, int sources, int e0, int total,
                                              const uint16_t *tg, const float *ww, int n_exc, int n, int first) {
    const int tid = threadIdx.x, nt = blockDim.x;
    int t[NB], rk[NB];
    float w[NB];
    bool inh[NB];
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const int e = e0 + q * nt + tid;
        rk[q] = -1;
        t[q] = 0;
        w[q] = 0.0f;
        inh[q] = false;
        if (e < total) {
            const int a = list_rank(B.off, sources, e);
            const uint32_t o = B.base[a] + (uint32_t)(e - B.off[a]);
            t[q] = (int)__ldg(tg + o) - first;
            w[q] = __ldg(ww + o);
            const int x = B.src[a];
            inh[q] = x >= n_exc && x < n;
            rk[q] = a;
        }
    }
    auto add = [&](int q) {
        float4 &x = M.x[t[q]];
        if (inh[q]) x.z += w[q];
        else x.y += w[q];
    };
    const int r_lo = list_rank(B.off, sources, e0);
    const int r_hi = list_rank(B.off, sources, min(e0 + NB * nt, total) - 1);
    if (r_hi - r_lo < kRoundSources) {
        for (int a = r_lo; a <= r_hi; ++a) {
#pragma unroll
            for (int q = 0; q < NB; ++q)
                if (rk[q] == a) add(q);
            __syncthreads();
        }
        return;
    }
    bool pending = true;
    while (__syncthreads_or(pending)) {
#pragma unroll
        for (int q = 0; q < NB; ++q)
            if (rk[q] >= 0) atomicMin(M.bid + (t[q] & (kBidSlots - 1)), (uint32_t)rk[q]);
        __syncthreads();
        pending = false;
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            if (rk[q] < 0) continue;
            uint32_t *slot = M.bid + (t[q] & (kBidSlots - 1));
            if (*(volatile uint32_t *)slot == (uint32_t)rk[q]) {
                add(q);
                *(volatile uint32_t *)slot = kNoBid;
                rk[q] = -1;
            } else {
                pending = true;
            }
        }
    }
}

// Neurons whose V this thread records after every step: it owns up to two observed
// ones (i: index in the tile, m: observed slot).
struct SweepObs {
    int i0, m0, i1, m1;
};

// The CTA's update of its tile at steps k .. k + run - 1, none of which but the first
// has deliveries: integrate, spike test, bitmask words into the steps' ring slots of
// every CTA of the network.  The sweep is bound by the instructions of this loop: a
// neuron's state is one 16-byte word of shared memory, loaded once for the steps, and
// the refractory class selects (no branches).
template <int INTEG, bool TRAJ, int EN, bool CL>
__device__ __forceinline__ void sweep_update(const SweepDev &G, const SweepSmem &M, const SweepLif &L, const SweepLif &Ls,
                                             const SweepObs &O, int nl, int first, int run, int slot0, int wc, int64_t x0,
                                             float *trace) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, ctas = G.ctas;
    const float dt = G.dt_ms;
    const int wrap = G.R * wc;
    for (int i = tid; i - lane < nl; i += nt) {
        const bool valid = i < nl;
        float4 x = M.x[valid ? i : 0];
        int rr = __float_as_int(x.w);
        int word = slot0 * wc + ((first + i) >> 5);
        for (int t = 0; t < run; ++t) {
            const bool late = (unsigned)rr < (unsigned)L.r_free;  // refractory, and not the -1 of no spike yet
            const bool frozen = late && rr < L.r_frac0, part = late && !frozen;
            const int fi = part ? rr - L.r_frac0 : 0;
            float f = 1.0f;
            if (part) f = Ls.frac[fi];
            if (TRAJ && valid) {
                const int64_t o = x0 + t * G.n_total + i;
                G.tV[o] = x.x;
                G.tE[o] = x.y;
                G.tI[o] = x.z;
            }
            sw_integrate<INTEG, EN>(L, dt, x.x, x.y, x.z, frozen ? 1 : 2, f);
            if (rr >= 0) rr++;
            const bool sp = x.x > L.v_thr;
            x.x = sp ? L.e_leak : x.x;
            rr = sp ? 0 : rr;
            if (TRAJ && valid)
                G.tcode[x0 + t * G.n_total + i] = (uint8_t)((frozen ? 1 : part ? 2 : 0) | (fi << 2) | (sp ? kCodeSpike : 0));
            if (x.x != x.x) { x.x = L.e_leak; x.y = 0.0f; x.z = 0.0f; }
            if (i == O.i0) trace[t * G.n_obs + O.m0] = x.x;
            if (i == O.i1) trace[t * G.n_obs + O.m1] = x.x;
            const unsigned m = __ballot_sync(0xffffffffu, sp && valid);
            if (CL) { if (lane < ctas) cluster_store(M.ring + word, lane, m); }
            else if (lane == 0) M.ring[word] = m;
            word += wc;
            if (word >= wrap) word -= wrap;
        }
        x.w = __int_as_float(rr);
        if (valid) M.x[i] = x;
    }
}

// Append the spikes of steps k_first .. k_first + len - 1 to the network's record, in
// (step, neuron) order, from the ring's bitmasks (one CTA, whole block).
__device__ __forceinline__ void drain_window(const SweepDev &G, const SweepSmem &M, const SweepNet &S, int net, int64_t k_first,
                                             int len, int wc, uint32_t *s_cnt, uint32_t &rec_n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int s = warp; s < len; s += nwarps) {
        const uint32_t *row = M.ring + (int)((uint32_t)(k_first + s) % (uint32_t)G.R) * wc;
        int c = 0;
        for (int a = lane; a < S.wn; a += 32) c += __popc(row[a]);
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) s_cnt[s] = (uint32_t)c;
    }
    __syncthreads();
    uint32_t at = rec_n;
    for (int s = 0; s < len; ++s) {
        const uint32_t c = s_cnt[s];
        if ((s & (nwarps - 1)) == warp && c) {
            const uint32_t *row = M.ring + (int)((uint32_t)(k_first + s) % (uint32_t)G.R) * wc;
            uint32_t pos = at;
            for (int a = 0; a < S.wn; a += 32) {
                uint32_t w = a + lane < S.wn ? row[a + lane] : 0u;
                if (!__any_sync(0xffffffffu, w != 0)) continue;
                const int n = __popc(w);
                const int incl = warp_incl_scan(n, lane);
                uint32_t x = pos + (uint32_t)(incl - n);
                while (w) {
                    const int b = __ffs(w) - 1;
                    w &= w - 1u;
                    if ((int64_t)x < S.rec_cap) G.rec[S.rec_off + x] = (uint16_t)((a + lane) * 32 + b);
                    else atomicOr(G.flags, FLAG_RECORD_OVERFLOW);
                    ++x;
                }
                pos += (uint32_t)__shfl_sync(0xffffffffu, incl, 31);
            }
        }
        at += c;
        if (threadIdx.x == 0) G.rec_end[(int64_t)net * G.steps_max + (k_first + s - 1)] = (int32_t)at;
    }
    rec_n = at;
}

template <int INTEG, bool TRAJ, bool CL>
__device__ void sweep_network(const SweepDev &G, const SweepSmem &M, const SweepNet &S, const SweepLif &Ls, int net, int tile,
                              int64_t k0, int nsteps, int wc, int64_t traj_k0) {
    __shared__ int s_cnt[kSweepWindow];   // sources of each step of the window
    __shared__ uint32_t s_win[kSweepWindow];
    const int n = S.n, n_exc = S.n_exc;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    const int R = G.R, C = G.ctas, wn = S.wn, cap = M.cap;
    const int first = (wn + C - 1) / C * 32 * tile;               // the tile's neurons
    const int nl = max(0, min(n - first, (wn + C - 1) / C * 32));
    const int64_t so = S.state_off + first;
    const uint16_t *tg = G.tgt + S.syn_off;
    const float *ww = G.w + S.syn_off;
    const SweepLif L = Ls;  // in registers; the fractions are indexed in shared memory

    for (int i = tid; i < nl; i += nt)
        M.x[i] = make_float4(G.V[so + i], G.gE[so + i], G.gI[so + i], __int_as_float(G.refr[so + i]));
    for (int x = tid; x < R * wc; x += nt) {
        const int slot = x / wc, q = x - slot * wc;
        M.ring[x] = q < wn ? G.ring[S.ring_off + (int64_t)slot * wn + q] : 0u;
    }
    // observed neurons: written by their owners while nobody owns more than two, else
    // read by the block after every step
    SweepObs O{-1, 0, -1, 0};
    bool many = G.n_obs > kOwnObs;
    const int32_t *obs = G.obs + (int64_t)net * G.n_obs;
    if (!many)
        for (int m = 0; m < G.n_obs; ++m) {
            const int i = obs[m] - first;
            if (i < 0 || i >= nl || i % nt != tid) continue;
            many = many || O.i1 >= 0;
            if (O.i0 < 0) { O.i0 = i; O.m0 = m; }
            else { O.i1 = i; O.m1 = m; }
        }
    many = __syncthreads_or(many);
    if (many) O.i0 = O.i1 = -1;
    unsigned long long events = 0;
    uint32_t rec_n = tile == 0 ? G.rec_cnt[net] : 0u;
    int64_t cur = G.in_cursor[net];  // this warp's place in the input spikes
    if (CL) cluster_sync();  // every ring is loaded before another CTA's spikes reach it

    for (int w0 = 0; w0 < nsteps; w0 += G.window) {
        const int64_t kw = k0 + w0 + 1;  // the window's first step
        const int len = min(G.window, nsteps - w0);
        for (int s = warp; s < len; s += nwarps) {
            cur = seek_input(G, S, cur, (int32_t)((kw + s) * 4), lane);
            const int c = list_step(G, M, S, M.list(s), cur, kw + s, 0, wc, tile, lane);
            if (lane == 0) s_cnt[s] = c;
        }
        __syncthreads();
        for (int s = 0; s < len;) {
            const int64_t k = kw + s;
            const int sources = s_cnt[s];
            // ------------------------------------------------ 1. deliveries
            if (sources > 0) {
                if (s > 0) __syncthreads();  // the last update is done
                const SweepList B = M.list(s);
                for (int p0 = 0;; p0 += cap) {
                    const int Sn = min(sources - p0, cap);
                    const int total = B.off[Sn];
                    for (int e0 = 0; e0 < total;) {
                        if (total - e0 <= nt) {
                            deliver_batch<1>(M, B, Sn, e0, total, tg, ww, n_exc, n, first);
                            e0 += nt;
                        } else {
                            deliver_batch<kBatch>(M, B, Sn, e0, total, tg, ww, n_exc, n, first);
                            e0 += kBatch * nt;
                        }
                    }
                    if (tid == 0) events += (unsigned long long)total;
                    if (p0 + cap >= sources) break;
                    __syncthreads();  // every thread is done with this pass's list
                    if (warp == 0) {
                        const int64_t c0 = seek_input(G, S, G.in_cursor[net], (int32_t)(k * 4), lane);
                        list_step(G, M, S, B, c0, k, p0 + cap, wc, tile, lane);
                    }
                    __syncthreads();
                }
            }
            // ---------------------------------------------- 2. update, 3. spikes
            int run = 1;
            if (!many)
                while (s + run < len && s_cnt[s + run] == 0) ++run;
            const int slot = (int)((uint32_t)k % (uint32_t)R);
            const int64_t x0 = TRAJ ? (k - traj_k0 - 1) * G.n_total + so : 0;
            float *trace = G.trace + ((int64_t)net * G.steps_max + (k - 1)) * G.n_obs;
            if (L.en == 3) sweep_update<INTEG, TRAJ, 3, CL>(G, M, L, Ls, O, nl, first, run, slot, wc, x0, trace);
            else sweep_update<INTEG, TRAJ, -1, CL>(G, M, L, Ls, O, nl, first, run, slot, wc, x0, trace);
            if (many) {
                __syncthreads();
                for (int m = tid; m < G.n_obs; m += nt) {
                    const int i = obs[m] - first;
                    if (i >= 0 && i < nl) trace[m] = M.x[i].x;
                }
                __syncthreads();  // read before the next step writes them
            }
            s += run;
        }
        if (CL) cluster_sync();
        else __syncthreads();
        if (tile == 0) drain_window(G, M, S, net, kw, len, wc, s_win, rec_n);
    }
    // save the network's state
    for (int i = tid; i < nl; i += nt) {
        const float4 x = M.x[i];
        G.V[so + i] = x.x;
        G.refr[so + i] = __float_as_int(x.w);
        G.gE[so + i] = x.y;
        G.gI[so + i] = x.z;
    }
    if (CL) cluster_sync();  // every CTA has read the input cursor
    if (tile == 0) {
        for (int x = tid; x < R * wn; x += nt) {
            const int s = x / wn, q = x - s * wn;
            G.ring[S.ring_off + x] = M.ring[s * wc + q];
        }
        if (warp == 0) {
            cur = seek_input(G, S, cur, (int32_t)((k0 + nsteps + 1) * 4), lane);
            if (lane == 0) G.in_cursor[net] = cur;
        }
    }
    if (tid == 0) {
        if (tile == 0) G.rec_cnt[net] = rec_n;
        if (CL) atomicAdd(&G.events[net], events);
        else G.events[net] += events;
    }
    __syncthreads();
}

template <int INTEG, bool TRAJ, bool CL>
__global__ void __launch_bounds__(1024) k_sweep(SweepDev G, int nsteps, int max_tile, int wc, int64_t traj_k0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SweepSmem M;
    M.x = reinterpret_cast<float4 *>(smem_raw);
    M.ring = reinterpret_cast<uint32_t *>(M.x + max_tile);
    M.bid = M.ring + G.R * wc;
    M.lists = reinterpret_cast<int32_t *>(M.bid + kBidSlots);
    for (int x = threadIdx.x; x < kBidSlots; x += blockDim.x) M.bid[x] = kNoBid;  // (barriers follow before the first bid)
    M.cap = G.list_cap;
    __shared__ int s_net;
    __shared__ SweepLif s_L;
    __shared__ SweepNet s_desc;
    const int64_t k0 = *G.step;
    const int tile = CL ? (int)cluster_rank() : 0;
    for (;;) {
        if (threadIdx.x == 0) s_net = CL ? (int)blockIdx.x / G.ctas : atomicAdd(G.queue, 1);  // CL: a cluster per network
        __syncthreads();
        const int qi = s_net;
        if (qi >= G.n_nets) break;
        const int net = G.order[qi];
        {
            const int *src = reinterpret_cast<const int *>(G.nets + net);
            int *dst = reinterpret_cast<int *>(&s_desc);
            for (int x = threadIdx.x; x < (int)(sizeof(SweepNet) / sizeof(int)); x += blockDim.x) dst[x] = src[x];
        }
        __syncthreads();
        if (threadIdx.x == 0) s_L = s_desc.L;
        __syncthreads();
        sweep_network<INTEG, TRAJ, CL>(G, M, s_desc, s_L, net, tile, k0, nsteps, wc, traj_k0);
        if (CL) break;
    }
}

// The initial state of every network (blockIdx.y): V = E_leak, no conductance, never
// spiked, empty ring and records, step 0.  (Record ends are written before they are read.)
__global__ void __launch_bounds__(256) k_sweep_reset(SweepDev G) {
    const int net = blockIdx.y;
    const SweepNet &S = G.nets[net];
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (int i = i0; i < S.n; i += stride) {
        const int64_t o = S.state_off + i;
        G.V[o] = S.L.e_leak;
        G.gE[o] = 0.0f;
        G.gI[o] = 0.0f;
        G.refr[o] = -1;
    }
    for (int64_t x = i0; x < (int64_t)G.R * S.wn; x += stride) G.ring[S.ring_off + x] = 0u;
    if (i0 == 0) {
        G.in_cursor[net] = 0;
        G.rec_cnt[net] = 0u;
        G.events[net] = 0ull;
        if (net == 0) {
            *G.flags = 0u;
            *G.queue = 0;
            *G.step = 0;
        }
    }
}

// After a chunk: advance the step counter and re-arm the network queue.
__global__ void k_sweep_advance(int64_t *step, int *queue, int nsteps) {
    *step += nsteps;
    *queue = 0;
}

}  // namespace

// ------------------------------------------------------------------- host --
namespace {

using SweepFn = void (*)(SweepDev, int, int, int, int64_t);

template <int INTEG>
SweepFn sweep_fn_t(bool traj, bool clustered) {
    if (clustered) return traj ? k_sweep<INTEG, true, true> : k_sweep<INTEG, false, true>;
    return traj ? k_sweep<INTEG, true, false> : k_sweep<INTEG, false, false>;
}

SweepFn sweep_fn(int integ, bool traj, bool clustered) {
    switch (integ) {
    case INTEG_EULER: return sweep_fn_t<INTEG_EULER>(traj, clustered);
    case INTEG_RK2: return sweep_fn_t<INTEG_RK2>(traj, clustered);
    default: return sweep_fn_t<INTEG_RK4>(traj, clustered);
    }
}

}  // namespace

namespace ebsw {

// (pointers and sizes of the arrays that k_sweep_copy moves)
struct StateCopy {
    uint32_t *live[8], *saved[8];
    int64_t words[8];
};

int enqueue_chunk(eb_sweep *h, int nsteps, cudaStream_t st, bool traj, int64_t traj_k0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(h->grid);
    cfg.blockDim = dim3(h->block);
    cfg.dynamicSmemBytes = h->smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = h->G.ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = h->G.ctas > 1 ? 1 : 0;
    SK(cudaLaunchKernelEx(&cfg, sweep_fn(h->integ, traj, h->G.ctas > 1), h->G, nsteps, h->max_tile, h->wc, traj_k0));
    k_sweep_advance<<<1, 1, 0, st>>>(h->G.step, h->G.queue, nsteps);
    SK(cudaGetLastError());
    return EB_OK;
}

// The arrays that make up the dynamic state, in checkpoint order, and their places in a
// checkpoint slot (256-byte aligned).  All are whole 32-bit words.
constexpr int kStateArrays = 8;

static size_t state_arrays(eb_sweep *h, StateCopy &c, void *slot) {
    const size_t nt = (size_t)h->state_n, B = (size_t)h->n_nets;
    void *p[kStateArrays] = {h->G.V, h->G.gE, h->G.gI, h->G.refr, h->G.ring, h->G.in_cursor, h->G.rec_cnt, h->G.events};
    const size_t words[kStateArrays] = {nt, nt, nt, nt, (size_t)h->ring_words, 2 * B, B, 2 * B};
    size_t off = 0;
    for (int i = 0; i < kStateArrays; ++i) {
        c.live[i] = (uint32_t *)p[i];
        c.saved[i] = (uint32_t *)slot + off;
        c.words[i] = (int64_t)words[i];
        off += (words[i] + 63) / 64 * 64;
    }
    return 4 * off;
}

size_t checkpoint_bytes(eb_sweep *h) {
    StateCopy c;
    return state_arrays(h, c, nullptr);
}

// All arrays of the state in one launch (eight copies cost the host 3 us each, and a
// segment of the adjoint has two such sets); step >= 0 also sets the step counter and
// re-arms the network queue.
__global__ void __launch_bounds__(256) k_sweep_copy(StateCopy c, int restore, int64_t step, int64_t *d_step, int *queue) {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    for (int a = 0; a < kStateArrays; ++a) {
        uint32_t *dst = restore ? c.live[a] : c.saved[a];
        const uint32_t *src = restore ? c.saved[a] : c.live[a];
        for (int64_t i = i0; i < c.words[a]; i += stride) dst[i] = src[i];
    }
    if (i0 == 0 && step >= 0) {
        *d_step = step;
        *queue = 0;
    }
}

static int checkpoint_copy(eb_sweep *h, int slot, int restore, int64_t step, cudaStream_t st) {
    StateCopy c;
    const size_t bytes = state_arrays(h, c, h->ckpt[slot]);
    const int blocks = (int)std::min<size_t>(148 * 4, bytes / 4096 + 1);
    k_sweep_copy<<<blocks, 256, 0, st>>>(c, restore, step, h->G.step, h->G.queue);
    SK(cudaGetLastError());
    return EB_OK;
}

int checkpoint_save(eb_sweep *h, int c, cudaStream_t st) { return checkpoint_copy(h, c, 0, -1, st); }

int checkpoint_restore(eb_sweep *h, int c, int64_t step, cudaStream_t st) {
    h->counts_ok = false;
    return checkpoint_copy(h, c, 1, step, st);
}

int upload_params(eb_sweep *h, cudaStream_t st) {
    if (!h->nets_dirty) return EB_OK;
    SK(cudaMemcpyAsync(h->d_nets, h->nets.data(), sizeof(SweepNet) * h->nets.size(), cudaMemcpyHostToDevice, st));
    h->nets_dirty = false;
    return EB_OK;
}

}  // namespace ebsw

namespace {

// LIF parameters of a network from its 10 .cfg values (decay factors and the
// inverse capacitance computed like the plain path's finalize).
int fill_lif(eb_sweep *h, const float *lif_params, SweepLif &L);

// Precomputed refractory classes: the plain path's lif_deriv decides per call from
// l = refr * dt * 1000 (double); here the same comparisons run once per refr value.
int refractory_classes(float tau_ref, float dt_s, SweepLif &L) {
    const float dt_ms = dt_s * 1000.0f;
    L.r_frac0 = -1;
    for (int r = 0;; ++r) {
        const double l = ((double)r * (double)dt_s) * 1000.0;
        if (l > (double)tau_ref) {
            L.r_free = r;
            break;
        }
        if (l + (double)dt_ms > (double)tau_ref) {
            if (L.r_frac0 < 0) L.r_frac0 = r;
            if (r - L.r_frac0 >= kMaxFrac) return EB_ERR_UNSUPPORTED;
            L.frac[r - L.r_frac0] = (float)((l + (double)dt_ms - (double)tau_ref) / (double)dt_ms);
        }
        if (r > (1 << 24)) return EB_ERR_UNSUPPORTED;
    }
    if (L.r_frac0 < 0) L.r_frac0 = L.r_free;
    return EB_OK;
}

int fill_lif(eb_sweep *h, const float *lif_params, SweepLif &L) {
    const int en = L.en;
    memset(&L, 0, sizeof(L));
    L.en = en;
    L.e_exc = lif_params[0];
    L.e_inh = lif_params[1];
    L.e_leak = lif_params[2];
    L.v_thr = lif_params[3];
    L.g_leak = lif_params[8];
    L.inv_c_m = inv_double(lif_params[4]);
    const float dt_ms = h->dt * 1000.0f;
    const float el = (h->integ == INTEG_RK4) ? dt_ms * 0.5f : dt_ms;
    L.decay[0] = decay_factor(el, lif_params[5]);
    L.decay[1] = decay_factor(el, lif_params[6]);
    if (refractory_classes(lif_params[7], h->dt, L)) {
        set_error("refractory period %g ms unsupported at dt %g s", lif_params[7], h->dt);
        return EB_ERR_UNSUPPORTED;
    }
    return EB_OK;
}

}  // namespace

extern "C" {

int eb_sweep_create(int device, int n_networks, int integrator, float dt_s, float delay_s, uint64_t seed,
                    eb_sweep **out) {
    if (!out || n_networks <= 0 || n_networks > 65535 || integrator < INTEG_EULER || integrator > INTEG_RK4 || !(dt_s > 0) ||
        !(delay_s > 0)) {
        set_error("eb_sweep_create: bad argument (1..65535 networks, integrator Euler/RK2/RK4, dt > 0, delay > 0)");
        return EB_ERR_ARG;
    }
    SK(cudaSetDevice(device));
    eb_sweep *h = new eb_sweep();
    h->device = device;
    h->n_nets = n_networks;
    h->integ = integrator;
    h->dt = dt_s;
    h->delay = delay_s;
    h->seed = seed;
    h->nets.resize(n_networks);
    h->in_time.resize(n_networks);
    h->in_cell.resize(n_networks);
    h->xsrc.resize(n_networks);
    h->xtgt.resize(n_networks);
    h->xw.resize(n_networks);
    for (auto &s : h->nets) memset(&s, 0, sizeof(s));
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete h;
        set_error("stream: %s", cudaGetErrorString(e));
        return EB_ERR_CUDA;
    }
    *out = h;
    return EB_OK;
}

int eb_sweep_destroy(eb_sweep *h) {
    if (h) {
        cudaSetDevice(h->device);
        delete h;
    }
    return EB_OK;
}

int eb_sweep_set_network(eb_sweep *h, int i, int n, int n_in, int n_exc, const float *lif_params, float p,
                         float w_exc_max, float w_inh_max, float w_in_max) {
    if (!h || i < 0 || i >= h->n_nets || n <= 0 || n > kSweepMaxN || n_in < 0 || n + n_in > 65535 || n_exc < 0 ||
        n_exc > n || !lif_params || !(p >= 0.0f && p <= 1.0f)) {
        set_error("eb_sweep_set_network: bad argument (1 <= n <= %d, n + n_in <= 65535, 0 <= p <= 1)", kSweepMaxN);
        return EB_ERR_ARG;
    }
    if (h->built) { set_error("eb_sweep_set_network after eb_sweep_build"); return EB_ERR_STATE; }
    SweepNet &S = h->nets[i];
    S.n = n;
    S.n_in = n_in;
    S.n_exc = n_exc;
    S.wn = (n + 31) / 32;
    S.p = p;
    S.w_max[0] = w_exc_max;
    S.w_max[1] = w_inh_max;
    S.w_max[2] = w_in_max;
    for (int j = 0; j < 10; ++j) S.params[j] = lif_params[j];
    S.explicit_syn = 0;
    h->xsrc[i].clear();
    h->xtgt[i].clear();
    h->xw[i].clear();
    S.L.en = 0;
    const int rc = fill_lif(h, lif_params, S.L);
    if (rc) return rc;
    return EB_OK;
}

int eb_sweep_set_inputs(eb_sweep *h, int i, int64_t n, const float *time_s, const int32_t *cell) {
    if (!h || i < 0 || i >= h->n_nets || n < 0 || (n > 0 && (!time_s || !cell))) {
        set_error("eb_sweep_set_inputs: bad argument");
        return EB_ERR_ARG;
    }
    if (h->built) { set_error("eb_sweep_set_inputs after eb_sweep_build"); return EB_ERR_STATE; }
    for (int64_t q = 0; q < n; ++q)
        if (!(time_s[q] >= 0.0f)) { set_error("input spike %lld: negative or NaN time", (long long)q); return EB_ERR_ARG; }
    h->in_time[i].assign(time_s, time_s + n);
    h->in_cell[i].assign(cell, cell + n);
    return EB_OK;
}

int eb_sweep_set_synapses(eb_sweep *h, int i, int64_t m, const int32_t *src, const int32_t *tgt, const float *w) {
    if (!h || i < 0 || i >= h->n_nets || m < 0 || (m > 0 && (!src || !tgt || !w))) {
        set_error("eb_sweep_set_synapses: bad argument");
        return EB_ERR_ARG;
    }
    if (h->built) { set_error("eb_sweep_set_synapses after eb_sweep_build"); return EB_ERR_STATE; }
    SweepNet &S = h->nets[i];
    if (S.n <= 0) { set_error("eb_sweep_set_synapses: eb_sweep_set_network(%d) first", i); return EB_ERR_STATE; }
    for (int64_t k = 0; k < m; ++k)
        if (src[k] < 0 || src[k] >= S.n + S.n_in || tgt[k] < 0 || tgt[k] >= S.n) {
            set_error("eb_sweep_set_synapses: synapse %lld out of range", (long long)k);
            return EB_ERR_ARG;
        }
    h->xsrc[i].assign(src, src + m);
    h->xtgt[i].assign(tgt, tgt + m);
    h->xw[i].assign(w, w + m);
    S.explicit_syn = 1;
    return EB_OK;
}

int eb_sweep_build(eb_sweep *h, int64_t n_steps_max, float max_rate_hz) {
    if (!h || n_steps_max <= 0 || n_steps_max > (1 << 28) || !(max_rate_hz > 0)) {
        set_error("eb_sweep_build: bad argument");
        return EB_ERR_ARG;
    }
    if (h->built) { set_error("eb_sweep_build: already built"); return EB_ERR_STATE; }
    SK(cudaSetDevice(h->device));
    const int N = h->n_nets;
    for (int i = 0; i < N; ++i)
        if (h->nets[i].n <= 0) { set_error("eb_sweep_build: network %d not set", i); return EB_ERR_STATE; }
    // update times (the plain path's double accumulation) and the arrival step of
    // each source step: the first k with t_k > t_j + d
    const int64_t units = delay_units(h->delay);
    const double dd = (double)units * 0.0001;
    const int64_t T = n_steps_max + (int64_t)std::ceil(dd / (double)h->dt) + 16;
    std::vector<double> t(T + 1);
    t[0] = 0.0;
    for (int64_t k = 1; k <= T; ++k) t[k] = t[k - 1] + (double)h->dt;
    std::vector<int32_t> grp_lo(n_steps_max + 2, 0);
    std::vector<int8_t> grp_n(n_steps_max + 2, 0);
    h->h_arr_step.assign(n_steps_max + 1, INT32_MAX);
    int64_t dmax = 1, lag = INT32_MAX;
    {
        int64_t ka = 2;
        for (int64_t j = 1; j <= n_steps_max; ++j) {
            const double a = t[j] + dd;
            if (ka < j + 1) ka = j + 1;
            while (ka <= T && t[ka] <= a) ++ka;
            if (ka > n_steps_max) break;
            h->h_arr_step[j] = (int32_t)ka;
            if (grp_n[ka] == 0) grp_lo[ka] = (int32_t)j;
            if (++grp_n[ka] > kMaxGroups) { set_error("eb_sweep_build: dt too small for the delay grid"); return EB_ERR_UNSUPPORTED; }
            dmax = std::max(dmax, ka - j);
            lag = std::min(lag, ka - j);
        }
    }
    const SweepRing ring = sweep_ring(dmax, lag);
    const int R = ring.slots;
    h->G.window = ring.window;
    h->G.R = R;
    h->G.steps_max = (int)n_steps_max;
    h->G.dt_ms = h->dt * 1000.0f;
    h->G.integ = h->integ;
    // layout and input arrivals
    int64_t src_off = 0, state_off = 0, in_off = 0, ring_off = 0, rec_off = 0;
    std::vector<int32_t> in_key;
    std::vector<uint16_t> in_src;
    h->max_n = 0;
    for (int i = 0; i < N; ++i) {
        SweepNet &S = h->nets[i];
        S.src_off = src_off;
        src_off += S.n + S.n_in + 1;
        S.state_off = state_off;
        state_off += S.n;
        S.ring_off = ring_off;
        ring_off += (int64_t)R * S.wn;
        S.rec_off = rec_off;
        S.rec_cap = (int64_t)std::ceil((double)S.n * (double)n_steps_max * (double)h->dt * (double)max_rate_hz) + 64;
        rec_off += S.rec_cap;
        h->max_n = std::max(h->max_n, S.n);
        // input spikes: arrival a = t_in + d reaches the first step with t_k > a;
        // phase = arriving source steps with a_j <= a (their spikes come first)
        struct Rec { int32_t key; float time; int32_t cell; };
        std::vector<Rec> recs;
        recs.reserve(h->in_time[i].size());
        for (size_t q = 0; q < h->in_time[i].size(); ++q) {
            const int32_t c = h->in_cell[i][q];
            if (c < 0 || c >= S.n_in) { set_error("network %d: input cell %d out of range", i, c); return EB_ERR_ARG; }
            const double a = (double)h->in_time[i][q] + dd;
            const int64_t ka = std::upper_bound(t.begin() + 1, t.end(), a) - t.begin();
            if (ka > n_steps_max) continue;
            int phase = 0;
            for (int g = 0; g < grp_n[ka]; ++g)
                if (t[grp_lo[ka] + g] + dd <= a) phase = g + 1;
            recs.push_back({(int32_t)(ka * 4 + phase), h->in_time[i][q], c});
        }
        std::stable_sort(recs.begin(), recs.end(), [](const Rec &x, const Rec &y) {
            if (x.key != y.key) return x.key < y.key;
            if (x.time != y.time) return x.time < y.time;
            return x.cell < y.cell;
        });
        S.in_off = in_off;
        S.n_in_spikes = (int64_t)recs.size();
        for (const Rec &x : recs) {
            in_key.push_back(x.key);
            in_src.push_back((uint16_t)x.cell);
        }
        in_off += (int64_t)recs.size();
    }
    h->state_n = state_off;
    h->ring_words = ring_off;
    h->n_sources = src_off;
    h->h_in_key = in_key;
    h->G.n_total = state_off;
    int rc;
    SweepNet *d_nets;
    if ((rc = h->upload((void **)&d_nets, h->nets.data(), sizeof(SweepNet) * N))) return rc;
    h->d_nets = d_nets;
    h->G.nets = d_nets;
    h->G.n_nets = N;
    // connectivity: count per source, scan on the host, fill
    uint32_t *d_optr;
    if ((rc = h->upload((void **)&d_optr, nullptr, sizeof(uint32_t) * (size_t)src_off))) return rc;
    SK(cudaMemsetAsync(d_optr, 0, sizeof(uint32_t) * (size_t)src_off, h->stream));
    k_sweep_count<<<dim3(512, N), 256, 0, h->stream>>>(d_nets, h->seed, d_optr);
    SK(cudaGetLastError());
    std::vector<uint32_t> cnt(src_off);
    SK(cudaMemcpyAsync(cnt.data(), d_optr, sizeof(uint32_t) * (size_t)src_off, cudaMemcpyDeviceToHost, h->stream));
    SK(cudaStreamSynchronize(h->stream));
    // explicit networks: synapses sorted by (source, target), the reference's order
    // for one delay (qsort_inters, src/spike/Network.cpp:45-68), ties by caller order
    std::vector<std::vector<int64_t>> xord(N);
    for (int i = 0; i < N; ++i) {
        if (!h->nets[i].explicit_syn) continue;
        const SweepNet &S = h->nets[i];
        auto &o = xord[i];
        o.resize(h->xsrc[i].size());
        for (size_t k = 0; k < o.size(); ++k) o[k] = (int64_t)k;
        const auto &xs = h->xsrc[i], &xt = h->xtgt[i];
        std::stable_sort(o.begin(), o.end(), [&](int64_t a, int64_t b) {
            return xs[a] != xs[b] ? xs[a] < xs[b] : xt[a] < xt[b];
        });
        for (size_t k = 1; k < o.size(); ++k)
            if (xs[o[k]] == xs[o[k - 1]] && xt[o[k]] == xt[o[k - 1]]) {
                set_error("network %d: two synapses from %d to %d (one per pair in a sweep network)", i, xs[o[k]], xt[o[k]]);
                return EB_ERR_UNSUPPORTED;
            }
        for (int s = 0; s < S.n + S.n_in; ++s) cnt[S.src_off + s] = 0;
        for (size_t k = 0; k < o.size(); ++k) cnt[S.src_off + xs[k]]++;
    }
    int64_t syn_off = 0;
    for (int i = 0; i < N; ++i) {
        SweepNet &S = h->nets[i];
        S.syn_off = syn_off;
        uint64_t acc = 0, n_e = 0, n_i = 0;
        for (int s = 0; s < S.n + S.n_in; ++s) {
            const uint32_t c = cnt[S.src_off + s];
            cnt[S.src_off + s] = (uint32_t)acc;
            acc += c;
            if (s >= S.n_exc && s < S.n) n_i += c; else n_e += c;
        }
        if (acc > 0xffffffffull) { set_error("network %d: too many synapses", i); return EB_ERR_UNSUPPORTED; }
        cnt[S.src_off + S.n + S.n_in] = (uint32_t)acc;
        syn_off += (int64_t)acc;
        // conductance types present among the network's synapses
        S.L.en = (n_e ? 1 : 0) | (n_i ? 2 : 0);
    }
    h->total_syn = syn_off;
    SK(cudaMemcpy(d_nets, h->nets.data(), sizeof(SweepNet) * N, cudaMemcpyHostToDevice));
    SK(cudaMemcpy(d_optr, cnt.data(), sizeof(uint32_t) * (size_t)src_off, cudaMemcpyHostToDevice));
    h->G.optr = d_optr;
    uint16_t *d_tgt;
    float *d_w;
    if ((rc = h->upload((void **)&d_tgt, nullptr, sizeof(uint16_t) * (size_t)syn_off))) return rc;
    if ((rc = h->upload((void **)&d_w, nullptr, sizeof(float) * (size_t)syn_off))) return rc;
    h->G.tgt = d_tgt;
    h->G.w = d_w;
    k_sweep_fill<<<dim3(64, N), 256, 0, h->stream>>>(d_nets, d_optr, h->seed, d_tgt, d_w);
    SK(cudaGetLastError());
    // explicit networks' targets and weights, and the sweep -> caller synapse order
    {
        std::vector<int64_t> perm(syn_off);
        std::vector<uint16_t> xt;
        std::vector<float> xw;
        for (int i = 0; i < N; ++i) {
            const SweepNet &S = h->nets[i];
            const int64_t mi = (i + 1 < N ? h->nets[i + 1].syn_off : syn_off) - S.syn_off;
            if (!S.explicit_syn) {
                for (int64_t k = 0; k < mi; ++k) perm[S.syn_off + k] = S.syn_off + k;
                continue;
            }
            const auto &o = xord[i];
            xt.resize(o.size());
            xw.resize(o.size());
            for (size_t k = 0; k < o.size(); ++k) {
                xt[k] = (uint16_t)h->xtgt[i][o[k]];
                xw[k] = h->xw[i][o[k]];
                perm[S.syn_off + (int64_t)k] = S.syn_off + o[k];
            }
            if (!o.empty()) {
                SK(cudaMemcpyAsync(d_tgt + S.syn_off, xt.data(), sizeof(uint16_t) * o.size(), cudaMemcpyHostToDevice, h->stream));
                SK(cudaMemcpyAsync(d_w + S.syn_off, xw.data(), sizeof(float) * o.size(), cudaMemcpyHostToDevice, h->stream));
                SK(cudaStreamSynchronize(h->stream));
            }
        }
        if ((rc = h->upload((void **)&h->perm, perm.data(), sizeof(int64_t) * perm.size()))) return rc;
    }
    // state and tables
    if ((rc = h->upload((void **)&h->G.V, nullptr, sizeof(float) * (size_t)state_off))) return rc;
    if ((rc = h->upload((void **)&h->G.gE, nullptr, sizeof(float) * (size_t)state_off))) return rc;
    if ((rc = h->upload((void **)&h->G.gI, nullptr, sizeof(float) * (size_t)state_off))) return rc;
    if ((rc = h->upload((void **)&h->G.refr, nullptr, sizeof(int32_t) * (size_t)state_off))) return rc;
    if ((rc = h->upload((void **)&h->G.ring, nullptr, sizeof(uint32_t) * (size_t)ring_off))) return rc;
    if ((rc = h->upload((void **)&h->G.grp_lo, grp_lo.data(), sizeof(int32_t) * grp_lo.size()))) return rc;
    if ((rc = h->upload((void **)&h->G.grp_n, grp_n.data(), sizeof(int8_t) * grp_n.size()))) return rc;
    if ((rc = h->upload((void **)&h->G.in_key, in_key.data(), sizeof(int32_t) * in_key.size()))) return rc;
    if ((rc = h->upload((void **)&h->G.in_src, in_src.data(), sizeof(uint16_t) * in_src.size()))) return rc;
    if ((rc = h->upload((void **)&h->G.in_cursor, nullptr, sizeof(int64_t) * N))) return rc;
    if ((rc = h->upload((void **)&h->G.rec, nullptr, sizeof(uint16_t) * (size_t)rec_off))) return rc;
    if ((rc = h->upload((void **)&h->G.rec_end, nullptr, sizeof(int32_t) * (size_t)N * n_steps_max))) return rc;
    if ((rc = h->upload((void **)&h->G.rec_cnt, nullptr, sizeof(uint32_t) * N))) return rc;
    if ((rc = h->upload((void **)&h->G.events, nullptr, sizeof(unsigned long long) * N))) return rc;
    if ((rc = h->upload((void **)&h->G.flags, nullptr, sizeof(uint32_t)))) return rc;
    if ((rc = h->upload((void **)&h->G.queue, nullptr, sizeof(int)))) return rc;
    if ((rc = h->upload((void **)&h->G.step, nullptr, sizeof(int64_t)))) return rc;
    if ((rc = h->upload((void **)&h->d_arr_step, h->h_arr_step.data(), sizeof(int32_t) * h->h_arr_step.size()))) return rc;
    std::vector<int32_t> order(N);
    for (int i = 0; i < N; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return h->nets[a].n > h->nets[b].n; });
    if ((rc = h->upload((void **)&h->G.order, order.data(), sizeof(int32_t) * N))) return rc;
    SK(cudaStreamSynchronize(h->stream));
    h->built = true;
    if ((rc = eb_sweep_reset(h))) return rc;
    return eb_sweep_configure(h, 0, 0);
}

int eb_sweep_reset(eb_sweep *h) {
    if (!h || !h->built) { set_error("eb_sweep_reset: sweep not built"); return EB_ERR_STATE; }
    SK(cudaSetDevice(h->device));
    int rc = upload_params(h, h->stream);
    if (rc) return rc;
    h->counts_ok = false;
    k_sweep_reset<<<dim3(8, h->n_nets), 256, 0, h->stream>>>(h->G);
    SK(cudaGetLastError());
    SK(cudaStreamSynchronize(h->stream));
    h->steps_done = 0;
    h->needs_reset = false;
    h->ckpt_upto = h->ckpt_every > 0 ? 0 : -1;
    return EB_OK;
}

int eb_sweep_configure(eb_sweep *h, int block, int steps_per_launch) {
    if (!h || !h->built) { set_error("eb_sweep_configure: sweep not built"); return EB_ERR_STATE; }
    SK(cudaSetDevice(h->device));
    int nsm = 0;
    SK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device));
    // CTAs per network: with fewer networks than SMs, as many as leave each at least
    // kTileMin neurons on average of the largest network, and the SMs one CTA each.  Each
    // halving of the tile halves the update, while listing and meeting repeat: 24
    // networks of up to 1,500, RK4, 500 steps with read-backs: 1.97 ms on one CTA, 1.77
    // on two, 1.58 on four; 8 networks of up to 10,000, a fitting step: 14.4 ms on two,
    // 9.2 on eight.
    int ctas = 1;
    while (ctas < 8 && 2 * ctas * h->n_nets <= nsm && 2 * ctas * kTileMin <= h->max_n) ctas *= 2;
    const int words = (h->max_n + 31) / 32;
    int max_smem = 0;
    SK(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device));
    auto tile_of = [&](int c) { return (words + c - 1) / c * 32; };
    // sources a pass lists: 128, or 64 where the state needs the shared memory
    auto smem_of = [&](int c, int cap) { return sweep_smem_bytes(tile_of(c), h->G.R, words, h->G.window, cap); };
    const size_t room = (size_t)max_smem - 1024;
    while (ctas < 8 && smem_of(ctas, 64) > room) ctas *= 2;
    const int cap = smem_of(ctas, 128) <= room ? 128 : 64;
    const int tile = tile_of(ctas);
    int nb = block ? block : h->block;
    // threads per CTA unless the caller chose: two CTAs of 512 share an SM; a lone one
    // takes 1,024 when its tile gives them two neurons each, and fewer than 512 only
    // leave warps without a neuron out
    if (!nb) {
        nb = 512;
        if ((int64_t)ctas * h->n_nets <= nsm && tile >= 2048) nb = 1024;
        while (nb > 128 && nb / 2 >= tile) nb /= 2;
    }
    if (nb != 128 && nb != 256 && nb != 512 && nb != 1024) { set_error("block must be 128, 256, 512 or 1024"); return EB_ERR_ARG; }
    if (steps_per_launch < 0) { set_error("steps_per_launch < 0"); return EB_ERR_ARG; }
    const size_t smem = smem_of(ctas, cap);
    // The attribute belongs to the kernel, not to the handle: every handle sets the most
    // there is, so that none takes away what another one's launches need, in whatever order
    // their threads come here.
    for (bool traj : {false, true}) {
        const cudaError_t e = smem > room ? cudaErrorInvalidValue
                                          : cudaFuncSetAttribute((const void *)sweep_fn(h->integ, traj, ctas > 1),
                                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room);
        if (e != cudaSuccess) {
            cudaGetLastError();
            set_error("sweep kernel: %zu bytes of shared memory unavailable (%s)", smem, cudaGetErrorString(e));
            return EB_ERR_UNSUPPORTED;
        }
    }
    int occ = 0;
    SK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, sweep_fn(h->integ, false, ctas > 1), nb, smem));
    if (occ < 1) {
        set_error("sweep kernel does not fit (block %d, %zu bytes of shared memory)", nb, smem);
        return EB_ERR_UNSUPPORTED;
    }
    const int cl = ctas == 8 ? 3 : ctas / 2;  // log2
    if (ctas > 1 && !h->tile_ptr[cl]) {
        int rc = h->dalloc((void **)&h->tile_ptr[cl], sizeof(uint32_t) * (size_t)h->n_sources * (ctas + 1));
        if (rc) return rc;
        k_sweep_tiles<<<dim3(64, h->n_nets), 256, 0, h->stream>>>(h->G, ctas, h->tile_ptr[cl]);
        SK(cudaGetLastError());
    }
    h->block = nb;
    h->max_tile = tile;
    h->wc = words;
    h->smem = smem;
    h->G.ctas = ctas;
    h->G.list_cap = cap;
    h->G.tptr = ctas > 1 ? h->tile_ptr[cl] : h->G.optr;
    h->G.tstride = ctas > 1 ? ctas + 1 : 1;
    h->grid = ctas > 1 ? ctas * h->n_nets : std::min(occ * nsm, h->n_nets);
    if (steps_per_launch) h->steps_per_launch = steps_per_launch;
    if (h->graph) {
        cudaGraphExecDestroy(h->graph);
        h->graph = nullptr;
        h->graph_chunks = 0;
    }
    return EB_OK;
}

int eb_sweep_run_async(eb_sweep *h, int64_t n_steps) {
    if (!h || !h->built) { set_error("eb_sweep_run: sweep not built"); return EB_ERR_STATE; }
    if (h->needs_reset) { set_error("eb_sweep_run: the adjoint left the sweep mid-run; eb_sweep_reset first"); return EB_ERR_STATE; }
    if (n_steps < 0 || h->steps_done + n_steps > h->G.steps_max) {
        set_error("eb_sweep_run: %lld steps exceed the %d built for", (long long)(h->steps_done + n_steps), h->G.steps_max);
        return EB_ERR_ARG;
    }
    SK(cudaSetDevice(h->device));
    h->counts_ok = false;
    if (int rc = upload_params(h, h->stream)) return rc;
    if (h->ckpt_every > 0) {
        // chunks aligned to the checkpoint interval, the state saved before each
        const int E = h->ckpt_every;
        if (h->steps_done % E) { set_error("eb_sweep_run: checkpointed runs start at a multiple of %d steps", E); return EB_ERR_STATE; }
        const bool from0 = h->ckpt_upto == h->steps_done;
        int64_t done = 0;
        while (done < n_steps) {
            const int64_t k = h->steps_done + done;
            const int len = (int)std::min<int64_t>(E, n_steps - done);
            int rc = checkpoint_save(h, (int)(k / E), h->stream);
            if (!rc) rc = enqueue_chunk(h, len, h->stream);
            if (rc) return rc;
            done += len;
        }
        h->steps_done += n_steps;
        h->ckpt_upto = from0 ? h->steps_done : -1;
        return EB_OK;
    }
    const int spl = h->steps_per_launch;
    const int chunks = (int)(n_steps / spl);
    if (chunks > 0) {
        // the multi-step loop as one CUDA graph: chunks x (sweep kernel, advance)
        if (!h->graph || h->graph_chunks != chunks) {
            if (h->graph) cudaGraphExecDestroy(h->graph);
            h->graph = nullptr;
            cudaGraph_t g;
            SK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
            int rc = EB_OK;
            for (int c = 0; c < chunks && rc == EB_OK; ++c) rc = enqueue_chunk(h, spl, h->stream);
            cudaError_t e = cudaStreamEndCapture(h->stream, &g);
            if (rc) return rc;
            SK(e);
            e = cudaGraphInstantiate(&h->graph, g, 0);
            cudaGraphDestroy(g);
            SK(e);
            h->graph_chunks = chunks;
        }
        SK(cudaGraphLaunch(h->graph, h->stream));
    }
    const int rem = (int)(n_steps - (int64_t)chunks * spl);
    if (rem > 0) {
        int rc = enqueue_chunk(h, rem, h->stream);
        if (rc) return rc;
    }
    h->steps_done += n_steps;
    return EB_OK;
}

int eb_sweep_sync(eb_sweep *h) {
    if (!h || !h->built) { set_error("eb_sweep_sync: sweep not built"); return EB_ERR_STATE; }
    SK(cudaSetDevice(h->device));
    SK(cudaStreamSynchronize(h->stream));
    uint32_t f = 0;
    SK(cudaMemcpy(&f, h->G.flags, sizeof(f), cudaMemcpyDeviceToHost));
    if (f & FLAG_RECORD_OVERFLOW) { set_error("sweep: spike record overflow (raise max_rate_hz)"); return EB_ERR_OVERFLOW; }
    return EB_OK;
}

int eb_sweep_run(eb_sweep *h, int64_t n_steps) {
    int rc = eb_sweep_run_async(h, n_steps);
    if (rc) return rc;
    return eb_sweep_sync(h);
}

// Times `trial_steps` steps from the initial state for each launch configuration
// (threads per CTA, hence neurons per thread; steps per launch) and keeps the
// fastest.  Leaves the sweep reset to its initial state.
int eb_sweep_autotune(eb_sweep *h, int64_t trial_steps, int *best_block, int *best_spl, float *best_ms) {
    if (!h || !h->built || trial_steps <= 0 || trial_steps > h->G.steps_max) {
        set_error("eb_sweep_autotune: sweep not built or bad trial length");
        return EB_ERR_ARG;
    }
    SK(cudaSetDevice(h->device));
    cudaEvent_t e0, e1;
    SK(cudaEventCreate(&e0));
    SK(cudaEventCreate(&e1));
    const int blocks[4] = {128, 256, 512, 1024};
    const int64_t spls[2] = {std::max<int64_t>(1, trial_steps / 4), trial_steps};
    float best = 0;
    int bb = 0, bs = 0;
    int rc = EB_OK;
    bool warmed = false;
    for (int b : blocks) {
        for (int64_t s : spls) {
            if ((rc = eb_sweep_configure(h, b, (int)s))) {
                if (rc == EB_ERR_ARG || rc == EB_ERR_UNSUPPORTED) { rc = EB_OK; continue; }
                break;
            }
            for (int rep = warmed ? 1 : 0; rep < 2; ++rep) {
                if ((rc = eb_sweep_reset(h))) break;
                cudaEventRecord(e0, h->stream);
                if ((rc = eb_sweep_run_async(h, trial_steps))) break;
                cudaEventRecord(e1, h->stream);
                if ((rc = eb_sweep_sync(h))) break;
            }
            warmed = true;
            if (rc) break;
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            if (!bb || ms < best) { best = ms; bb = b; bs = (int)s; }
        }
        if (rc) break;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (!bb) { set_error("eb_sweep_autotune: no launch configuration fits"); return EB_ERR_UNSUPPORTED; }
    if ((rc = eb_sweep_configure(h, bb, bs))) return rc;
    if ((rc = eb_sweep_reset(h))) return rc;
    if (best_block) *best_block = bb;
    if (best_spl) *best_spl = bs;
    if (best_ms) *best_ms = best;
    return EB_OK;
}

int eb_sweep_get_spikes(eb_sweep *h, int i, int64_t cap, int64_t *n, int32_t *step, int32_t *cell) {
    if (!h || !h->built || i < 0 || i >= h->n_nets || !n || cap < 0) { set_error("eb_sweep_get_spikes: bad argument"); return EB_ERR_ARG; }
    SK(cudaSetDevice(h->device));
    const SweepNet &S = h->nets[i];
    const int64_t ns = h->steps_done;
    // The first query after a run brings every network's count at once, so that most size
    // queries copy nothing; a drain copies the steps' ends and the record, to pageable
    // memory.  24 networks, first read of a handle and later ones: 0.85 and 0.73 ms.  With
    // pinned memory, which took 2 ms and more to allocate whenever it grew, 5 ms and up to
    // hundreds, then 0.8; with the steps' ends copied for the size query, too, 1.5 and 1.4.
    // (An adjoint leaves the counts at an earlier step, the ends where they were.)
    int64_t cnt = 0;
    if (h->needs_reset && ns) {
        uint32_t c = 0;
        SK(cudaMemcpyAsync(&c, h->G.rec_end + (int64_t)i * h->G.steps_max + ns - 1, sizeof(c), cudaMemcpyDeviceToHost, h->stream));
        SK(cudaStreamSynchronize(h->stream));
        cnt = c;
    } else if (ns) {
        if (!h->counts_ok) {
            h->counts.resize(h->n_nets);
            SK(cudaMemcpyAsync(h->counts.data(), h->G.rec_cnt, sizeof(uint32_t) * h->n_nets, cudaMemcpyDeviceToHost, h->stream));
            SK(cudaStreamSynchronize(h->stream));
            h->counts_ok = true;
        }
        cnt = h->counts[i];
    }
    *n = cnt;
    if (cnt > S.rec_cap) { set_error("network %d: spike record overflowed (raise max_rate_hz)", i); return EB_ERR_OVERFLOW; }
    if (cnt > cap) { set_error("eb_sweep_get_spikes: buffer holds %lld of %lld spikes", (long long)cap, (long long)cnt); return EB_ERR_OVERFLOW; }
    if (!cnt) return EB_OK;
    if ((int64_t)h->ends.size() < ns) h->ends.resize(ns);
    if ((int64_t)h->cells.size() < cnt) h->cells.resize(cnt);
    const int32_t *end = h->ends.data();
    const uint16_t *buf = h->cells.data();
    SK(cudaMemcpyAsync(h->ends.data(), h->G.rec_end + (int64_t)i * h->G.steps_max, sizeof(int32_t) * (size_t)ns, cudaMemcpyDeviceToHost, h->stream));
    SK(cudaMemcpyAsync(h->cells.data(), h->G.rec + S.rec_off, sizeof(uint16_t) * (size_t)cnt, cudaMemcpyDeviceToHost, h->stream));
    SK(cudaStreamSynchronize(h->stream));
    int64_t b = 0;
    for (int64_t k = 0; k < ns; ++k) {
        const int64_t e = (uint32_t)end[k];
        for (int64_t q = b; q < e; ++q) {
            if (step) step[q] = (int32_t)(k + 1);
            if (cell) cell[q] = buf[q];
        }
        b = e;
    }
    return EB_OK;
}

int eb_sweep_spike_counts(eb_sweep *h, int64_t *counts) {
    if (!h || !h->built || !counts) { set_error("eb_sweep_spike_counts: bad argument"); return EB_ERR_ARG; }
    SK(cudaSetDevice(h->device));
    SK(cudaStreamSynchronize(h->stream));
    std::vector<uint32_t> c(h->n_nets);
    SK(cudaMemcpy(c.data(), h->G.rec_cnt, sizeof(uint32_t) * h->n_nets, cudaMemcpyDeviceToHost));
    for (int i = 0; i < h->n_nets; ++i) counts[i] = c[i];
    return EB_OK;
}

int eb_sweep_get_synapses(eb_sweep *h, int i, int64_t cap, int64_t *m, int32_t *src, int32_t *tgt, float *w) {
    if (!h || !h->built || i < 0 || i >= h->n_nets || !m || cap < 0) { set_error("eb_sweep_get_synapses: bad argument"); return EB_ERR_ARG; }
    SK(cudaSetDevice(h->device));
    SK(cudaStreamSynchronize(h->stream));
    const SweepNet &S = h->nets[i];
    const int ns = S.n + S.n_in;
    std::vector<uint32_t> optr(ns + 1);
    SK(cudaMemcpy(optr.data(), h->G.optr + S.src_off, sizeof(uint32_t) * (ns + 1), cudaMemcpyDeviceToHost));
    const int64_t mm = optr[ns];
    *m = mm;
    if (mm > cap) { set_error("eb_sweep_get_synapses: buffer holds %lld of %lld synapses", (long long)cap, (long long)mm); return EB_ERR_OVERFLOW; }
    std::vector<uint16_t> t(mm);
    if (mm) {
        SK(cudaMemcpy(t.data(), h->G.tgt + S.syn_off, sizeof(uint16_t) * mm, cudaMemcpyDeviceToHost));
        if (w) SK(cudaMemcpy(w, h->G.w + S.syn_off, sizeof(float) * mm, cudaMemcpyDeviceToHost));
    }
    for (int s = 0; s < ns; ++s)
        for (int64_t o = optr[s]; o < (int64_t)optr[s + 1]; ++o) {
            if (src) src[o] = s;
            if (tgt) tgt[o] = t[o];
        }
    return EB_OK;
}

int eb_sweep_get_state(eb_sweep *h, int i, int var, float *out) {
    if (!h || !h->built || i < 0 || i >= h->n_nets || var < 0 || var > 2 || !out) { set_error("eb_sweep_get_state: bad argument"); return EB_ERR_ARG; }
    SK(cudaSetDevice(h->device));
    SK(cudaStreamSynchronize(h->stream));
    const float *src = var == 0 ? h->G.V : (var == 1 ? h->G.gE : h->G.gI);
    SK(cudaMemcpy(out, src + h->nets[i].state_off, sizeof(float) * h->nets[i].n, cudaMemcpyDeviceToHost));
    return EB_OK;
}

int eb_sweep_info(eb_sweep *h, int64_t *synapses, int64_t *device_bytes, int64_t *events, int *block,
                  int *steps_per_launch, int *grid) {
    if (!h) { set_error("eb_sweep_info: null handle"); return EB_ERR_ARG; }
    if (synapses) *synapses = h->total_syn;
    if (device_bytes) *device_bytes = h->dev_bytes;
    if (events) {
        *events = 0;
        if (h->built) {
            SK(cudaSetDevice(h->device));
            SK(cudaStreamSynchronize(h->stream));
            std::vector<unsigned long long> ev(h->n_nets);
            SK(cudaMemcpy(ev.data(), h->G.events, sizeof(unsigned long long) * h->n_nets, cudaMemcpyDeviceToHost));
            for (auto v : ev) *events += (int64_t)v;
        }
    }
    if (block) *block = h->block;
    if (steps_per_launch) *steps_per_launch = h->steps_per_launch;
    if (grid) *grid = h->grid;
    return EB_OK;
}

int eb_sweep_stream(eb_sweep *h, void **stream) {
    if (!h || !stream) { set_error("eb_sweep_stream: bad argument"); return EB_ERR_ARG; }
    *stream = (void *)h->stream;
    return EB_OK;
}

int eb_sweep_set_params(eb_sweep *h, int i, const float *lif_params) {
    if (!h || i < 0 || i >= h->n_nets || !lif_params || h->nets[i].n <= 0) { set_error("eb_sweep_set_params: bad argument"); return EB_ERR_ARG; }
    SweepNet &S = h->nets[i];
    SweepLif L = S.L;
    int rc = fill_lif(h, lif_params, L);
    if (rc) return rc;
    S.L = L;
    for (int j = 0; j < 10; ++j) S.params[j] = lif_params[j];
    h->nets_dirty = h->built;  // all changed networks go to the device at once, before the next launch
    return EB_OK;
}

namespace {
__global__ void k_perm_gather(const int64_t *perm, int64_t m, const float *src, float *dst) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < m; p += (int64_t)gridDim.x * blockDim.x)
        dst[p] = src[perm[p]];
}
__global__ void k_perm_scatter(const int64_t *perm, int64_t m, const float *src, float *dst) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < m; p += (int64_t)gridDim.x * blockDim.x)
        dst[perm[p]] = src[p];
}
}  // namespace

static int weights_io(eb_sweep *h, float *buf, int on_device, int to_sweep) {
    if (!h || !h->built || !buf) { set_error("eb_sweep weights: sweep not built or null buffer"); return EB_ERR_ARG; }
    SK(cudaSetDevice(h->device));
    const int64_t m = h->total_syn;
    if (!m) return EB_OK;
    float *dev = buf;
    float *tmp = nullptr;
    if (!on_device) {
        SK(cudaMallocAsync((void **)&tmp, sizeof(float) * m, h->stream));
        dev = tmp;
        if (to_sweep) SK(cudaMemcpyAsync(tmp, buf, sizeof(float) * m, cudaMemcpyHostToDevice, h->stream));
    }
    float *w = const_cast<float *>(h->G.w);
    if (to_sweep) k_perm_gather<<<592, 256, 0, h->stream>>>(h->perm, m, dev, w);
    else k_perm_scatter<<<592, 256, 0, h->stream>>>(h->perm, m, w, dev);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && !on_device && !to_sweep) e = cudaMemcpyAsync(buf, tmp, sizeof(float) * m, cudaMemcpyDeviceToHost, h->stream);
    if (tmp) cudaFreeAsync(tmp, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) { set_error("eb_sweep weights: %s", cudaGetErrorString(e)); return EB_ERR_CUDA; }
    return EB_OK;
}

int eb_sweep_set_weights(eb_sweep *h, const float *w, int on_device) {
    return weights_io(h, const_cast<float *>(w), on_device, 1);
}

int eb_sweep_get_weights(eb_sweep *h, float *w, int on_device) { return weights_io(h, w, on_device, 0); }

int eb_sweep_set_observed(eb_sweep *h, int m, const int32_t *idx) {
    if (!h || !h->built || m < 0 || (m > 0 && !idx)) { set_error("eb_sweep_set_observed: sweep not built or bad argument"); return EB_ERR_ARG; }
    for (int i = 0; i < h->n_nets; ++i)
        for (int q = 0; q < m; ++q)
            if (idx[(int64_t)i * m + q] < 0 || idx[(int64_t)i * m + q] >= h->nets[i].n) {
                set_error("eb_sweep_set_observed: network %d index %d out of range", i, idx[(int64_t)i * m + q]);
                return EB_ERR_ARG;
            }
    if (m <= h->G.n_obs && m > 0) {
        SK(cudaMemcpy((void *)h->G.obs, idx, sizeof(int32_t) * (size_t)h->n_nets * m, cudaMemcpyHostToDevice));
    } else if (m > 0) {
        int rc;
        int32_t *d_obs;
        float *d_trace;
        if ((rc = h->upload((void **)&d_obs, idx, sizeof(int32_t) * (size_t)h->n_nets * m))) return rc;
        if ((rc = h->dalloc((void **)&d_trace, sizeof(float) * (size_t)h->n_nets * h->G.steps_max * m))) return rc;
        h->G.obs = d_obs;
        h->G.trace = d_trace;
    }
    h->G.n_obs = m;
    h->obs_slot_ok = false;
    if (h->graph) {
        cudaGraphExecDestroy(h->graph);
        h->graph = nullptr;
        h->graph_chunks = 0;
    }
    return EB_OK;
}

int eb_sweep_get_trace(eb_sweep *h, float *out, int on_device) {
    if (!h || !h->built || !out) { set_error("eb_sweep_get_trace: bad argument"); return EB_ERR_ARG; }
    const int m = h->G.n_obs;
    if (!m || !h->steps_done) return EB_OK;
    SK(cudaSetDevice(h->device));
    const size_t row = sizeof(float) * (size_t)h->steps_done * m;
    const size_t pitch = sizeof(float) * (size_t)h->G.steps_max * m;
    SK(cudaMemcpy2DAsync(out, row, h->G.trace, pitch, row, h->n_nets,
                         on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, h->stream));
    SK(cudaStreamSynchronize(h->stream));
    return EB_OK;
}

int eb_sweep_set_checkpoints(eb_sweep *h, int every) {
    if (!h || !h->built || every < 0) { set_error("eb_sweep_set_checkpoints: sweep not built or bad interval"); return EB_ERR_ARG; }
    if (every == 0) { h->ckpt_every = 0; return EB_OK; }
    if (every > 255) { set_error("eb_sweep_set_checkpoints: at most 255 steps between checkpoints"); return EB_ERR_ARG; }
    SK(cudaSetDevice(h->device));
    const int n = (int)((h->G.steps_max + every - 1) / every);
    const size_t b = checkpoint_bytes(h);
    while ((int)h->ckpt.size() < n) {
        void *p;
        int rc = h->dalloc(&p, b);
        if (rc) return rc;
        h->ckpt.push_back(p);
    }
    h->ckpt_every = every;
    h->n_ckpt = n;
    h->ckpt_upto = h->steps_done == 0 ? 0 : -1;
    return EB_OK;
}

}  // extern "C"
