// Functional delivery op: fold a batch of synaptic arrivals into conductance
// arrays in the reference's delivery order, on the device.
//
// The reference CPU models add each arriving weight straight into the target's
// conductance as the event is processed (NeuronModel::ProcessInputSpike,
// src/neuron_model/LIFTimeDrivenModel.cpp:77-83), i.e. per target in order of
// arrival time, ties in event order (src/spike/PropagatedSpikeGroup.cpp:112-149);
// its GPU models instead sum a step's arrivals on the host into AuxState
// (src/neuron_model/LIFTimeDrivenModel_GPU_C_INTERFACE.cu:66-70).  This op gives
// a host-driven engine the CPU models' rounding on the GPU: arrivals are grouped
// per target (linked lists -- integer atomics only), sorted per target by (time,
// position in the batch), and added in that order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "edlut_b200.h"
#include "eb_runtime.h"

using namespace eb;

namespace {

struct FoldRec {
    double t;
    uint32_t i;
    uint32_t pad;
};

__device__ __forceinline__ bool fold_less(const FoldRec &a, const FoldRec &b) {
    return a.t < b.t || (a.t == b.t && a.i < b.i);
}

// Arrivals of one target as a linked list: the last linked arrival (kNone: none) and how
// many more there are, less one (most targets' only arrival takes one atomic); next[i] is
// the arrival linked before arrival i.  The order of the links is whatever the atomics
// give; the fold sorts.
constexpr uint32_t kNone = 0xffffffffu;
struct alignas(8) FoldList {
    uint32_t last, more;
};

__global__ void __launch_bounds__(256) k_fold_link(int64_t n, const int32_t *__restrict__ target, FoldList *list,
                                                   uint32_t *__restrict__ next) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        FoldList *l = list + target[i];
        const uint32_t before = atomicExch(&l->last, (uint32_t)i);
        next[i] = before;
        if (before != kNone) atomicAdd(&l->more, 1u);
    }
}

// Restore the heap property below node j of the max-heap r[0..c) by (time, index).
__device__ __forceinline__ void sift_down(FoldRec *r, uint32_t j, uint32_t c) {
    const FoldRec v = r[j];
    for (;;) {
        uint32_t ch = 2 * j + 1;
        if (ch >= c) break;
        if (ch + 1 < c && fold_less(r[ch], r[ch + 1])) ++ch;
        if (!fold_less(v, r[ch])) break;
        r[j] = r[ch];
        j = ch;
    }
    r[j] = v;
}

// Sort r[0..c) by (time, index) in place: insertion sort for the few arrivals a
// target usually gets, heapsort (O(c log c), no extra memory) beyond, so a batch
// that sends every arrival to one target stays bounded.  The keys are distinct
// (the index), so both give the same order.
constexpr uint32_t kFoldInsertionMax = 32;

__device__ __forceinline__ void fold_sort(FoldRec *r, uint32_t c) {
    if (c <= kFoldInsertionMax) {
        for (uint32_t a = 1; a < c; ++a) {
            FoldRec v = r[a];
            int b = (int)a - 1;
            while (b >= 0 && fold_less(v, r[b])) { r[b + 1] = r[b]; --b; }
            r[b + 1] = v;
        }
        return;
    }
    for (uint32_t j = c / 2; j-- > 0;) sift_down(r, j, c);
    for (uint32_t e = c - 1; e > 0; --e) {
        const FoldRec top = r[0];
        r[0] = r[e];
        r[e] = top;
        sift_down(r, 0, e);
    }
}

// The same by a warp, in place: a bitonic sort whose every comparison moves the smaller
// record down (the first of each merge compares mirrored places), so that the places
// beyond c may be left out.
__device__ __forceinline__ void fold_sort_warp(FoldRec *r, uint64_t c, int lane) {
    auto order = [&](uint64_t i, uint64_t j) {
        const FoldRec x = r[i], y = r[j];
        if (fold_less(y, x)) { r[i] = y; r[j] = x; }
    };
    for (uint64_t k = 2; k < 2 * c; k <<= 1) {
        for (uint64_t p = lane;; p += 32) {
            const uint64_t lo = p / (k / 2) * k, o = p % (k / 2);
            if (lo + k / 2 >= c) break;  // no pair of this merge or a later one
            if (lo + k - 1 - o < c) order(lo + o, lo + k - 1 - o);
        }
        __syncwarp();
        for (uint64_t s = k / 4; s > 0; s >>= 1) {
            for (uint64_t p = lane;; p += 32) {
                const uint64_t i = p / s * 2 * s + p % s;
                if (i + s >= c) break;
                order(i, i + s);
            }
            __syncwarp();
        }
    }
}

// One thread per target: walk its list, keep the arrivals sorted by (time, index), then
// add the weights in that order.  Bound by the walk's dependent loads (0.7 us an arrival),
// so everything an arrival needs is loaded as it is met.  More than kFoldLocal arrivals are
// gathered into `rec` (a run of it taken with `used`, which starts one below zero) and
// sorted there: by the thread, or beyond kFoldThread by the whole warp, one such list after
// the other, unless the warp has more than kFoldLong of them to sort at once.  100,000
// arrivals at 30,000 targets: 29 us; with 1,000 of them at each of four targets 0.44 ms
// (thread's sort of counted and scattered records 1.6, of a list walked three times 4.1);
// 10,000 at 8 targets 0.52 ms (6.3, 7.0).
constexpr uint32_t kFoldLocal = 16, kFoldThread = 96;
constexpr int kFoldLong = 12;

__global__ void __launch_bounds__(128) k_fold_apply(int64_t m, const FoldList *__restrict__ list, const uint32_t *__restrict__ next, const double *__restrict__ time,
                                                    const int8_t *__restrict__ type, const float *__restrict__ weight,
                                                    uint32_t *used, FoldRec *rec, float *g_exc, float *g_inh, float *g_nmda,
                                                    int per_warp) {
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t t = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per_warp + lane;
    const FoldList own = lane < per_warp && t < m ? list[t] : FoldList{kNone, kNone};
    const uint32_t c = own.last == kNone ? 0u : own.more + 2u;
    if (!__any_sync(full, c != 0)) return;
    float ge = 0.0f, gi = 0.0f, gn = 0.0f;
    if (c) {
        ge = g_exc ? g_exc[t] : 0.0f;
        gi = g_inh ? g_inh[t] : 0.0f;
        gn = g_nmda ? g_nmda[t] : 0.0f;
    }
    auto add = [&](int ty, float w) {
        if (ty == 0) ge += w;
        else if (ty == 1) gi += w;
        else gn += w;
    };
    FoldRec *r = nullptr;
    if (c > kFoldLocal) {
        r = rec + (atomicAdd(used, c) + 1u);
        uint32_t a = 0;
        for (uint32_t q = own.last; q != kNone; q = next[q]) r[a++] = FoldRec{time ? time[q] : 0.0, q, 0};
    } else if (c) {
        FoldRec key[kFoldLocal];
        float w[kFoldLocal];
        int8_t ty[kFoldLocal];
        uint32_t q = own.last;
        for (uint32_t a = 0; a < c; ++a) {
            const FoldRec v{time ? time[q] : 0.0, q, 0};
            const float vw = weight[q];
            const int8_t vt = type[q];
            q = next[q];
            int b = (int)a - 1;
            while (b >= 0 && fold_less(v, key[b])) {
                key[b + 1] = key[b];
                w[b + 1] = w[b];
                ty[b + 1] = ty[b];
                --b;
            }
            key[b + 1] = v;
            w[b + 1] = vw;
            ty[b + 1] = vt;
        }
        for (uint32_t a = 0; a < c; ++a) add(ty[a], w[a]);
    }
    unsigned longer = __ballot_sync(full, c > kFoldThread);
    if (__popc(longer) > kFoldLong) longer = 0;
    if (c > kFoldLocal && !(longer >> lane & 1)) {
        fold_sort(r, c);
        for (uint32_t a = 0; a < c; ++a) add(type[r[a].i], weight[r[a].i]);
    }
    for (; longer; longer &= longer - 1u) {
        const int l = __ffs(longer) - 1;
        FoldRec *rl = (FoldRec *)__shfl_sync(full, (unsigned long long)r, l);
        const uint32_t cl = __shfl_sync(full, c, l);
        __syncwarp();  // the owner's records are written
        fold_sort_warp(rl, cl, lane);
        for (uint32_t a0 = 0; a0 < cl; a0 += 32) {  // 32 loaded at once, added by the owner in order
            const uint32_t k = min(32u, cl - a0);
            int vt = 0;
            float vw = 0.0f;
            if (lane < k) {
                const uint32_t i = rl[a0 + lane].i;
                vt = type[i];
                vw = weight[i];
            }
            for (uint32_t u = 0; u < k; ++u) {
                const int tu = __shfl_sync(full, vt, u);
                const float wu = __shfl_sync(full, vw, u);
                if (lane == l) add(tu, wu);
            }
        }
    }
    if (c) {
        if (g_exc) g_exc[t] = ge;
        if (g_inh) g_inh[t] = gi;
        if (g_nmda) g_nmda[t] = gn;
    }
}

// Scratch layout shared by the entry points: lists (m), the count of records taken, links
// (n), then the records (16-byte aligned).
constexpr size_t fold_words(int64_t n, int64_t m) { return 2 * (size_t)m + 1 + (size_t)n; }

constexpr size_t fold_scratch_bytes(int64_t n, int64_t m) {
    return ((fold_words(n, m) * sizeof(uint32_t) + 255) & ~(size_t)255) + (size_t)n * sizeof(FoldRec);
}

// Three launches (clear, link, fold); counting, scanning and scattering the arrivals
// instead took eight (100,000 arrivals at 30,000 targets: 97 us a call among others, 29).
int fold_enqueue(cudaStream_t st, void *scratch, int64_t n, const int32_t *target, const int8_t *type,
                 const float *weight, const double *time, int64_t m, float *g_exc, float *g_inh, float *g_nmda) {
    if (n == 0) return EB_OK;
    FoldList *list = (FoldList *)scratch;
    uint32_t *used = (uint32_t *)(list + m), *next = used + 1;
    FoldRec *rec = (FoldRec *)((char *)scratch + ((fold_words(n, m) * sizeof(uint32_t) + 255) & ~(size_t)255));
    cudaError_t e = cudaMemsetAsync(list, 0xff, sizeof(uint32_t) * (size_t)(2 * m + 1), st);  // no arrivals, no records
    if (e != cudaSuccess) { set_error("cudaMemsetAsync: %s", cudaGetErrorString(e)); return EB_ERR_CUDA; }
    k_fold_link<<<(int)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, st>>>(n, target, list, next);
    // few targets take a warp each, or a few a warp, until every SM sub-partition has one; not
    // with hardly an arrival each (1,000 at 1,000 targets: 18.5 us a call spread, 17.8)
    const int per_warp = n < 4 * m ? 32 : (int)std::min<int64_t>(32, (m + 148 * 4 - 1) / (148 * 4));
    k_fold_apply<<<(int)((m + 4 * per_warp - 1) / (4 * per_warp)), 128, 0, st>>>(m, list, next, time, type, weight, used, rec, g_exc, g_inh,
                                                                                g_nmda, per_warp);
    e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("fold kernels: %s", cudaGetErrorString(e)); return EB_ERR_CUDA; }
    return EB_OK;
}

constexpr int64_t kMaxTargets = 1 << 20;

int fold_check(int64_t n, const int32_t *target, const int8_t *type, const float *weight, int64_t m) {
    if (n < 0 || m <= 0 || (n > 0 && (!target || !type || !weight))) { set_error("bad fold arguments"); return EB_ERR_ARG; }
    if (m > kMaxTargets) { set_error("fold: more than %lld targets", (long long)kMaxTargets); return EB_ERR_ARG; }
    if (n >= (int64_t)UINT32_MAX) { set_error("fold: too many arrivals"); return EB_ERR_ARG; }
    return EB_OK;
}

}  // namespace

namespace {

constexpr int kMaxDevices = 64;

// Id of the calling thread's current context, never that of an earlier one; 0 where the
// driver does not tell.  What is kept per device below belongs to a context: it dies with
// it in cudaDeviceReset, and its handle or address must not be used after that.
unsigned long long context_id() {
    using Fn = int (*)(void *, unsigned long long *);  // cuCtxGetId: (CUcontext, id), 0 on success
    static const Fn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? (Fn)p : nullptr;
    }();
    unsigned long long id = 0;
    return fn && fn(nullptr, &id) == 0 ? id : 0;
}

// The op's own memory pool on the current device, null where the device's current pool
// serves instead.  Each call takes its scratch from it on the caller's stream and gives it
// back there, so calls on different streams and threads never share a block, and the pool
// keeps up to kPoolKept bytes of returned blocks when the device synchronises: the default
// pool keeps none unless the process set it so, and every call after a synchronisation
// mapped its scratch anew (100,000 arrivals, waited for: 480-530 us, 48 with this pool).
// Above kPoolKept everything goes back.  A pool that the process set with
// cudaDeviceSetMemPool is used as before, and so is the default one in any context but
// the first that called on the device (after a reset of it, say).
constexpr uint64_t kPoolKept = 32ull << 20;

cudaMemPool_t fold_pool() {
    struct Own {
        cudaMemPool_t pool, standard;  // its own, and the device's default one
        unsigned long long ctx;        // that of the first call, 0 before
    };
    static std::mutex mu;
    static Own own[kMaxDevices] = {};
    int dev = 0;
    cudaMemPool_t now = nullptr;
    const unsigned long long ctx = context_id();
    if (!ctx || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices ||
        cudaDeviceGetMemPool(&now, dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mu);
    Own &o = own[dev];
    if (!o.ctx) {
        cudaMemPool_t standard = nullptr;
        if (cudaDeviceGetDefaultMemPool(&standard, dev) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        if (now != standard) return nullptr;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        uint64_t kept = kPoolKept;
        cudaMemPool_t p = nullptr;
        cudaError_t e = cudaMemPoolCreate(&p, &props);
        if (e == cudaSuccess && (e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &kept)) != cudaSuccess)
            cudaMemPoolDestroy(p);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        o = Own{p, standard, ctx};
    }
    return o.ctx == ctx && now == o.standard ? o.pool : nullptr;
}

}  // namespace

extern "C" int eb_fold_arrivals(void *stream, int64_t n, const int32_t *target, const int8_t *type,
                                const float *weight, const double *time, int64_t n_targets, float *g_exc,
                                float *g_inh, float *g_nmda) {
    int rc = fold_check(n, target, type, weight, n_targets);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    void *scratch = nullptr;
    const size_t bytes = fold_scratch_bytes(n, n_targets);
    if (n == 0) return EB_OK;
    // under stream capture the scratch is a node of the graph, which owns it
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &capture);
    if (e == cudaSuccess) {
        const cudaMemPool_t pool = capture == cudaStreamCaptureStatusNone ? fold_pool() : nullptr;
        e = pool ? cudaMallocFromPoolAsync(&scratch, bytes, pool, st) : cudaMallocAsync(&scratch, bytes, st);
    }
    if (e != cudaSuccess) { set_error("fold scratch (%zu bytes): %s", bytes, cudaGetErrorString(e)); return EB_ERR_NOMEM; }
    rc = fold_enqueue(st, scratch, n, target, type, weight, time, n_targets, g_exc, g_inh, g_nmda);
    cudaFreeAsync(scratch, st);
    return rc;
}

// ------------------------------------------------------ allocation-free form --
// Some callers cannot allocate device memory while they run: a closed-loop
// (real-time) controller whose step deadline must not contain allocator calls,
// or a host engine that claims all device memory for itself at start-up.  This
// form of the op takes its scratch from a fixed array in the library's device
// image instead.  Every GPU that loads the library holds that array (about
// 7 MiB) until the process exits; it bounds one call to kNoAllocMaxArrivals
// arrivals and kNoAllocMaxTargets targets.  All calls share the one array and
// it keeps the previous call's contents: the counters that must start clear
// are cleared at the start of every call, and two calls whose work overlaps on
// the GPU (different streams, or different host threads on the same device)
// race on it.
namespace {

constexpr int64_t kNoAllocMaxArrivals = 1 << 18;
constexpr int64_t kNoAllocMaxTargets = 1 << 18;
constexpr size_t kNoAllocScratchBytes = fold_scratch_bytes(kNoAllocMaxArrivals, kNoAllocMaxTargets);

static __device__ __align__(256) unsigned char g_fold_scratch[kNoAllocScratchBytes];

// The array's device address on each device, looked up once per device and
// context (with that device current); in host code g_fold_scratch only names a
// host-side stand-in, never the device memory.
std::mutex g_scratch_mu;
void *g_scratch_ptr[kMaxDevices] = {};
unsigned long long g_scratch_ctx[kMaxDevices] = {};

int scratch_for_current_device(void **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) { set_error("cudaGetDevice: %s", cudaGetErrorString(e)); return EB_ERR_CUDA; }
    if (dev < 0 || dev >= kMaxDevices) { set_error("device index %d above %d", dev, kMaxDevices - 1); return EB_ERR_ARG; }
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_ptr[dev] || !ctx || g_scratch_ctx[dev] != ctx) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_fold_scratch);
        if (e != cudaSuccess || !p) {
            set_error("cudaGetSymbolAddress(scratch) on device %d: %s", dev, cudaGetErrorString(e));
            return EB_ERR_CUDA;
        }
        g_scratch_ptr[dev] = p;
        g_scratch_ctx[dev] = context_id();
    }
    *out = g_scratch_ptr[dev];
    return EB_OK;
}

}  // namespace

extern "C" int eb_fold_arrivals_noalloc(void *stream, int64_t n, const int32_t *target, const int8_t *type,
                                        const float *weight, const double *time, int64_t n_targets,
                                        float *g_exc, float *g_inh, float *g_nmda) {
    int rc = fold_check(n, target, type, weight, n_targets);
    if (rc) return rc;
    if (n > kNoAllocMaxArrivals || n_targets > kNoAllocMaxTargets) {
        set_error("eb_fold_arrivals_noalloc: %lld arrivals / %lld targets exceed its fixed scratch "
                  "(at most %lld arrivals and %lld targets per call); use eb_fold_arrivals",
                  (long long)n, (long long)n_targets, (long long)kNoAllocMaxArrivals, (long long)kNoAllocMaxTargets);
        return EB_ERR_ARG;
    }
    void *scratch = nullptr;
    if ((rc = scratch_for_current_device(&scratch))) return rc;
    return fold_enqueue((cudaStream_t)stream, scratch, n, target, type, weight, time, n_targets, g_exc, g_inh,
                        g_nmda);
}
