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

// Arrivals of one target as a linked list: head[t] is its last linked arrival, next[i]
// the one linked before arrival i (kNone: none).  The order of the links is whatever the
// atomics give; the fold sorts.
constexpr uint32_t kNone = 0xffffffffu;

__global__ void __launch_bounds__(256) k_fold_link(int64_t n, const int32_t *__restrict__ target, uint32_t *head,
                                                   uint32_t *__restrict__ next) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        next[i] = atomicExch(head + target[i], (uint32_t)i);
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

// One thread per target: walk its list, keep the arrivals sorted by (time, index), then
// add the weights in that order.  Bound by the walk's dependent loads, so everything an
// arrival needs is loaded as it is met.  More than kFoldLocal arrivals are gathered into
// `rec` (a run of it taken with `used`, which starts one below zero) and sorted there.
constexpr uint32_t kFoldLocal = 16;

__global__ void __launch_bounds__(128) k_fold_apply(int64_t m, const uint32_t *__restrict__ head, const uint32_t *__restrict__ next,
                                                    const double *__restrict__ time, const int8_t *__restrict__ type,
                                                    const float *__restrict__ weight, uint32_t *used, FoldRec *rec,
                                                    float *g_exc, float *g_inh, float *g_nmda) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m) return;
    const uint32_t i = head[t];
    if (i == kNone) return;
    float ge = g_exc ? g_exc[t] : 0.0f, gi = g_inh ? g_inh[t] : 0.0f, gn = g_nmda ? g_nmda[t] : 0.0f;
    auto add = [&](int ty, float w) {
        if (ty == 0) ge += w;
        else if (ty == 1) gi += w;
        else gn += w;
    };
    FoldRec key[kFoldLocal];
    float w[kFoldLocal];
    int8_t ty[kFoldLocal];
    uint32_t c = 0;
    uint32_t rest = i;
    for (; rest != kNone && c < kFoldLocal; ++c) {
        const FoldRec v{time ? time[rest] : 0.0, rest, 0};
        const float vw = weight[rest];
        const int8_t vt = type[rest];
        rest = next[rest];
        int b = (int)c - 1;
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
    if (rest == kNone) {
        for (uint32_t a = 0; a < c; ++a) add(ty[a], w[a]);
    } else {
        for (uint32_t q = rest; q != kNone; q = next[q]) ++c;
        FoldRec *r = rec + (atomicAdd(used, c) + 1u);
        uint32_t a = 0;
        for (uint32_t q = i; q != kNone; q = next[q]) r[a++] = FoldRec{time ? time[q] : 0.0, q, 0};
        fold_sort(r, c);
        for (a = 0; a < c; ++a) add(type[r[a].i], weight[r[a].i]);
    }
    if (g_exc) g_exc[t] = ge;
    if (g_inh) g_inh[t] = gi;
    if (g_nmda) g_nmda[t] = gn;
}

// Scratch layout shared by the entry points: heads (m) and the count of records taken,
// links (n), then the records (16-byte aligned).
size_t fold_words(int64_t n, int64_t m) { return (size_t)(m + 1) + (size_t)n; }

size_t fold_scratch_bytes(int64_t n, int64_t m) {
    return ((fold_words(n, m) * sizeof(uint32_t) + 255) & ~(size_t)255) + (size_t)n * sizeof(FoldRec);
}

// Three launches (clear, link, fold); counting, scanning and scattering the arrivals
// instead took eight.  100,000 arrivals at 30,000 targets: 34 us a
// call among others with the copies of three conductance arrays, 57 before.
int fold_enqueue(cudaStream_t st, void *scratch, int64_t n, const int32_t *target, const int8_t *type,
                 const float *weight, const double *time, int64_t m, float *g_exc, float *g_inh, float *g_nmda) {
    if (n == 0) return EB_OK;
    uint32_t *head = (uint32_t *)scratch, *used = head + m, *next = head + m + 1;
    FoldRec *rec = (FoldRec *)((char *)scratch + ((fold_words(n, m) * sizeof(uint32_t) + 255) & ~(size_t)255));
    cudaError_t e = cudaMemsetAsync(head, 0xff, sizeof(uint32_t) * (size_t)(m + 1), st);  // no arrivals, no records
    if (e != cudaSuccess) { set_error("cudaMemsetAsync: %s", cudaGetErrorString(e)); return EB_ERR_CUDA; }
    k_fold_link<<<(int)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, st>>>(n, target, head, next);
    k_fold_apply<<<(int)((m + 127) / 128), 128, 0, st>>>(m, head, next, time, type, weight, used, rec, g_exc, g_inh, g_nmda);
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
        cudaMemPool_t pool;
        unsigned long long ctx;  // that of the first call, 0 before
    };
    static std::mutex mu;
    static Own own[kMaxDevices] = {};
    int dev = 0;
    cudaMemPool_t now = nullptr, standard = nullptr;
    const unsigned long long ctx = context_id();
    if (!ctx || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices ||
        cudaDeviceGetMemPool(&now, dev) != cudaSuccess || cudaDeviceGetDefaultMemPool(&standard, dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (now != standard) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    Own &o = own[dev];
    if (!o.ctx) {
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
        o = Own{p, ctx};
    }
    return o.ctx == ctx ? o.pool : nullptr;
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
// 6 MiB) until the process exits; it bounds one call to kNoAllocMaxArrivals
// arrivals and kNoAllocMaxTargets targets.  All calls share the one array and
// it keeps the previous call's contents: the counters that must start clear
// are cleared at the start of every call, and two calls whose work overlaps on
// the GPU (different streams, or different host threads on the same device)
// race on it.
namespace {

constexpr int64_t kNoAllocMaxArrivals = 1 << 18;
constexpr int64_t kNoAllocMaxTargets = 1 << 18;
constexpr size_t kNoAllocScratchBytes =
    (((size_t)(kNoAllocMaxTargets + 1 + kNoAllocMaxArrivals) * sizeof(uint32_t) + 255) & ~(size_t)255) +
    (size_t)kNoAllocMaxArrivals * sizeof(FoldRec);

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
