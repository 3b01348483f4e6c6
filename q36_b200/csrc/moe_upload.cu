// GGUF MXFP4 blocks in (pageable) host memory -> split planes on the device: the MXFP4 branch of upload()
// (q36_engine.cu:202-228).
//
// The device does the re-arrangement.  The blocks go into pinned staging as they are (host threads, each with two slots of
// its own) and k_repack reads a slot over PCIe, 16 bytes per thread, and writes codes and scales where they belong: no
// second host copy, no device staging, and the threads' copies overlap the transfer.  What bounds it is then the PCIe
// link and the host's copy into pinned memory.  A layer of 64 + 1 experts (109 MB, six uploads) takes
// 3.7 to 4.3 ms; 47.6 when one host thread took the blocks apart and a pageable copy followed; 45 when every upload pinned its own
// staging, as the first one of a process does (3 to 21 ms, once).
#include <cuda.h>
#include <string.h>

#include <atomic>
#include <mutex>
#include <utility>

#include "common.cuh"
#include "host_threads.h"
#include "kernels.cuh"

namespace q36 {

constexpr int RP_BLOCKS = 256;                          // 17-byte blocks per CTA (272 x 16 B)
constexpr int UP_SLOT_BLOCKS = 32768;                   // blocks per staging slot (544 KB)
constexpr uint64_t UP_SLOT_BYTES = (uint64_t)UP_SLOT_BLOCKS * 17;
constexpr int UP_MAX_THREADS = 8;
// Smaller tensors are re-arranged on the host: a launch, its wait and the first byte's copy cost more than one thread takes for
// them, and nothing has to be pinned.  us on the host / on the device, sources in memory, on three machines: 17 KB 39 to 43 / 54 to
// 69, 136 KB 59 to 63 / 59 to 84, 272 KB 80 to 107 / 73 to 105, 544 KB 128 to 145 / 105 to 141, 1088 KB 234 to 260 / 168 to 201.
constexpr int UP_MIN_BLOCKS = 16384;
static_assert(RP_BLOCKS * 17 % 16 == 0 && UP_SLOT_BYTES % 16 == 0, "16-byte loads of whole slots");

// src: n consecutive blocks (16-byte aligned, readable up to the next multiple of 16 bytes), the first of them block
// `first` of the tensor; plane: blocks per expert.  dst and the experts' stride (plane * 17) are multiples of 16 bytes.
__global__ void __launch_bounds__(RP_BLOCKS)
k_repack(const uint4 *__restrict__ src, uint64_t first, int n, uint64_t plane, uint8_t *__restrict__ dst) {
    Q36_GDS();
    __shared__ uint4 s4[RP_BLOCKS * 17 / 16 + 1];       // (+ 1: the last block's shifted reads touch one word more)
    const int b0 = blockIdx.x * RP_BLOCKS, nb = min(RP_BLOCKS, n - b0);
    const int words = (nb * 17 + 15) / 16;
    for (int i = threadIdx.x; i < words; i += RP_BLOCKS) s4[i] = src[(size_t)blockIdx.x * (RP_BLOCKS * 17 / 16) + i];
    __syncthreads();
    if ((int)threadIdx.x >= nb) return;
    const uint64_t i = first + b0 + threadIdx.x, e = i / plane, r = i - e * plane;
    uint8_t *codes = dst + e * plane * 17;
    const uint32_t o = threadIdx.x * 17 + 1, sh = (o & 3) * 8;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(s4) + (o >> 2);
    const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
    *reinterpret_cast<uint4 *>(codes + r * 16) = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh),
                                                            __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
    codes[plane * 16 + r] = reinterpret_cast<const uint8_t *>(s4)[threadIdx.x * 17];
}

// A slot's transfer takes 10 us and a kernel's start and end 6 more, so kernels have to overlap.  Every thread has a stream of
// its own for that: "the slot's kernel is over" is then one event, whatever the others do.  One stream with overlapping kernels
// would need each of them to wait for the one before it before it ends, else the end of one says nothing about the ones before:
// that chain leaves two kernels in flight.  Loads of 64 + 1 experts with 8 streams 3.8 ms, 4 streams 4.4, 2 streams 4.7; one
// stream 5.8 (kernels in turn) or 5.3 (overlapping, with the wait).
//
// Pinned staging.  Pinning costs more than the transfer (4 to 10 ms for the 8.5 MB of one upload, which takes 1.5), so one
// staging area of at most that size stays with the process between uploads; q36_moe_upload_release gives it back.  An upload
// that finds it in use by another thread pins and frees its own.
namespace {
struct Staging { uint8_t *p; uint64_t bytes; };
std::mutex g_staging_mutex;                             // (also of g_lanes)
Staging g_staging = {nullptr, 0};

Staging staging_swap(Staging s, bool only_larger) {
    std::lock_guard<std::mutex> lock(g_staging_mutex);
    if (!only_larger || s.bytes > g_staging.bytes) std::swap(s, g_staging);
    return s;
}
// (a device reset takes pinned memory away with the context)
bool staging_alive(const Staging &s) {
    cudaPointerAttributes at;
    const bool alive = s.p && cudaPointerGetAttributes(&at, s.p) == cudaSuccess && at.type == cudaMemoryTypeHost;
    (void)cudaGetLastError();
    return alive;
}
Staging staging_take(uint64_t bytes) {
    Staging s = staging_swap(Staging{nullptr, 0}, false);
    if (staging_alive(s)) {
        if (s.bytes >= bytes) return s;
        cudaFreeHost(s.p);
    }
    s = Staging{nullptr, bytes};
    if (cudaHostAlloc((void **)&s.p, bytes, cudaHostAllocPortable) != cudaSuccess) s = Staging{nullptr, 0};
    (void)cudaGetLastError();
    return s;
}
cudaError_t staging_put(Staging s) {
    s = staging_swap(s, true);                          // keep the larger one
    return s.p ? cudaFreeHost(s.p) : cudaSuccess;
}

// The threads' streams stay as well: making one and destroying it costs 120 us, as much as a small upload.  One set per device,
// of the context it was made in; an upload that finds it in use makes and destroys its own.
struct Lanes { unsigned long long ctx; cudaStream_t st[UP_MAX_THREADS]; };
Lanes g_lanes[MAX_DEVICES] = {};

void *driver_fn(const char *name) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? p : nullptr;
}
// The calling thread's context and its id (no two contexts of a process have the same one); id 0 if it cannot be had.  A program
// may work in a context of its own instead of the runtime's: its memory is not there for a kernel launched in another one.
struct Context { CUcontext c; unsigned long long id; };
Context current_context() {
    static const auto get = (CUresult (*)(CUcontext *))driver_fn("cuCtxGetCurrent");
    static const auto get_id = (CUresult (*)(CUcontext, unsigned long long *))driver_fn("cuCtxGetId");
    Context x = {nullptr, 0};
    if (!get || !get_id || get(&x.c) != CUDA_SUCCESS || !x.c || get_id(x.c, &x.id) != CUDA_SUCCESS) x.id = 0;
    return x;
}
cudaError_t enter_context(CUcontext c) {
    static const auto set = (CUresult (*)(CUcontext))driver_fn("cuCtxSetCurrent");
    return set && set(c) == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidDevice;
}
// Is it another context's memory?  (Memory of a pool belongs to none: the context is null then, or the query is refused.)
bool elsewhere(const void *p, CUcontext c) {
    static const auto get = (CUresult (*)(void *, CUpointer_attribute, CUdeviceptr))driver_fn("cuPointerGetAttribute");
    CUcontext owner = nullptr;
    return get && get(&owner, CU_POINTER_ATTRIBUTE_CONTEXT, (CUdeviceptr)(uintptr_t)p) == CUDA_SUCCESS && owner && owner != c;
}
Lanes lanes_take(int dev, unsigned long long ctx) {
    Lanes l = {};
    {
        std::lock_guard<std::mutex> lock(g_staging_mutex);
        std::swap(l, g_lanes[dev]);
    }
    if (l.ctx != ctx) l = Lanes{ctx, {}};               // (another context's streams went, or go, with it)
    return l;
}
cudaError_t lanes_put(int dev, Lanes l, bool keep) {
    if (keep) {
        std::lock_guard<std::mutex> lock(g_staging_mutex);
        if (!g_lanes[dev].ctx) std::swap(l, g_lanes[dev]);
    }
    cudaError_t e = cudaSuccess;
    for (cudaStream_t st : l.st)
        if (st) { const cudaError_t d = cudaStreamDestroy(st); if (e == cudaSuccess) e = d; }
    return e;
}
}  // namespace

int upload_release() {
    cudaError_t el = cudaSuccess;
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess) (void)cudaGetLastError();
    for (int dev = 0; dev < MAX_DEVICES; dev++) {
        bool any;
        {
            std::lock_guard<std::mutex> lock(g_staging_mutex);
            any = g_lanes[dev].ctx != 0;
        }
        if (!any || (dev != cur && cudaSetDevice(dev) != cudaSuccess)) continue;
        const cudaError_t e = lanes_put(dev, lanes_take(dev, current_context().id), false);
        if (el == cudaSuccess) el = e;
        if (dev != cur && cur >= 0) (void)cudaSetDevice(cur);
    }
    const Staging s = staging_swap(Staging{nullptr, 0}, false);
    cudaError_t e = staging_alive(s) ? cudaFreeHost(s.p) : cudaSuccess;
    if (e == cudaSuccess) e = el;
    if (e != cudaSuccess) { last_cuda_error() = (int)e; return Q36_MOE_ECUDA; }
    return Q36_MOE_OK;
}

// Returns UPLOAD_NOT_TAKEN when this route does not apply (see the rule) or pinned memory cannot be had; the caller then
// re-arranges on the host.  Synchronous, ordered like a cudaMemcpy: the first byte's copy waits for
// what the legacy default stream would wait for, and the threads' streams wait for that stream.
int upload_repacked(const void *host_blocks, uint64_t plane, uint64_t e0, uint64_t n_expert, void *dev_dst) {
    // 16-byte stores need an aligned destination and a stride that keeps every expert aligned; the kernel runs on the
    // current device, so the destination has to be that device's own memory (cudaMemcpy takes any device's)
    int dev;
    cudaPointerAttributes at;
    if (n_expert * plane < UP_MIN_BLOCKS || (uintptr_t)dev_dst % 16 || plane % 16 || (dev = current_device()) < 0) return UPLOAD_NOT_TAKEN;
    if (cudaPointerGetAttributes(&at, dev_dst) != cudaSuccess || at.type != cudaMemoryTypeDevice || at.device != dev) {
        (void)cudaGetLastError();
        return UPLOAD_NOT_TAKEN;
    }
    const Context ctx = current_context();      // (the call above has made one if there was none)
    if (!ctx.id || elsewhere(dev_dst, ctx.c)) return UPLOAD_NOT_TAKEN;
    const uint8_t *src = (const uint8_t *)host_blocks + e0 * plane * 17;
    // The first byte goes by a plain copy: it waits for the work before it and is refused (a stream capture under way, say)
    // just like the one copy of the whole tensor that the host route makes.
    if (const cudaError_t e = cudaMemcpy(dev_dst, src + 1, 1, cudaMemcpyHostToDevice)) { last_cuda_error() = (int)e; return Q36_MOE_ECUDA; }
    const uint64_t n = n_expert * plane, chunks = (n + UP_SLOT_BLOCKS - 1) / UP_SLOT_BLOCKS;
    const unsigned hw = std::thread::hardware_concurrency();
    const int threads = (int)min(min((uint64_t)UP_MAX_THREADS, (uint64_t)(hw > 1 ? hw : 1)), (chunks + 1) / 2);
    const Staging staging = staging_take((chunks > 1 ? (uint64_t)threads * 2 : 1) * UP_SLOT_BYTES);
    if (!staging.p) return UPLOAD_NOT_TAKEN;
    Lanes lanes = lanes_take(dev, ctx.id);
    std::atomic<uint64_t> next{0};
    std::atomic<int> err{0};
    auto work = [&](int w) {
        cudaError_t e = w ? enter_context(ctx.c) : cudaSuccess;
        cudaEvent_t ev[2] = {nullptr, nullptr};
        cudaStream_t &st = lanes.st[w];
        if (e == cudaSuccess && !st) e = cudaStreamCreate(&st);      // (a blocking stream: it waits for the first byte's copy)
        for (int s = 0; s < 2 && e == cudaSuccess; s++) e = cudaEventCreateWithFlags(&ev[s], cudaEventDisableTiming);
        for (int s = 0, used = 0; e == cudaSuccess && !err.load(std::memory_order_relaxed); s ^= 1, used++) {
            const uint64_t c = next.fetch_add(1);
            if (c >= chunks) break;
            if (used >= 2 && (e = cudaEventSynchronize(ev[s])) != cudaSuccess) break;   // the slot's last transfer
            const uint64_t b0 = c * UP_SLOT_BLOCKS;
            const int nb = (int)min((uint64_t)UP_SLOT_BLOCKS, n - b0);
            uint8_t *slot = staging.p + (uint64_t)(2 * w + s) * UP_SLOT_BYTES;
            memcpy(slot, src + b0 * 17, (size_t)nb * 17);
            k_repack<<<(nb + RP_BLOCKS - 1) / RP_BLOCKS, RP_BLOCKS, 0, st>>>((const uint4 *)slot, b0, nb, plane, (uint8_t *)dev_dst);
            if ((e = cudaGetLastError()) == cudaSuccess) e = cudaEventRecord(ev[s], st);
        }
        if (st) {                                       // (also before the staging is used again)
            const cudaError_t es = cudaStreamSynchronize(st);
            if (e == cudaSuccess) e = es;
        }
        if (e != cudaSuccess) err = (int)e;
        for (int s = 0; s < 2; s++) if (ev[s]) cudaEventDestroy(ev[s]);
    };
    run_on_threads<UP_MAX_THREADS>(threads, work);
    cudaError_t e = (cudaError_t)err.load();
    const cudaError_t el = lanes_put(dev, lanes, true), ep = staging_put(staging);
    if (e == cudaSuccess) e = el;
    if (e == cudaSuccess) e = ep;
    if (e != cudaSuccess) { last_cuda_error() = (int)e; return Q36_MOE_ECUDA; }
    return Q36_MOE_OK;
}

}  // namespace q36
