// Devices, memory, streams, events and graph replay for libscrapgpu_sm100 (the part of the backend
// vtable that is not arithmetic: include/scrapgpu/backend.h:33-44 of the reference).
#include "sm100_common.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

namespace sm100 {

static thread_local std::string t_error;
static std::atomic<uint64_t> g_launches{0};
static std::atomic<int> g_pdl{1};

int fail(int status, const char * fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    t_error = buf;
    return status;
}

int cuda_fail(cudaError_t e, const char * what) {
    const int st = e == cudaErrorMemoryAllocation ? ST_OOM : ST_BACKEND;
    return fail(st, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
}

static thread_local int t_serialized = 0;

static thread_local int t_serialized_inner = 0;   // the library's own bracket, independent of the caller's
void thread_serialized(bool on) { t_serialized_inner = on ? 1 : 0; }

// kind of the last launch per stream (stream handle + 8 with the kind in the low bits; the legacy stream 0 can so be
// told from an empty slot); a handful of slots serves the few streams a process drives at a time, a lost entry only
// costs speed
static std::atomic<uintptr_t> g_tail[8];
void stream_tail_set(cudaStream_t stream, int kind) {
    const uintptr_t key = ((uintptr_t) stream + 8) & ~(uintptr_t) 7;
    for (auto & slot : g_tail) {
        if ((slot.load(std::memory_order_relaxed) & ~(uintptr_t) 7) != key) continue;
        slot.store(kind == TAIL_OTHER ? 0 : key | (uintptr_t) kind, std::memory_order_relaxed);
        return;
    }
    if (kind == TAIL_OTHER) return;
    for (auto & slot : g_tail) {
        uintptr_t empty = 0;
        if (slot.compare_exchange_strong(empty, key | (uintptr_t) kind, std::memory_order_relaxed)) return;
    }
    g_tail[(key >> 6) % 8].store(key | (uintptr_t) kind, std::memory_order_relaxed);
}
int stream_tail(cudaStream_t stream) {
    const uintptr_t key = ((uintptr_t) stream + 8) & ~(uintptr_t) 7;
    for (auto & slot : g_tail) {
        const uintptr_t v = slot.load(std::memory_order_relaxed);
        if ((v & ~(uintptr_t) 7) == key) return (int) (v & 7);
    }
    return TAIL_OTHER;
}
bool pdl_enabled() { return t_serialized == 0 && t_serialized_inner == 0 && g_pdl.load(std::memory_order_relaxed) != 0; }
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { (void) cudaGetLastError(); return 0; }
    return dev < 0 || dev >= MAX_DEVICES ? 0 : dev;
}

int sm_count() {
    static std::mutex mu;
    static std::vector<int> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    std::lock_guard<std::mutex> lock(mu);
    if ((int) cache.size() <= dev) cache.resize(dev + 1, 0);
    if (cache[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cache[dev] = n;
    }
    return cache[dev];
}

// Per-device scratch owned by the library, one buffer per slot (0 = attention partials, 1 = GEMM
// activations, 2 = quantized activation columns of the multi-column matvec), grown on demand.  A buffer that was
// handed out once is NEVER freed or moved: a CUDA graph captured earlier has its address baked into its kernel
// nodes and may be replayed at any time.  Growing therefore allocates a second, larger block (at least twice the
// old size, so the blocks left behind add up to less than the live one) and later calls use that; replays of older
// graphs keep working on the block they were captured with.  Calls that use the same slot must be ordered on one
// stream.  Allocation cannot happen while a stream is capturing: the first call of a shape (or sm100_scratch_reserve)
// has to come before the capture.
int device_scratch(int slot, size_t bytes, void ** out) {
    constexpr int SLOTS = 3;
    struct Entry { void * ptr[SLOTS] = {nullptr, nullptr, nullptr}; size_t size[SLOTS] = {0, 0, 0}; std::vector<void *> retired; };
    static std::mutex mu;
    static std::vector<Entry> table;
    if (slot < 0 || slot >= SLOTS) return fail(ST_INVALID, "device_scratch: bad slot");
    int dev = 0;
    SM100_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if ((int) table.size() <= dev) table.resize(dev + 1);
    Entry & e = table[dev];
    if (e.size[slot] < bytes) {
        size_t want = bytes < (size_t) (8u << 20) ? (size_t) (8u << 20) : bytes;
        if (want < 2 * e.size[slot]) want = 2 * e.size[slot];
        void * fresh = nullptr;
        const cudaError_t me = cudaMalloc(&fresh, want);
        if (me == cudaErrorStreamCaptureUnsupported || me == cudaErrorStreamCaptureInvalidated) {
            (void) cudaGetLastError();
            return fail(ST_BACKEND, "the library's scratch buffer for this op does not exist yet (or is too small) and cannot be allocated while a "
                                    "stream is capturing: issue the same call once outside the capture first");
        }
        if (me != cudaSuccess) return cuda_fail(me, "cudaMalloc(scratch)");
        SM100_CUDA(cudaMemset(fresh, 0, want));   // the attention kernels keep counters in it that start at zero
        if (e.ptr[slot] != nullptr) e.retired.push_back(e.ptr[slot]);   // stays allocated: earlier graphs may still name it
        e.ptr[slot] = fresh;
        e.size[slot] = want;
    }
    *out = e.ptr[slot];
    return ST_OK;
}

// For the duration of a scope the calling thread may allocate and create although a stream is capturing (its own, or
// another thread's in the global mode): calls that CUDA otherwise refuses, which would invalidate the capture.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    const bool set = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
    ~RelaxedCapture() {
        if (set) (void) cudaThreadExchangeStreamCaptureMode(&mode);
    }
};

// ---- memory of one call ----
// Outside a capture: from a stream-ordered pool of the library's own (per device, at most CALL_POOL_KEEP bytes stay with it
// between synchronisations), given back in stream order: concurrent streams and threads get blocks of their own.
// Inside a capture: a block that lives as long as the captured graph and everything instantiated or copied from it (a user
// object of the graph), so that the graph holds kernel nodes only.  A later call of the same capture shares the block if the
// graph orders it behind the block's last user, as it does for calls on one stream.
constexpr uint64_t CALL_POOL_KEEP = (uint64_t) 128 << 20;
struct GraphBlock {
    unsigned long long capture;   // id, never used twice
    void * ptr;
    size_t bytes;
    cudaGraphNode_t last;         // the last kernel that uses it; null while a call is being recorded
};
struct CallMemory {
    std::mutex mu;
    cudaMemPool_t pools[MAX_DEVICES] = {};
    std::vector<GraphBlock *> blocks;     // of graphs that are alive
    std::mutex dead_mu;                   // nothing of CUDA is called while it is held
    std::vector<GraphBlock *> dead;       // of graphs that are gone: their destructor may not call CUDA
    std::atomic<int> dead_count{0};
};
static CallMemory & call_memory() {
    static CallMemory * m = new CallMemory;   // graphs may be destroyed after this library's static objects
    return *m;
}
static void CUDART_CB graph_block_dead(void * p) {
    CallMemory & cm = call_memory();
    std::lock_guard<std::mutex> lock(cm.dead_mu);
    cm.dead.push_back((GraphBlock *) p);
    cm.dead_count.fetch_add(1, std::memory_order_release);
}
// frees the blocks of destroyed graphs; the caller holds cm.mu and a RelaxedCapture
static void free_dead_blocks(CallMemory & cm) {
    std::vector<GraphBlock *> gone;
    {
        std::lock_guard<std::mutex> lock(cm.dead_mu);
        gone.swap(cm.dead);
        cm.dead_count.store(0, std::memory_order_release);
    }
    for (GraphBlock * b : gone) {
        for (size_t i = 0; i < cm.blocks.size(); ++i)
            if (cm.blocks[i] == b) { cm.blocks[i] = cm.blocks.back(); cm.blocks.pop_back(); break; }
        if (cudaFree(b->ptr) != cudaSuccess) (void) cudaGetLastError();
        delete b;
    }
}
// Does the graph order `node` before a node that depends on `deps`?  Looks at 64 nodes at most: "no" only costs a block.
static bool precedes(cudaGraphNode_t node, const cudaGraphNode_t * deps, size_t count) {
    std::vector<cudaGraphNode_t> seen(deps, deps + count);
    for (size_t i = 0; i < seen.size() && i < 64; ++i) {
        if (seen[i] == node) return true;
        size_t n = 0;
        if (cudaGraphNodeGetDependencies_v2(seen[i], nullptr, nullptr, &n) != cudaSuccess) { (void) cudaGetLastError(); return false; }
        std::vector<cudaGraphNode_t> from(n);
        std::vector<cudaGraphEdgeData> edges(n);
        if (n > 0 && cudaGraphNodeGetDependencies_v2(seen[i], from.data(), edges.data(), &n) != cudaSuccess) { (void) cudaGetLastError(); return false; }
        for (size_t j = 0; j < n; ++j)
            if (std::find(seen.begin(), seen.end(), from[j]) == seen.end()) seen.push_back(from[j]);
    }
    return false;
}
void call_scratch_collect() {
    CallMemory & cm = call_memory();
    if (cm.dead_count.load(std::memory_order_acquire) == 0) return;
    std::lock_guard<std::mutex> lock(cm.mu);
    RelaxedCapture relaxed;
    free_dead_blocks(cm);
}

// SM100_CALL_SCRATCH=0: every call takes the path that needs no memory (for tests)
int call_scratch_alloc(cudaStream_t s, size_t bytes, CallScratch * out) {
    static const bool off = [] { const char * e = getenv("SM100_CALL_SCRATCH"); return e != nullptr && e[0] == '0'; }();
    *out = CallScratch{};
    if (off) return ST_OOM;
    int dev = 0;
    SM100_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) return fail(ST_UNSUPPORTED, "device ordinal %d is beyond the table of %d", dev, MAX_DEVICES);
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    cudaGraph_t graph = nullptr;
    const cudaGraphNode_t * deps = nullptr;
    const cudaGraphEdgeData * edges = nullptr;
    size_t dep_count = 0;
    SM100_CUDA(cudaStreamGetCaptureInfo_v3(s, &status, &capture, &graph, &deps, &edges, &dep_count));
    CallMemory & cm = call_memory();
    std::lock_guard<std::mutex> lock(cm.mu);
    RelaxedCapture relaxed;
    free_dead_blocks(cm);
    if (status == cudaStreamCaptureStatusActive) {
        size_t want = bytes;
        for (GraphBlock * b : cm.blocks) {
            if (b->capture != capture || b->last == nullptr || !precedes(b->last, deps, dep_count)) continue;
            if (b->bytes >= bytes) {
                b->last = nullptr;
                out->ptr = b->ptr;
                out->block = b;
                return ST_OK;
            }
            if (want < 2 * b->bytes) want = 2 * b->bytes;   // the smaller ones add up to less than the largest
        }
        GraphBlock * block = new GraphBlock{capture, nullptr, want, nullptr};
        cudaError_t e = cudaMalloc(&block->ptr, want);
        if (e != cudaSuccess) {
            (void) cudaGetLastError();
            delete block;
            return cuda_fail(e, "cudaMalloc(memory of a captured call)");
        }
        cudaUserObject_t owner = nullptr;
        e = cudaUserObjectCreate(&owner, block, graph_block_dead, 1, cudaUserObjectNoDestructorSync);
        if (e == cudaSuccess) {
            e = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
            if (e != cudaSuccess) {
                (void) cudaGetLastError();
                (void) cudaUserObjectRelease(owner, 1);   // the destructor gives the block back
                return cuda_fail(e, "cudaGraphRetainUserObject");
            }
        } else {
            (void) cudaGetLastError();
            (void) cudaFree(block->ptr);
            delete block;
            return cuda_fail(e, "cudaUserObjectCreate");
        }
        cm.blocks.push_back(block);
        out->ptr = block->ptr;
        out->block = block;
        return ST_OK;
    }
    if (cm.pools[dev] == nullptr) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t fresh = nullptr;
        SM100_CUDA(cudaMemPoolCreate(&fresh, &props));
        uint64_t keep = CALL_POOL_KEEP;
        SM100_CUDA(cudaMemPoolSetAttribute(fresh, cudaMemPoolAttrReleaseThreshold, &keep));
        cm.pools[dev] = fresh;
    }
    const cudaError_t e = cudaMallocFromPoolAsync(&out->ptr, bytes, cm.pools[dev], s);
    if (e != cudaSuccess) {
        (void) cudaGetLastError();
        out->ptr = nullptr;
        return cuda_fail(e, "cudaMallocFromPoolAsync");
    }
    out->pooled = true;
    return ST_OK;
}
int call_scratch_free(cudaStream_t s, const CallScratch & m) {
    if (m.pooled) SM100_CUDA(cudaFreeAsync(m.ptr, s));
    if (m.block != nullptr) {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        const cudaGraphNode_t * deps = nullptr;
        const cudaGraphEdgeData * edges = nullptr;
        size_t dep_count = 0;
        SM100_CUDA(cudaStreamGetCaptureInfo_v3(s, &status, nullptr, nullptr, &deps, &edges, &dep_count));
        CallMemory & cm = call_memory();
        std::lock_guard<std::mutex> lock(cm.mu);
        if (status == cudaStreamCaptureStatusActive && dep_count == 1) m.block->last = deps[0];   // the call's last kernel
    }
    return ST_OK;
}

// ---- fault words ----
// One word per device and kernel family in mapped host memory: a kernel that gives up on a bounded wait writes its wait site + 1
// there (it goes on to the end, so the word has arrived when the stream is synchronised).  Reading them costs no call, so every
// synchronisation looks at all of them, whatever was launched and however: directly, from a graph, on another stream.
struct FaultWords { int word[MAX_DEVICES][16]; };   // a cache line per device
static std::atomic<FaultWords *> g_faults{nullptr};
static int fault_words(FaultWords ** out) {
    static std::mutex mu;
    FaultWords * f = g_faults.load(std::memory_order_acquire);
    if (f == nullptr) {
        std::lock_guard<std::mutex> lock(mu);
        f = g_faults.load(std::memory_order_acquire);
        if (f == nullptr) {
            RelaxedCapture relaxed;
            SM100_CUDA(cudaHostAlloc((void **) &f, sizeof(FaultWords), cudaHostAllocPortable | cudaHostAllocMapped));
            std::memset(f, 0, sizeof(FaultWords));
            g_faults.store(f, std::memory_order_release);
        }
    }
    *out = f;
    return ST_OK;
}
int fault_word(int family, int ** out) {
    FaultWords * f = nullptr;
    const int st = fault_words(&f);
    *out = st == ST_OK ? &f->word[current_device()][family] : nullptr;
    return st;
}
static int poll_faults(int dev) {
    FaultWords * f = g_faults.load(std::memory_order_acquire);
    if (f == nullptr || dev < 0 || dev >= MAX_DEVICES) return ST_OK;
    static const char * const what[FAULT_FAMILIES] = {"the tensor-core GEMM gave up waiting on a pipeline barrier", "the split tensor-core GEMM gave up waiting on a pipeline barrier",
                                                      "the Q4_K matvec gave up waiting for a weight copy"};
    for (int i = 0; i < FAULT_FAMILIES; ++i) {
        const int v = __atomic_load_n(&f->word[dev][i], __ATOMIC_ACQUIRE) == 0 ? 0 : __atomic_exchange_n(&f->word[dev][i], 0, __ATOMIC_ACQ_REL);
        if (v != 0) return fail(ST_BACKEND, "mul_mat: %s (site %d); its output is incomplete", what[i], v - 1);
    }
    return ST_OK;
}

// Waits for the stream, then reads the fault words of the STREAM's device (the current device may be another one in a process
// that drives several GPUs).
static int sync_and_poll(cudaStream_t st) {
    SM100_CUDA(cudaStreamSynchronize(st));
    call_scratch_collect();
    int dev = 0;
    if (st == nullptr || cudaStreamGetDevice(st, &dev) != cudaSuccess) {
        if (st != nullptr) (void) cudaGetLastError();
        dev = current_device();
    }
    return poll_faults(dev);
}

}  // namespace sm100

using namespace sm100;

extern "C" {

const char * sm100_last_error(void) { return t_error.c_str(); }

int sm100_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int sm100_device_info(int device, char * name, size_t name_size, uint64_t * total_memory, uint32_t * sms,
                      uint32_t * cc_major, uint32_t * cc_minor, uint64_t * shared_per_block) {
    cudaDeviceProp p;
    SM100_CUDA(cudaGetDeviceProperties(&p, device));
    if (name != nullptr && name_size > 0) {
        std::strncpy(name, p.name, name_size - 1);
        name[name_size - 1] = '\0';
    }
    if (total_memory) *total_memory = p.totalGlobalMem;
    if (sms) *sms = (uint32_t) p.multiProcessorCount;
    if (cc_major) *cc_major = (uint32_t) p.major;
    if (cc_minor) *cc_minor = (uint32_t) p.minor;
    if (shared_per_block) *shared_per_block = p.sharedMemPerBlockOptin;
    return ST_OK;
}

int sm100_set_device(int device) {
    SM100_CUDA(cudaSetDevice(device));
    return ST_OK;
}

int sm100_malloc(int device, size_t size, void ** out) {
    if (out == nullptr || size == 0) return fail(ST_INVALID, "sm100_malloc: out is null or size is 0");
    *out = nullptr;
    SM100_CUDA(cudaSetDevice(device));
    SM100_CUDA(cudaMalloc(out, size));  // cudaMalloc returns at least 256-byte aligned memory
    return ST_OK;
}

int sm100_free(int device, void * ptr) {
    if (ptr == nullptr) return ST_OK;
    SM100_CUDA(cudaSetDevice(device));
    SM100_CUDA(cudaFree(ptr));
    return ST_OK;
}

int sm100_host_alloc(size_t size, void ** out) {
    if (out == nullptr || size == 0) return fail(ST_INVALID, "sm100_host_alloc: out is null or size is 0");
    SM100_CUDA(cudaHostAlloc(out, size, cudaHostAllocPortable));
    return ST_OK;
}

int sm100_host_free(void * ptr) {
    if (ptr != nullptr) SM100_CUDA(cudaFreeHost(ptr));
    return ST_OK;
}

int sm100_stream_create(int device, sm100_stream_t * out) {
    if (out == nullptr) return fail(ST_INVALID, "sm100_stream_create: out is null");
    SM100_CUDA(cudaSetDevice(device));
    cudaStream_t s = nullptr;
    SM100_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    *out = s;
    return ST_OK;
}

int sm100_stream_destroy(int device, sm100_stream_t stream) {
    if (stream == nullptr) return ST_OK;
    SM100_CUDA(cudaSetDevice(device));
    stream_tail_set((cudaStream_t) stream, TAIL_OTHER);   // a later stream may get the same handle
    SM100_CUDA(cudaStreamDestroy((cudaStream_t) stream));
    return ST_OK;
}

int sm100_stream_sync(sm100_stream_t stream) { return sync_and_poll((cudaStream_t) stream); }

int sm100_memcpy_h2d(sm100_stream_t s, void * dst, const void * src, size_t n, int blocking) {
    if (n == 0) return ST_OK;
    stream_tail_set((cudaStream_t) s, TAIL_OTHER);
    SM100_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, (cudaStream_t) s));
    if (blocking) SM100_CUDA(cudaStreamSynchronize((cudaStream_t) s));
    return ST_OK;
}

int sm100_memcpy_d2h(sm100_stream_t s, void * dst, const void * src, size_t n, int blocking) {
    if (n == 0) return ST_OK;
    stream_tail_set((cudaStream_t) s, TAIL_OTHER);
    SM100_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, (cudaStream_t) s));
    // a blocking read makes results visible like a stream_sync does (include/scrapgpu/op.h:190-194), so a kernel that
    // gave up on a bounded wait is reported here too instead of handing out an incomplete result with status OK
    if (blocking) return sync_and_poll((cudaStream_t) s);
    return ST_OK;
}

int sm100_memcpy_d2d(sm100_stream_t s, void * dst, const void * src, size_t n, int blocking) {
    if (n == 0) return ST_OK;
    stream_tail_set((cudaStream_t) s, TAIL_OTHER);
    // overlapping ranges get memmove semantics through a stream-ordered temporary
    const char * a = (const char *) src;
    char * b = (char *) dst;
    if (a == b) return ST_OK;
    if ((b > a && b < a + n) || (a > b && a < b + n)) {
        void * tmp = nullptr;
        SM100_CUDA(cudaMallocAsync(&tmp, n, (cudaStream_t) s));
        cudaError_t e = cudaMemcpyAsync(tmp, src, n, cudaMemcpyDeviceToDevice, (cudaStream_t) s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst, tmp, n, cudaMemcpyDeviceToDevice, (cudaStream_t) s);
        cudaFreeAsync(tmp, (cudaStream_t) s);
        if (e != cudaSuccess) return cuda_fail(e, "sm100_memcpy_d2d");
    } else {
        SM100_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToDevice, (cudaStream_t) s));
    }
    if (blocking) SM100_CUDA(cudaStreamSynchronize((cudaStream_t) s));
    return ST_OK;
}

int sm100_memset(sm100_stream_t s, void * dst, int byte, size_t n, int blocking) {
    if (n == 0) return ST_OK;
    stream_tail_set((cudaStream_t) s, TAIL_OTHER);
    SM100_CUDA(cudaMemsetAsync(dst, byte, n, (cudaStream_t) s));
    if (blocking) SM100_CUDA(cudaStreamSynchronize((cudaStream_t) s));
    return ST_OK;
}

int sm100_memcpy_peer(sm100_stream_t dst_stream, int dst_device, void * dst, sm100_stream_t src_stream, int src_device,
                      const void * src, size_t n) {
    if (n == 0) return ST_OK;
    // order: after everything enqueued on src_stream, before later work on dst_stream
    cudaEvent_t ready = nullptr;
    SM100_CUDA(cudaSetDevice(src_device));
    SM100_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(ready, (cudaStream_t) src_stream);
    if (e == cudaSuccess) e = cudaSetDevice(dst_device);
    if (e == cudaSuccess) e = cudaStreamWaitEvent((cudaStream_t) dst_stream, ready, 0);
    if (e == cudaSuccess) e = cudaMemcpyPeerAsync(dst, dst_device, src, src_device, n, (cudaStream_t) dst_stream);
    cudaEventDestroy(ready);
    if (e != cudaSuccess) return cuda_fail(e, "sm100_memcpy_peer");
    return ST_OK;
}

int sm100_peer_access(int device, int peer) {
    if (device == peer) return ST_OK;
    int can = 0;
    SM100_CUDA(cudaDeviceCanAccessPeer(&can, device, peer));
    if (!can) return fail(ST_UNSUPPORTED, "device %d cannot map the memory of device %d", device, peer);
    int cur = 0;
    SM100_CUDA(cudaGetDevice(&cur));
    SM100_CUDA(cudaSetDevice(device));
    const cudaError_t e = cudaDeviceEnablePeerAccess(peer, 0);
    (void) cudaSetDevice(cur);
    if (e == cudaErrorPeerAccessAlreadyEnabled) {
        (void) cudaGetLastError();
        return ST_OK;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceEnablePeerAccess");
    return ST_OK;
}

int sm100_event_create(sm100_event_t * out) {
    if (out == nullptr) return fail(ST_INVALID, "sm100_event_create: out is null");
    cudaEvent_t e = nullptr;
    SM100_CUDA(cudaEventCreate(&e));
    *out = e;
    return ST_OK;
}

int sm100_event_destroy(sm100_event_t e) {
    if (e != nullptr) SM100_CUDA(cudaEventDestroy((cudaEvent_t) e));
    return ST_OK;
}

int sm100_event_record(sm100_event_t e, sm100_stream_t s) {
    SM100_CUDA(cudaEventRecord((cudaEvent_t) e, (cudaStream_t) s));
    return ST_OK;
}

int sm100_stream_wait_event(sm100_stream_t s, sm100_event_t e) {
    SM100_CUDA(cudaStreamWaitEvent((cudaStream_t) s, (cudaEvent_t) e, 0));
    return ST_OK;
}

int sm100_event_sync(sm100_event_t e) {
    SM100_CUDA(cudaEventSynchronize((cudaEvent_t) e));
    return ST_OK;
}

int sm100_event_elapsed_ms(sm100_event_t start, sm100_event_t stop, float * ms) {
    SM100_CUDA(cudaEventElapsedTime(ms, (cudaEvent_t) start, (cudaEvent_t) stop));
    return ST_OK;
}

int sm100_fault_word(int device, int family, int ** word_out) {
    if (word_out == nullptr || device < 0 || device >= MAX_DEVICES || family < 0 || family >= FAULT_FAMILIES) return fail(ST_INVALID, "fault_word: bad argument");
    FaultWords * f = nullptr;
    const int st = fault_words(&f);
    if (st == ST_OK) *word_out = &f->word[device][family];
    return st;
}

int sm100_graph_begin(sm100_stream_t s) {
    SM100_CUDA(cudaStreamBeginCapture((cudaStream_t) s, cudaStreamCaptureModeThreadLocal));
    return ST_OK;
}

int sm100_graph_end(sm100_stream_t s, sm100_graph_t * out) {
    if (out == nullptr) return fail(ST_INVALID, "sm100_graph_end: out is null");
    cudaGraph_t g = nullptr;
    SM100_CUDA(cudaStreamEndCapture((cudaStream_t) s, &g));
    cudaGraphExec_t exec = nullptr;
    cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate");
    *out = exec;
    return ST_OK;
}

int sm100_graph_launch(sm100_graph_t g, sm100_stream_t s) {
    stream_tail_set((cudaStream_t) s, TAIL_OTHER);
    SM100_CUDA(cudaGraphLaunch((cudaGraphExec_t) g, (cudaStream_t) s));
    return ST_OK;
}

int sm100_graph_destroy(sm100_graph_t g) {
    if (g != nullptr) SM100_CUDA(cudaGraphExecDestroy((cudaGraphExec_t) g));
    call_scratch_collect();
    return ST_OK;
}

uint64_t sm100_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

int sm100_scratch_reserve(int slot, size_t bytes) {
    void * p = nullptr;
    return device_scratch(slot, bytes, &p);
}

int sm100_set_pdl(int enabled) {
    g_pdl.store(enabled ? 1 : 0, std::memory_order_relaxed);
    return ST_OK;
}

int sm100_launch_serialized(int on) {
    t_serialized = on ? 1 : 0;
    return ST_OK;
}

}  // extern "C"
