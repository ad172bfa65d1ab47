// mem_pool.cpp — the library's stream-ordered memory pools.
//
// Builds allocate and free their working arrays on the build's stream.  The
// device's default pool hands freed memory back to the driver at every
// synchronisation, so each build would map its scratch again (hundreds of
// MB for a 1024^3 mesh build).  The library therefore keeps one pool per
// device whose release threshold is unbounded: freed scratch stays mapped
// for the next build until svo_trim_memory() returns it.
//
// Octrees themselves (words and descriptor tables) live in a second pool that
// keeps at most kHandleKeep of freed memory mapped (the words of loaded octrees
// and of those made from words are the driver's), so that a program that
// replaces an octree every frame does not map and unmap it each time: a
// rebuilt 200x131x177 volume spent 130 us freeing the octree before it and 100
// allocating its own, of 385.  A pool holding more than that in live octrees
// returns whatever is freed at the next synchronisation, as before.  Arrays of
// kHandleDirect bytes or more, which it would not keep for long, are the
// driver's, for the pool maps memory more slowly: with a 1 GB table the first
// trace of a 2048^3 terrain waited 3.2 ms for it, 2.3 ms with the driver's.
//
// A pool hands out freed memory again at once, so the device has to be done
// with an octree before its memory goes back.  cudaDeviceSynchronize cannot be
// that wait: it is refused while any stream of any thread is captured, and it
// ends the capture.  cudaFree waits for all streams (also non-blocking ones: a
// 20 ms kernel held it for 20 ms) and minds no capture of another thread in
// thread-local or relaxed mode, so the wait is the cudaFree of 256 bytes taken
// for it: 2 us where another small block keeps their 2 MB mapped, 58 where not
// (a rebuilt and viewed 200x131x177 volume takes 165 to 175 us with either).
// What cannot be waited for (in a global capture, where cudaFree is refused
// too) is parked until the next octree is destroyed or memory is trimmed.
#include <cstring>
#include <mutex>
#include <vector>

#include "svo_internal.h"

namespace svo {

namespace {
constexpr int kMaxDevices = 64;
constexpr uint64_t kHandleKeep = 1ull << 30;
constexpr size_t kHandleDirect = 512ull << 20;
enum Pool { kScratch, kHandles, kPools };
std::mutex g_pool_mtx;
cudaMemPool_t g_pools[kMaxDevices][kPools] = {};
cudaStream_t g_streams[kMaxDevices] = {};
// host slots: a call takes one for its duration, so the calls of up to
// kMaxSlots threads run side by side
constexpr int kMaxSlots = 16;
std::vector<HostSlot *> g_free_slots[kMaxDevices];
int g_slots[kMaxDevices] = {};
std::vector<HandleMemory> g_parked[kMaxDevices];
void *g_small[kMaxDevices] = {};  // keeps the block that wait_for_device's 256 bytes come from mapped

cudaError_t pool_for_current_device(Pool which, cudaMemPool_t *out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_pool_mtx);
    cudaMemPool_t &slot = g_pools[dev][which];
    if (!slot) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool;
        e = cudaMemPoolCreate(&pool, &props);
        if (e != cudaSuccess) return e;
        uint64_t keep = which == kScratch ? ~0ull : kHandleKeep;
        e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return e;
        }
        slot = pool;
        if (!g_small[dev] && cudaMalloc(&g_small[dev], 256) != cudaSuccess) {
            g_small[dev] = nullptr;
            cudaGetLastError();
        }
    }
    *out = slot;
    return cudaSuccess;
}

// Waits for everything that the device runs, or is refused (see the top).
cudaError_t wait_for_device() {
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, 256);
    if (e == cudaSuccess) e = cudaFree(p);
    else if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        e = cudaDeviceSynchronize();
    }
    if (e != cudaSuccess) cudaGetLastError();  // a refusal is no later call's error
    return e;
}

cudaError_t pool_alloc(Pool which, void **p, size_t bytes, cudaStream_t st) {
    cudaMemPool_t pool;
    cudaError_t e = pool_for_current_device(which, &pool);
    if (e != cudaSuccess) return e;
    return cudaMallocFromPoolAsync(p, bytes, pool, st);
}
}  // namespace

cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t st) { return pool_alloc(kScratch, p, bytes, st); }

cudaError_t handle_alloc(void **p, size_t bytes, cudaStream_t st) {
    return bytes < kHandleDirect ? pool_alloc(kHandles, p, bytes, st) : cudaMalloc(p, bytes);
}

cudaError_t handle_free(void *p, size_t bytes, cudaStream_t st) {
    return bytes < kHandleDirect ? cudaFreeAsync(p, st) : cudaFree(p);
}

void handle_retire(const HandleMemory *blocks, int n) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
    std::vector<HandleMemory> ready(blocks, blocks + n);
    {
        // what is parked before the wait may go after it
        std::lock_guard<std::mutex> lk(g_pool_mtx);
        ready.insert(ready.end(), g_parked[dev].begin(), g_parked[dev].end());
        g_parked[dev].clear();
    }
    cudaStream_t st = nullptr;
    const bool waited = library_stream(&st) == cudaSuccess && wait_for_device() == cudaSuccess;
    std::vector<HandleMemory> left;
    for (const HandleMemory &m : ready) {
        if (!m.p) continue;
        if (waited && (m.plain ? cudaFree(m.p) : handle_free(m.p, m.bytes, st)) == cudaSuccess) continue;
        if (waited) cudaGetLastError();  // refused since: a capture has begun
        left.push_back(m);
    }
    if (left.empty()) return;
    std::lock_guard<std::mutex> lk(g_pool_mtx);
    g_parked[dev].insert(g_parked[dev].end(), left.begin(), left.end());
}

size_t words_bytes(uint64_t n) { return (size_t)(status_offset(n) + kStatusWords) * sizeof(uint32_t); }

cudaError_t alloc_words(uint32_t **words, uint64_t n, cudaStream_t st, bool plain) {
    void *p = nullptr;
    const uint64_t at = status_offset(n);
    cudaError_t e = plain ? cudaMalloc(&p, words_bytes(n)) : handle_alloc(&p, words_bytes(n), st);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync((uint32_t *)p + at, 0, kStatusWords * sizeof(uint32_t), st);
    if (e != cudaSuccess) {
        free_words((uint32_t *)p, n, st, plain);
        return e;
    }
    *words = (uint32_t *)p;
    return cudaSuccess;
}

void free_words(uint32_t *words, uint64_t n, cudaStream_t st, bool plain) {
    if (!words) return;
    if (plain) cudaFree(words);
    else handle_free(words, words_bytes(n), st);
}

cudaError_t library_stream(cudaStream_t *out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_pool_mtx);
    if (!g_streams[dev]) {
        e = cudaStreamCreateWithFlags(&g_streams[dev], cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            g_streams[dev] = nullptr;
            return e;
        }
    }
    *out = g_streams[dev];
    return cudaSuccess;
}

static void host_slot_free(HostSlot *s) {
    if (s->st) cudaStreamDestroy(s->st);
    if (s->order) cudaEventDestroy(s->order);
    if (s->host) cudaFreeHost(s->host);
    delete s;
}

HostSlot *host_slot_take() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    {
        std::lock_guard<std::mutex> lk(g_pool_mtx);
        if (!g_free_slots[dev].empty()) {
            HostSlot *s = g_free_slots[dev].back();
            g_free_slots[dev].pop_back();
            return s;
        }
        if (g_slots[dev] >= kMaxSlots) return nullptr;
        ++g_slots[dev];
    }
    HostSlot *s = new HostSlot{dev, nullptr, nullptr, nullptr, nullptr};
    void *h = nullptr, *d = nullptr;
    cudaError_t e = cudaHostAlloc(&h, kHostSlotBytes, cudaHostAllocMapped);
    s->host = (char *)h;
    if (e == cudaSuccess) e = cudaHostGetDevicePointer(&d, h, 0);
    s->dev = (char *)d;
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->order, cudaEventDisableTiming);
    if (e == cudaSuccess) return s;
    cudaGetLastError();  // the call takes the staged path instead
    host_slot_free(s);
    std::lock_guard<std::mutex> lk(g_pool_mtx);
    --g_slots[dev];
    return nullptr;
}

void host_slot_give(HostSlot *s) {
    std::lock_guard<std::mutex> lk(g_pool_mtx);
    g_free_slots[s->device].push_back(s);
}

cudaError_t Report::open(cudaStream_t st) {
    st_ = st;
    slot_ = host_slot_take();
    if (slot_) {
        std::memset(slot_->host, 0, kWords * sizeof(uint32_t));
        dev_ = (uint32_t *)slot_->dev;
        return cudaSuccess;
    }
    void *p = nullptr;
    cudaError_t e = scratch_alloc(&p, kWords * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    dev_ = (uint32_t *)p;
    return cudaMemsetAsync(dev_, 0, kWords * sizeof(uint32_t), st);
}

cudaError_t Report::wait() {
    cudaError_t e = cudaSuccess;
    if (!slot_) e = cudaMemcpyAsync(copy_, dev_, sizeof copy_, cudaMemcpyDeviceToHost, st_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
    busy_ = e != cudaSuccess;
    return e;
}

Report::~Report() {
    if (slot_) {
        if (busy_) cudaStreamSynchronize(st_);  // a call that ended early: its kernels may still write
        host_slot_give(slot_);
    } else if (dev_) {
        cudaFreeAsync(dev_, st_);
    }
}

// Frees the idle slots of a device.
static void host_slots_trim(int dev) {
    std::vector<HostSlot *> idle;
    {
        std::lock_guard<std::mutex> lk(g_pool_mtx);
        idle.swap(g_free_slots[dev]);
        g_slots[dev] -= (int)idle.size();
    }
    for (HostSlot *s : idle) host_slot_free(s);
}

}  // namespace svo

extern "C" int svo_trim_memory(void) {
    svo::clear_error();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return svo::cuda_fail(e, "cudaGetDevice");
    if (dev >= 0 && dev < svo::kMaxDevices) svo::host_slots_trim(dev);
    svo::handle_retire(nullptr, 0);  // what is parked
    cudaMemPool_t pools[svo::kPools] = {};
    {
        std::lock_guard<std::mutex> lk(svo::g_pool_mtx);
        for (int k = 0; k < svo::kPools; ++k)
            if (dev >= 0 && dev < svo::kMaxDevices) pools[k] = svo::g_pools[dev][k];
    }
    bool any = false;
    for (cudaMemPool_t p : pools) any = any || p;
    if (!any) return SVO_OK;
    e = cudaDeviceSynchronize();
    for (cudaMemPool_t p : pools)
        if (p && e == cudaSuccess) e = cudaMemPoolTrimTo(p, 0);
    if (e != cudaSuccess) return svo::cuda_fail(e, "trimming the memory pools");
    return SVO_OK;
}
