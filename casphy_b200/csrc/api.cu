// Library-wide C ABI helpers: status strings, last-error text, the per-device
// workspace arena, and device selection.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"
#include "runtime.h"

static thread_local char g_last_error[512] = "";

void casphy_set_last_cuda_error(cudaError_t e, const char* what, const char* file, int line) {
    snprintf(g_last_error, sizeof(g_last_error), "%s:%d %s -> %s (%s)", file, line, what,
             cudaGetErrorName(e), cudaGetErrorString(e));
}
void casphy_set_last_error_msg(const char* msg) {
    snprintf(g_last_error, sizeof(g_last_error), "%s", msg);
}

extern "C" int casphy_abi_version(void) { return CASPHY_ABI_VERSION; }

extern "C" const char* casphy_last_error(void) { return g_last_error; }

extern "C" int casphy_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

extern "C" int casphy_set_device(int device) {
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        casphy_set_last_cuda_error(e, "cudaSetDevice", __FILE__, __LINE__);
        return CASPHY_ECUDA;
    }
    return CASPHY_OK;
}

extern "C" const char* casphy_strerror(int s) {
    switch (s) {
        case CASPHY_OK: return "ok";
        case CASPHY_EINVAL: return "invalid argument";
        case CASPHY_ERANGE: return "value out of supported range";
        case CASPHY_ENOMEM: return "out of memory";
        case CASPHY_ECUDA: return "CUDA runtime error";
        case CASPHY_ETIMEOUT: return "device-side wait timed out";
        case CASPHY_EIO: return "input/output error";
        case CASPHY_ENODEV: return "no CUDA device";
        case CASPHY_EINTERNAL: return "internal error";
        default: return "unknown status";
    }
}

namespace casphy {

// Grow-only device arena per device.  Calls hold the device's lock for their
// whole duration, so one process runs one hot-path call per GPU at a time;
// separate processes (the R fork-cluster pattern) each have their own arena.
struct Arena {
    std::mutex mu;
    void* base = nullptr;
    size_t cap = 0;
    void* aux = nullptr;  // second grow-only block for outputs sized mid-call
    size_t auxCap = 0;
    char* pinned = nullptr;  // slots of staged copies, and when each was last copied out of or into
    cudaEvent_t slotFree[16] = {nullptr};
};
static std::mutex g_arenas_mu;
static std::vector<Arena*> g_arenas;

static Arena* arena_for(int dev) {
    std::lock_guard<std::mutex> g(g_arenas_mu);
    if ((int)g_arenas.size() <= dev) g_arenas.resize(dev + 1, nullptr);
    if (!g_arenas[dev]) g_arenas[dev] = new Arena();
    return g_arenas[dev];
}

DeviceScope::DeviceScope() {
    cudaGetDevice(&dev);
    arena = arena_for(dev);
    static_cast<Arena*>(arena)->mu.lock();
}
DeviceScope::~DeviceScope() { static_cast<Arena*>(arena)->mu.unlock(); }

// Grow-only block: a bigger request frees the old block and allocates
// 1/8 more than asked (or exactly the request when that fails).
static int grow(void** base, size_t* cap, size_t bytes, const char* what) {
    if (bytes > *cap) {
        if (*base) cudaFree(*base);
        *base = nullptr;
        *cap = 0;
        size_t want = bytes + (bytes >> 3);
        cudaError_t e = cudaMalloc(base, want);
        if (e != cudaSuccess) {
            cudaGetLastError();
            e = cudaMalloc(base, bytes);
            want = bytes;
        }
        if (e != cudaSuccess) {
            cudaGetLastError();
            *base = nullptr;
            casphy_set_last_cuda_error(e, what, __FILE__, __LINE__);
            return CASPHY_ENOMEM;
        }
        *cap = want;
    }
    return CASPHY_OK;
}

int DeviceScope::reserve(size_t bytes, void** out) {
    Arena* a = static_cast<Arena*>(arena);
    const int rc = grow(&a->base, &a->cap, bytes, "cudaMalloc(arena)");
    if (rc) return rc;
    *out = a->base;
    return CASPHY_OK;
}

int DeviceScope::reserve_aux(size_t bytes, void** out) {
    Arena* a = static_cast<Arena*>(arena);
    const int rc = grow(&a->aux, &a->auxCap, bytes, "cudaMalloc(aux)");
    if (rc) return rc;
    *out = a->aux;
    return CASPHY_OK;
}

// Staged copies.  The driver copies a pageable buffer through its own staging
// on the calling thread: 12 GB/s on a B200 host whose link takes 55 GB/s, 20 where
// the buffer is in the host's caches.  kCopyThreads threads with four 1 MiB slots each
// reach 40 GB/s (eight were no faster: starting them took what they gained).  They
// live for one copy, so buffers below kCopyMin stay with the driver (a call around one
// upload by the driver and by threads, 10.1 MiB not in the caches 1.18 and 1.02 ms, 16
// MiB 1.79 and 1.30, 32 MiB 3.46 and 2.01; in the caches 0.78 and 0.91, 1.12 and 1.17,
// 2.15 and 1.72; around a download to new pages, 11 MiB 2.6 and 1.2 ms, 32 MiB 7.0
// and 2.7); the slots stay with the arena, whose lock the caller holds.
constexpr size_t kCopySlot = size_t(1) << 20, kCopyMin = size_t(10) << 20;
constexpr int kCopyThreads = 4, kCopyTurns = 4, kCopySlots = kCopyTurns * kCopyThreads;

static bool staging_ready(Arena* a) {
    if (a->pinned) return true;
    void* p = nullptr;
    if (cudaHostAlloc(&p, kCopySlot * kCopySlots, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    for (int i = 0; i < kCopySlots; i++)
        if (!a->slotFree[i] && cudaEventCreateWithFlags(&a->slotFree[i], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            cudaFreeHost(p);
            return false;
        }
    a->pinned = static_cast<char*>(p);
    return true;
}

// Whether a copy of this host buffer is worth staging: large and pageable.
static bool stage_copy(Arena* a, const void* host, size_t bytes) {
    if (bytes < kCopyMin) return false;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered && staging_ready(a);
}

// Runs work(i) on kCopyThreads threads, the caller's among them; fewer when the
// system refuses one (the shares come from a common counter, so nothing is left
// undone).  The first CUDA error of any of them is returned.
template <class F>
static cudaError_t on_threads(int dev, F work) {
    std::atomic<int> err{(int)cudaSuccess};
    auto body = [&](int i) {
        cudaError_t e = i ? cudaSetDevice(dev) : cudaSuccess;
        if (e == cudaSuccess) e = work(i);
        int ok = (int)cudaSuccess;
        if (e != cudaSuccess) err.compare_exchange_strong(ok, (int)e);
    };
    std::vector<std::thread> t;
    try {
        t.reserve(kCopyThreads);
        for (int i = 1; i < kCopyThreads; i++) t.emplace_back(body, i);
    } catch (...) {
    }
    body(0);
    for (auto& x : t) x.join();
    return (cudaError_t)err.load();
}

int Staged::to_device(DeviceScope& ds, void* dst, const void* src, size_t bytes, void* stream) {
    Arena* a = static_cast<Arena*>(ds.arena);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!stage_copy(a, src, bytes)) {
        CASPHY_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        return CASPHY_OK;
    }
    const size_t chunks = (bytes + kCopySlot - 1) / kCopySlot;
    std::atomic<size_t> next{0};
    CASPHY_CUDA_TRY(on_threads(ds.dev, [&](int i) {
        for (int turn = 0;; turn = (turn + 1) % kCopyTurns) {
            const size_t c = next.fetch_add(1);
            if (c >= chunks) return cudaSuccess;
            const int slot = kCopyTurns * i + turn;
            const size_t off = c * kCopySlot, len = std::min(kCopySlot, bytes - off);
            char* p = a->pinned + (size_t)slot * kCopySlot;
            cudaError_t e = cudaEventSynchronize(a->slotFree[slot]);
            if (e != cudaSuccess) return e;
            std::memcpy(p, static_cast<const char*>(src) + off, len);
            if ((e = cudaMemcpyAsync(static_cast<char*>(dst) + off, p, len, cudaMemcpyHostToDevice, st)) != cudaSuccess)
                return e;
            if ((e = cudaEventRecord(a->slotFree[slot], st)) != cudaSuccess) return e;
        }
    }));
    return CASPHY_OK;
}

int Staged::to_host(DeviceScope& ds, void* dst, const void* src, size_t bytes, void* stream) {
    Arena* a = static_cast<Arena*>(ds.arena);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!stage_copy(a, dst, bytes)) {
        CASPHY_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        CASPHY_CUDA_TRY(cudaStreamSynchronize(st));
        return CASPHY_OK;
    }
    const size_t chunks = (bytes + kCopySlot - 1) / kCopySlot;
    std::atomic<size_t> next{0};
    CASPHY_CUDA_TRY(on_threads(ds.dev, [&](int i) {
        size_t at[2] = {chunks, chunks};  // the chunk under way in each of two slots
        for (int turn = 0;; turn ^= 1) {
            const int slot = kCopyTurns * i + turn;
            const size_t c = next.fetch_add(1);
            cudaError_t e;
            if (c < chunks) {
                // (an earlier call's copy out of this slot may be under way)
                if ((e = cudaEventSynchronize(a->slotFree[slot])) != cudaSuccess) return e;
                const size_t off = c * kCopySlot, len = std::min(kCopySlot, bytes - off);
                if ((e = cudaMemcpyAsync(a->pinned + (size_t)slot * kCopySlot, static_cast<const char*>(src) + off, len,
                                         cudaMemcpyDeviceToHost, st)) != cudaSuccess)
                    return e;
                if ((e = cudaEventRecord(a->slotFree[slot], st)) != cudaSuccess) return e;
            }
            at[turn] = c;
            // empty the other slot while this one fills
            const int o = turn ^ 1;
            if (at[o] < chunks) {
                if ((e = cudaEventSynchronize(a->slotFree[kCopyTurns * i + o])) != cudaSuccess) return e;
                const size_t off = at[o] * kCopySlot;
                std::memcpy(static_cast<char*>(dst) + off, a->pinned + (size_t)(kCopyTurns * i + o) * kCopySlot,
                            std::min(kCopySlot, bytes - off));
                at[o] = chunks;
            }
            if (at[0] >= chunks && at[1] >= chunks) return cudaSuccess;
        }
    }));
    return CASPHY_OK;
}

int ReadBack::run(const u32* from, void* stream) const {
    constexpr size_t kTogether = 4096;
    u32 all[kTogether];
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    size_t n = 0;
    for (int i = 0; i < parts; i++) n += part[i].n;
    const bool together = n <= kTogether;
    if (together && n) CASPHY_CUDA_TRY(cudaMemcpyAsync(all, from, sizeof(u32) * n, cudaMemcpyDeviceToHost, st));
    for (int i = 0; i < parts && !together; from += part[i++].n)
        if (part[i].n)
            CASPHY_CUDA_TRY(cudaMemcpyAsync(part[i].to, from, sizeof(u32) * part[i].n, cudaMemcpyDeviceToHost, st));
    CASPHY_CUDA_TRY(cudaStreamSynchronize(st));
    const u32* p = all;
    for (int i = 0; i < parts && together; p += part[i++].n)
        if (part[i].n) std::memcpy(part[i].to, p, sizeof(u32) * part[i].n);
    return CASPHY_OK;
}

int require_device() {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        cudaGetLastError();
        casphy_set_last_error_msg("no CUDA device visible");
        return CASPHY_ENODEV;
    }
    return CASPHY_OK;
}

}  // namespace casphy
