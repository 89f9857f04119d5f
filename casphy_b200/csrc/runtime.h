// Host-side runtime pieces shared by the entry points: the per-device
// workspace arena (one lock per device held for a whole call) and a bump
// allocator that carves typed, 256-byte aligned buffers out of it.
#pragma once
#include <cstddef>
#include <cstdint>

namespace casphy {

struct DeviceScope {
    int dev = 0;
    void* arena = nullptr;
    DeviceScope();
    ~DeviceScope();
    // Returns a device block of at least `bytes`, valid until the scope ends.
    // A later reserve() in the same scope may move the block.
    int reserve(size_t bytes, void** out);
    // A second block, independent of reserve()'s, for outputs whose size is
    // only known part-way through a call.
    int reserve_aux(size_t bytes, void** out);
};

// Copies of large pageable host buffers: kCopyMin bytes and more go through
// pinned slots of the device's arena, filled or emptied by several host
// threads (the driver's own staging copies on one).  to_device returns when
// every copy is queued on the stream, with a pageable src read; a page-locked one
// may still be read until the stream has passed the copy.  to_host returns when
// dst has been written, after all work queued on the stream before.
struct Staged {
    static int to_device(DeviceScope& ds, void* dst, const void* src, size_t bytes, void* stream);
    static int to_host(DeviceScope& ds, void* dst, const void* src, size_t bytes, void* stream);
};

// Results that lie one behind the other on the device, read back to the host
// arrays they belong to.  A copy to pageable memory costs about 8 us, so a few KB
// come in one copy.
struct ReadBack {
    struct Part {
        uint32_t* to;
        size_t n;
    };
    Part part[5];
    int parts = 0;
    void add(uint32_t* to, size_t n) { part[parts++] = Part{to, n}; }
    // Waits for the stream; the parts are filled when it returns 0.
    int run(const uint32_t* from, void* stream) const;
};

struct Carve {
    size_t off = 0;
    char* base = nullptr;
    template <class T>
    T* take(size_t n) {
        off = (off + 255) & ~size_t(255);
        T* p = reinterpret_cast<T*>(base ? base + off : nullptr);
        off += n * sizeof(T);
        return p;
    }
};

int require_device();

}  // namespace casphy
