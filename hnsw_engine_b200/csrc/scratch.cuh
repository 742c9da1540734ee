// Device memory that a host thread keeps from one call to the next: one block for each device, since a thread
// may call on several and a block is memory of one. Host code; Mem does the allocating, so that a test can
// stand in for the GPU.
#pragma once

#include <cstddef>

// Mem: static bool device(int *ordinal);              the current device
//      static bool alloc(void **p, size_t bytes);     on the current device
//      static void release(int ordinal, void *p);     memory of that device, whichever is current
template <class Mem>
class DeviceScratch {
   public:
    static constexpr int MAX_DEVICES = 64;

    DeviceScratch() = default;
    DeviceScratch(const DeviceScratch &) = delete;
    DeviceScratch &operator=(const DeviceScratch &) = delete;
    ~DeviceScratch() {
        for (int d = 0; d < MAX_DEVICES; d++)
            if (blocks_[d].p) Mem::release(d, blocks_[d].p);
    }

    // The current device's block of at least `bytes` (it only grows), or NULL.
    void *get(size_t bytes) {
        int d = -1;
        if (!Mem::device(&d) || d < 0 || d >= MAX_DEVICES) return nullptr;
        Block &b = blocks_[d];
        if (bytes <= b.bytes) return b.p;
        if (b.p) Mem::release(d, b.p);
        b = Block{};
        void *p = nullptr;
        if (!Mem::alloc(&p, bytes)) return nullptr;
        b = Block{p, bytes};
        return p;
    }

   private:
    struct Block {
        void *p = nullptr;
        size_t bytes = 0;
    };
    Block blocks_[MAX_DEVICES];
};
