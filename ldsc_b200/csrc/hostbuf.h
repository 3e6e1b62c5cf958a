// hostbuf.h -- host memory of a context's copies.
#pragma once
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <vector>

namespace ldsc {

// Host end of a call's copies, kept by the context (grow-only): page-locked up
// to PINNED_MAX, so a copy neither blocks the host nor goes through the driver's
// staging buffer; larger, or where none can be locked, ordinary memory.  One
// pageable copy of each result left the device idle for 25 to 50 us before the
// next could start.  Locking and unlocking pages waits for the device and stalls
// the other contexts on it, so a context starts with what most calls need,
// growth at least doubles, and locked pages stay with the context to its end,
// outgrown ones too (together less than 2 PINNED_MAX).  A trim, which a server
// does to an idle slot while the others run, gives back ordinary memory alone.
struct HostBuf {
    static constexpr size_t PINNED_MAX = 64ull << 20;
    struct Block {
        uint8_t* p;
        size_t cap;
        bool pinned;
    };
    uint8_t* p = nullptr;
    size_t cap = 0;
    std::vector<Block> blocks;   // the last one is p
    uint8_t* ensure(size_t bytes) {   // null: out of memory
        if (bytes <= cap && p) return p;
        bytes = std::max(bytes + bytes / 8 + 4096, 2 * cap);
        Block b{nullptr, bytes, false};
        b.pinned = bytes <= PINNED_MAX &&
                   cudaHostAlloc(reinterpret_cast<void**>(&b.p), bytes, cudaHostAllocDefault) == cudaSuccess;
        if (!b.pinned) {
            cudaGetLastError();
            b.p = static_cast<uint8_t*>(std::malloc(bytes));
            if (!b.p) return nullptr;
        }
        blocks.push_back(b);
        use_last();
        return p;
    }
    void trim() {
        for (const Block& b : blocks)
            if (!b.pinned) std::free(b.p);
        blocks.erase(std::remove_if(blocks.begin(), blocks.end(), [](const Block& b) { return !b.pinned; }), blocks.end());
        use_last();
    }
    void release() {
        trim();
        for (const Block& b : blocks) cudaFreeHost(b.p);
        blocks.clear();
        use_last();
    }

private:
    void use_last() {
        p = blocks.empty() ? nullptr : blocks.back().p;
        cap = blocks.empty() ? 0 : blocks.back().cap;
    }
};

}  // namespace ldsc
