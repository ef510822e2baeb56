// Device memory of a handle.  Host only.
#pragma once

#include <cuda_runtime_api.h>

#include <algorithm>
#include <new>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

namespace nir {

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
// The device is out of memory: a caller that can do without may go on.
struct CudaNoMemory : std::bad_alloc {
    std::string text;
    explicit CudaNoMemory(std::string t) : text(std::move(t)) {}
    const char* what() const noexcept override { return text.c_str(); }
};

[[noreturn]] inline void cuda_failed(cudaError_t e, const char* call, const char* file, int line) {
    (void)cudaGetLastError();  // reported here and not by the next launch's check too
    const std::string t =
        std::string(call) + ": " + cudaGetErrorString(e) + " (" + file + ":" + std::to_string(line) + ")";
    if (e == cudaErrorMemoryAllocation) throw CudaNoMemory(t);
    throw CudaError(t);
}

#define NIR_CUDA(call)                                                            \
    do {                                                                          \
        cudaError_t e_ = (call);                                                  \
        if (e_ != cudaSuccess) nir::cuda_failed(e_, #call, __FILE__, __LINE__);   \
    } while (0)

// Device memory in chunks that allocations are carved from: large ones
// reserved beforehand for what is known to come, small ones on demand, and
// a block of its own for what is large and fits none.  A cudaMalloc takes
// 20 us below 64 KB, 70 at 300 KB and 330 from 2 MB on, its cudaFree as
// long, and a handle holds about 60 arrays.
struct DevArena {
    static constexpr size_t kAlign = 256, kOwn = size_t(1) << 20, kSmallChunk = size_t(128) << 10;
    static size_t aligned(size_t bytes) { return (std::max<size_t>(1, bytes) + kAlign - 1) / kAlign * kAlign; }
    struct Block {
        char* p;
        size_t size, used;
        bool carved;  // a chunk; false: one allocation
    };
    std::vector<Block> blocks;
    int cur = -1;  // the chunk being carved
    long long bytes = 0;

    char* block(size_t size, bool carved) {
        blocks.reserve(blocks.size() + 1);
        void* p = nullptr;
        NIR_CUDA(cudaMalloc(&p, size));
        blocks.push_back({static_cast<char*>(p), size, 0, carved});
        bytes += (long long)size;
        return static_cast<char*>(p);
    }
    void reserve(size_t size) {
        block(size, true);
        cur = int(blocks.size()) - 1;
    }
    void* alloc(size_t size) {
        size = aligned(size);
        if (cur < 0 || blocks[size_t(cur)].size - blocks[size_t(cur)].used < size) {
            if (size >= kOwn) return block(size, false);
            reserve(std::max(size, kSmallChunk));
        }
        Block& c = blocks[size_t(cur)];
        char* p = c.p + c.used;
        c.used += size;
        return p;
    }
    // Frees a block of its own; a carved allocation stays with its chunk.
    void release(void* p) {
        for (size_t i = 0; i < blocks.size(); ++i)
            if (blocks[i].p == p && !blocks[i].carved) {
                cudaFree(p);
                bytes -= (long long)blocks[i].size;
                blocks.erase(blocks.begin() + long(i));
                if (cur > int(i)) --cur;
                return;
            }
    }
    // Scratch is given back by rewinding to the mark set before it: what was
    // carved since, and the blocks that were added for it.
    struct Mark {
        size_t blocks;
        int cur;
        size_t used;
    };
    Mark mark() const { return {blocks.size(), cur, cur < 0 ? 0 : blocks[size_t(cur)].used}; }
    void rewind(const Mark& m) {
        while (blocks.size() > m.blocks) {
            cudaFree(blocks.back().p);
            bytes -= (long long)blocks.back().size;
            blocks.pop_back();
        }
        cur = m.cur;
        if (cur >= 0) blocks[size_t(cur)].used = m.used;
    }
    void clear() {
        for (auto& b : blocks) cudaFree(b.p);
        blocks.clear();
        cur = -1;
        bytes = 0;
    }
};

}  // namespace nir
