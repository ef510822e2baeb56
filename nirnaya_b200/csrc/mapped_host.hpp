// Small blocks of host memory that kernels write to, kept for the next
// handle: taking one from the driver costs 1 to 3 ms, giving it back 0.4,
// of the 4 a handle's creation takes.
//
// The memory is this process's own and only registered with the driver, for
// a program may reset the device between two handles, which drops every
// registration: a block is looked up again, and registered anew, each time
// it is handed out.  (Memory that the driver had allocated would be gone,
// and its address perhaps another's.)  Blocks are kept per device, so that
// resetting one leaves the handles on another alone.
#pragma once

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <map>
#include <mutex>
#include <new>
#include <vector>

namespace nir {

constexpr size_t kHostPage = 4096;  // blocks are whole pages: a registration takes pages

// Makes the block at p usable by kernels of the current device.
inline cudaError_t map_host_block(void* p, size_t bytes) {
    cudaPointerAttributes a{};
    cudaError_t e = cudaPointerGetAttributes(&a, p);
    if (e == cudaSuccess && a.type != cudaMemoryTypeHost) {
        e = cudaHostRegister(p, bytes, cudaHostRegisterMapped | cudaHostRegisterPortable);
        if (e == cudaSuccess) e = cudaPointerGetAttributes(&a, p);
    }
    // kernels are given the host's address (one address space on this platform)
    if (e == cudaSuccess && a.devicePointer != p) e = cudaErrorNotSupported;
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e;
}

// Blocks of one size.  At most kKeep per device stay, for the life of the
// process, beside those that handles hold.  Any thread may take and give; a
// block belongs to one handle in between, whose stream has ended when it is
// given back.
class MappedBlocks {
public:
    static constexpr size_t kKeep = 16;
    explicit MappedBlocks(size_t bytes) : bytes_((bytes + kHostPage - 1) / kHostPage * kHostPage) {}

    // On the current device, `device`.
    cudaError_t take(int device, void** out) {
        *out = nullptr;
        void* p = nullptr;
        {
            std::lock_guard<std::mutex> g(mu_);
            auto& f = free_[device];
            f.reserve(kKeep);
            if (!f.empty()) {
                p = f.back();
                f.pop_back();
            }
        }
        if (!p) p = std::aligned_alloc(kHostPage, bytes_);
        if (!p) return cudaErrorMemoryAllocation;
        const cudaError_t e = map_host_block(p, bytes_);
        if (e != cudaSuccess) {
            drop(p);
            return e;
        }
        *out = p;
        return cudaSuccess;
    }

    void give(int device, void* p) {
        {
            std::lock_guard<std::mutex> g(mu_);
            auto it = free_.find(device);
            if (it != free_.end() && it->second.size() < kKeep) {
                it->second.push_back(p);  // within the capacity reserved by take
                return;
            }
        }
        drop(p);
    }

private:
    static void drop(void* p) {
        if (cudaHostUnregister(p) != cudaSuccess) (void)cudaGetLastError();
        std::free(p);
    }
    const size_t bytes_;
    std::mutex mu_;
    std::map<int, std::vector<void*>> free_;
};

}  // namespace nir
