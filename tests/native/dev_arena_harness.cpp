// The engine's device memory (nirnaya_b200/csrc/dev_arena.hpp) on a host
// allocator in the place of the CUDA runtime's.
#include "dev_arena.hpp"

#include <cstdio>
#include <cstdlib>
#include <map>

namespace {
std::map<char*, size_t> g_live;
int bad = 0;

void expect(bool ok, const char* what) {
    if (!ok) {
        std::printf("%s\n", what);
        ++bad;
    }
}

bool inside(const void* p, size_t n) {
    const char* q = static_cast<const char*>(p);
    for (auto& b : g_live)
        if (q >= b.first && q + n <= b.first + b.second) return true;
    return false;
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    g_live[static_cast<char*>(*p)] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    g_live.erase(static_cast<char*>(p));
    std::free(p);
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

int main() {
    using nir::DevArena;
    {
        // scratch inside the chunk
        DevArena m;
        m.reserve(1 << 16);
        m.alloc(1000);
        const DevArena::Mark k = m.mark();
        void* s = m.alloc(5000);
        m.rewind(k);
        expect(m.alloc(5000) == s, "the scratch's place is taken again");
        m.clear();
    }
    for (size_t scratch : {size_t(20000), size_t(200000), size_t(3) << 20}) {
        // scratch that did not fit the chunk: in a small chunk, in one of
        // its size, in a block of its own
        DevArena m;
        m.reserve(size_t(1) << 20);
        m.alloc((size_t(1) << 20) - 16384);
        const DevArena::Mark k = m.mark();
        const long long bytes = m.bytes;
        m.alloc(scratch);
        m.alloc(100);
        m.rewind(k);
        expect(m.bytes == bytes && g_live.size() == 1, "the blocks added for scratch are given back");
        for (int i = 0; i < 40; ++i) {
            const size_t n = size_t(1000) << (i % 8);
            expect(inside(m.alloc(n), DevArena::aligned(n)), "an allocation outside of every block");
        }
        m.clear();
        expect(g_live.empty() && m.bytes == 0, "everything given back");
    }
    {
        // a mark before the first chunk
        DevArena m;
        const DevArena::Mark k = m.mark();
        m.alloc(100);
        m.rewind(k);
        expect(g_live.empty() && inside(m.alloc(100), 256), "from the start");
        m.clear();
    }
    std::printf("%s\n", bad ? "failed" : "ok");
    return bad;
}
