// The worker threads of a cluster plan (nirnaya_b200/csrc/cluster_plan.hpp)
// when the memory for one of them runs out while another already works.
#include "cluster_plan.hpp"

#include <cstdio>
#include <cstdlib>
#include <new>

namespace {
thread_local int t_allocations_left = -1;  // of this thread; < 0: any number
}

void* operator new(size_t n) {
    if (t_allocations_left == 0) throw std::bad_alloc();
    if (t_allocations_left > 0) --t_allocations_left;
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main() {
    int bad = 0;
    // the vector of threads, then none, one or two of them
    for (int left = 1; left <= 3; ++left) {
        std::atomic<int> done{0};
        t_allocations_left = left;
        nir::cl_for_each(1000, 8, [&](int) { ++done; });
        t_allocations_left = -1;
        if (done != 1000) ++bad;
    }
    std::printf("%s\n", bad ? "failed" : "ok");
    return bad;
}
