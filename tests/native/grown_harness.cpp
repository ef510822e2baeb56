// Grown buffers (nirnaya_b200/csrc/grown.hpp) on a memory that fails on
// demand and counts what is used after it was given back.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <set>

#include "grown.hpp"

namespace {

struct Mem {
    std::set<void*> live;
    bool fail = false;
    template <typename T>
    T* alloc(size_t n) {
        if (fail) throw std::bad_alloc();
        void* p = std::malloc(n * sizeof(T));
        live.insert(p);
        return static_cast<T*>(p);
    }
    void release(void* p) {
        if (live.erase(p) != 1) {
            std::printf("released twice\n");
            std::exit(1);
        }
        std::free(p);
    }
};

int bad = 0;
void expect(bool ok, const char* what) {
    if (!ok) {
        std::printf("%s\n", what);
        ++bad;
    }
}

}  // namespace

int main() {
    Mem m;
    nir::Grown<double> b;
    expect(b.ensure(m, 0) == nullptr && m.live.empty(), "nothing asked, nothing taken");
    double* p = b.ensure(m, 10);
    expect(p && b.len == 10 && b.ensure(m, 10) == p && b.ensure(m, 3) == p, "kept while it is large enough");
    m.fail = true;
    bool threw = false;
    try {
        b.ensure(m, 11);
    } catch (const std::bad_alloc&) {
        threw = true;
    }
    expect(threw && b.p == nullptr && b.len == 0 && m.live.empty(), "empty after a failure");
    threw = false;
    try {
        b.ensure(m, 3);  // used to be served from the memory given back
    } catch (const std::bad_alloc&) {
        threw = true;
    }
    expect(threw && b.p == nullptr, "a smaller request after a failure is a new one");
    m.fail = false;
    p = b.ensure(m, 3);
    expect(p && b.len == 3 && m.live.count(p) == 1, "works again");
    p = b.ensure(m, 20);
    expect(p && b.len == 20 && m.live.size() == 1 && m.live.count(p) == 1, "the smaller one was given back");
    p = b.renew(m, 5);
    expect(p && b.len == 5 && m.live.size() == 1, "renewed at a smaller size");
    m.fail = true;
    try {
        b.renew(m, 5);
    } catch (const std::bad_alloc&) {
    }
    expect(b.p == nullptr && b.len == 0 && m.live.empty(), "empty after a failed renewal");
    std::printf("%s\n", bad ? "failed" : "ok");
    return bad;
}
