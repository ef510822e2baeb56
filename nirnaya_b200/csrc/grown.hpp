// A device buffer that grows on demand.  Host only, no CUDA calls.
#pragma once

#include <cstddef>

namespace nir {

// mem.alloc<T>(n) and mem.release(p) give and take the memory.  The buffer
// is empty while it is replaced, so that after an allocation that failed
// (and threw) no later, smaller request is served from memory already given
// back.
template <typename T>
struct Grown {
    T* p = nullptr;
    size_t len = 0;

    // At least n entries; what it held is lost when it grows.
    template <class Mem>
    T* ensure(Mem& mem, size_t n) {
        return n <= len ? p : renew(mem, n);
    }
    // n new entries in the place of what it held.
    template <class Mem>
    T* renew(Mem& mem, size_t n) {
        T* const old = p;
        p = nullptr;
        len = 0;
        if (old) mem.release(old);
        p = mem.template alloc<T>(n);
        len = n;
        return p;
    }
};

}  // namespace nir
