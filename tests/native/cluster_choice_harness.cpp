// What a solve does where clusters cannot run (nirnaya_b200/csrc/cluster_plan.hpp).
#include "cluster_plan.hpp"

#include <cstdio>
#include <memory>
#include <stdexcept>

int main() {
    int bad = 0;
    auto expect = [&](bool ok, const char* what) {
        if (!ok) {
            std::printf("%s\n", what);
            ++bad;
        }
    };
    // a device that holds clusters of up to `most`
    for (int most : {0, 1, 2, 4, 8, 16})
        for (int C : {1, 2, 4, 8, 16})
            expect(nir::cl_size_held(C, [&](int c) { return c <= most ? 3 : 0; }) == (C <= most ? C : most), "size");
    // sizes it holds are not asked of others
    int asked = 0;
    expect(nir::cl_size_held(8, [&](int) { return ++asked; }) == 8 && asked == 1, "asked once");
    expect(nir::cl_size_held(0, [&](int) { return 1; }) == 0, "no cluster wanted");

    using Plan = std::unique_ptr<int>;
    expect(*nir::cl_if_memory([] { return std::make_unique<int>(7); }) == 7, "the plan");
    expect(nir::cl_if_memory([]() -> Plan { return nullptr; }) == nullptr, "no plan");
    expect(nir::cl_if_memory([]() -> Plan { throw std::bad_alloc(); }) == nullptr, "no memory");
    bool thrown = false;
    try {
        nir::cl_if_memory([]() -> Plan { throw std::runtime_error("a launch failed"); });
    } catch (const std::runtime_error&) {
        thrown = true;
    }
    expect(thrown, "other errors are reported");
    std::printf("%s\n", bad ? "failed" : "ok");
    return bad;
}
