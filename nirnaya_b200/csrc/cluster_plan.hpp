// The host's part of a cluster plan (k_cluster.cuh): which rows and columns
// each rank of an instance's cluster owns, their order, and the slices.
// Host only, no CUDA calls.
#pragma once

#include <vector_types.h>

#include <algorithm>
#include <atomic>
#include <exception>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace nir {

// f(0) .. f(n-1) on the calling thread and up to `threads - 1` more; the
// first exception is rethrown here once every thread has ended, and a
// thread that cannot be started only leaves more work to the others.
template <class F>
void cl_for_each(int n, int threads, F&& f) {
    std::atomic<int> next{0};
    std::exception_ptr err;
    std::mutex mu;
    auto work = [&]() {
        try {
            for (int i = next++; i < n; i = next++) f(i);
        } catch (...) {
            std::lock_guard<std::mutex> g(mu);
            if (!err) err = std::current_exception();
            next = n;
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(size_t(std::max(threads, 1)));
    for (int t = 1; t < threads; ++t) {
        try {
            pool.emplace_back(work);
        } catch (const std::exception&) {  // no thread, or no memory for one
            break;
        }
    }
    work();
    for (auto& th : pool) th.join();
    if (err) std::rethrow_exception(err);
}

// One side (rows of A, or rows of A') of every instance of a plan.
struct ClHostSide {
    std::vector<int> order;             // position -> row
    std::vector<int> pos;               // row -> position
    std::vector<unsigned char> rank;    // row -> rank
    std::vector<int> bound;             // [i (C+1) + r], instance-local positions
    std::vector<int> sl_lo, base;       // [i C + r], one entry more at the end
    std::vector<int4> slices;           // first row (rank-local), unit (rank-local), pairs | log2 T << 24, rows
    std::vector<int> owner;             // slice -> i C + r
};

// Work of a row beside its nonzeros, in nonzeros: the epilogue's loads and
// the stores to the ranks.
constexpr int kClRowWork = 4;
// Warps of a rank its slices are dealt to (k_cluster.cuh's CTA).
constexpr int kClPlanWarps = 24;
constexpr int kClStepsMin = 4, kClStepsMax = 16;

inline int cl_row_lanes(int len, int steps) {
    int lt = 0;
    while (lt < 5 && ((len + (1 << lt) - 1) >> lt) > steps) ++lt;
    return lt;
}

// The slices of one rank: rows longest first, so that the rows of a slice
// have about the same length.  T lanes share a row so that no lane has more
// than `steps` entries: the fewest steps with which every warp has at most
// one slice (a pass then takes one slice's latency, about 1,500 cycles
// however short it is), and 16 where the rank has more rows than that.
inline void cl_rank_slices(const int* order, const int* rp, int n, int owner, std::vector<int4>& out,
                           std::vector<int>& own, int* units) {
    int steps = kClStepsMax;
    if (n <= 32 * kClPlanWarps)
        for (int t = kClStepsMin; t < kClStepsMax; t += 2) {
            int p = 0, count = 0;
            while (p < n) {
                const int r = order[p];
                p += 32 >> cl_row_lanes(rp[r + 1] - rp[r], t);
                ++count;
            }
            if (count <= kClPlanWarps) {
                steps = t;
                break;
            }
        }
    int p = 0, unit = 0;
    while (p < n) {
        const int r = order[p], len = rp[r + 1] - rp[r], lt = cl_row_lanes(len, steps);
        const int cnt = std::min(32 >> lt, n - p);
        const int pairs = (((len + (1 << lt) - 1) >> lt) + 1) / 2;
        out.push_back(int4{p, unit, pairs | (lt << 24), cnt});
        own.push_back(owner);
        unit += pairs;
        p += cnt;
    }
    *units = unit;
}

// Partition, order and slices of one side for clusters of C CTAs.  off: the
// instances' row offsets; rp: the CSR row pointers.  Each rank gets a
// contiguous range of the instance's rows of about equal work, so that a
// block-structured matrix keeps its blocks together.
inline void cl_build_side(const std::vector<int>& off, const std::vector<int>& rp, int C, ClHostSide& s) {
    const int count = int(off.size()) - 1, rows = off[size_t(count)];
    s.order.resize(size_t(rows));
    s.pos.resize(size_t(rows));
    s.rank.resize(size_t(rows));
    s.bound.assign(size_t(count) * (C + 1), 0);
    s.sl_lo.assign(size_t(count) * C + 1, 0);
    s.base.assign(size_t(count) * C + 1, 0);
    std::vector<std::vector<int4>> sl(static_cast<size_t>(count));
    std::vector<std::vector<int>> own(static_cast<size_t>(count));
    std::vector<int> nsl(size_t(count) * C, 0), nun(size_t(count) * C, 0);
    auto one = [&](int i) {
        const int r0 = off[size_t(i)], r1 = off[size_t(i) + 1];
        auto work = [&](int r) { return (long long)rp[size_t(r)] + (long long)kClRowWork * r; };
        const long long w0 = work(r0), total = work(r1) - w0;
        int* b = &s.bound[size_t(i) * (C + 1)];
        std::vector<int> cnt;
        for (int k = 1; k <= C; ++k) {
            int e = r1;
            if (k < C) {
                // the first row at or past the k-th share
                int lo = r0 + b[k - 1], hi = r1;
                const long long target = w0 + total * k / C;
                while (lo < hi) {
                    const int mid = lo + (hi - lo) / 2;
                    if (work(mid) < target) lo = mid + 1;
                    else hi = mid;
                }
                e = lo;
            }
            b[k] = e - r0;
            const int s0 = r0 + b[k - 1], n = e - s0;
            // counting sort by length, longest first, stable
            int mx = 0;
            for (int r = s0; r < e; ++r) mx = std::max(mx, rp[size_t(r) + 1] - rp[size_t(r)]);
            cnt.assign(size_t(mx) + 2, 0);
            for (int r = s0; r < e; ++r) ++cnt[size_t(mx - (rp[size_t(r) + 1] - rp[size_t(r)])) + 1];
            for (int l = 0; l <= mx; ++l) cnt[size_t(l) + 1] += cnt[size_t(l)];
            for (int r = s0; r < e; ++r) {
                const int p = s0 + cnt[size_t(mx - (rp[size_t(r) + 1] - rp[size_t(r)]))]++;
                s.order[size_t(p)] = r;
                s.pos[size_t(r)] = p;
                s.rank[size_t(r)] = (unsigned char)(k - 1);
            }
            const size_t before = sl[size_t(i)].size();
            cl_rank_slices(s.order.data() + s0, rp.data(), n, i * C + k - 1, sl[size_t(i)], own[size_t(i)],
                           &nun[size_t(i) * C + size_t(k) - 1]);
            nsl[size_t(i) * C + size_t(k) - 1] = int(sl[size_t(i)].size() - before);
        }
    };
    const int threads = rows > 100000 ? int(std::min<unsigned>(8, std::max(1u, std::thread::hardware_concurrency()))) : 1;
    cl_for_each(count, threads, one);
    for (size_t b = 0; b < nsl.size(); ++b) {
        s.sl_lo[b + 1] = s.sl_lo[b] + nsl[b];
        s.base[b + 1] = s.base[b] + nun[b];
    }
    s.slices.clear();
    s.owner.clear();
    s.slices.reserve(size_t(s.sl_lo.back()));
    s.owner.reserve(size_t(s.sl_lo.back()));
    for (int i = 0; i < count; ++i) {
        s.slices.insert(s.slices.end(), sl[size_t(i)].begin(), sl[size_t(i)].end());
        s.owner.insert(s.owner.end(), own[size_t(i)].begin(), own[size_t(i)].end());
    }
}

// C, or the largest smaller cluster that the device can hold; 0 when it can
// hold none.  clusters(C) says how many of size C it holds at once.
template <class F>
int cl_size_held(int C, F&& clusters) {
    while (C > 0 && clusters(C) <= 0) C /= 2;
    return C;
}

// build's plan, or null when there is no memory for it: the per-launch
// kernels need none.
template <class Build>
auto cl_if_memory(Build&& build) -> decltype(build()) {
    try {
        return build();
    } catch (const std::bad_alloc&) {
        return nullptr;
    }
}

}  // namespace nir
