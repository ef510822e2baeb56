// Chunks of iterations inside one thread-block cluster per LP.
//
// A small or medium LP spends its iteration on latency, not on bandwidth:
// two overlapping kernels take about 5.9 us on a 2,000 x 5,000 LP of
// 40,000 nonzeros whose arithmetic takes a tenth of that, and a batch of
// such LPs gathers from a vector that would fit in shared memory.  Here a
// cluster of C CTAs (C = 1, 2, 4, 8 or 16) takes one LP through a whole
// chunk: K iterations, the KKT evaluation, the controller and the restart.
//
//   * Rank r of the cluster owns a contiguous range of the rows and of the
//     columns (equal work).  Within it the rows are held longest first, in
//     slices of 32 / T rows with T lanes per row (T = 1, 2, ... 32), and a
//     slice's entries are stored lane by lane in pairs, so that a warp
//     reads indices and values with coalesced 4 / 8 / 16-byte loads and a
//     lane sums its entries without staging products or scanning rows.
//   * The entries of x-bar (y) that a rank's rows (columns) gather sit in
//     its shared memory, numbered 0.. ("slots"), so an index takes 16 bits
//     and a gather costs bank conflicts instead of L2 latency.  Whoever
//     computes an entry sends it to the ranks that gather it, all of a
//     rank's entries by one bulk copy where the receiver takes an eighth of
//     them or more, one by one (st.async) where it takes few; the bytes
//     count on the receiver's mbarrier; a half-iteration starts when its
//     entries have come, with no barrier over the cluster (its release fence
//     alone took 490 cycles).  On a block-structured matrix a rank holds
//     little more than its own part.
//   * What else fits is kept in shared memory too: the own vector entries,
//     the slots to store to, and the matrix itself.
//
// Measured on B200 (us per iteration, checks included, against the
// per-launch kernels): 2.5 against 4.3 on a 60 x 150 LP, 4.6 against 5.9 on
// the 2,000 x 5,000 one (16 CTAs); 85 against 186 for a batch of 128
// multiperiod LPs of 500 to 20,000 rows (16M nonzeros, clusters of 4), 5.9
// against 9.1 for 96 LPs of 50 to 400 rows (clusters of 1).  Small LPs are
// bound by the latency of a pass, about 1,300 cycles from the last arrival
// to the last departure; large ones by the shared-memory pipe, where 32
// random 8-byte gathers take 6 wavefronts.
//
// Sums are FP64, in an order fixed by the plan (never by timing); there are
// no atomics.  The
// arithmetic per row is that of k_iter.cuh's epilogues and the controller
// is the same function.
//
// Reference correspondence: src/gpu/pdhg_solver.hpp:69-95 (the two
// half-iterations) on src/core/csc_matrix.hpp:99-120's products.
#pragma once

#include <type_traits>

#include "k_adaptive.cuh"
#include "k_setup.cuh"

namespace nir {

constexpr int kClThreads = 768;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClRanksMax = 16;
constexpr int kClSums = 12;          // quantities of a check (CtlSums)
constexpr int kClWeights = 64;       // iterations whose Halpern weights are tabulated
constexpr int kClBulkPart = 8;       // a rank that gathers 1/8 of another's entries gets all of them by one copy
constexpr int kClUnit = 64;          // stream entries of one step pair: 32 lanes x 2
// Slots 0 and 1 of both sides hold zero throughout: the padding of a slice
// gathers slot 0, and its product is 0 whatever the iterate holds (a real
// entry's slot there turned an overflow in it, 0 x inf, into a NaN in every
// padded row).  Two, so that whole segments stay at even slots.
constexpr int kClZeroSlots = 2;

// What an instance keeps in shared memory beside the gathered entries and
// the slices.
constexpr int kClOwnShared = 1, kClPushShared = 2, kClMatShared = 4;

// One side of the plan: the rows (A, dual step) or the columns (A', primal
// step).  Positions are the plan's order of the side's rows; an instance's
// positions fill its own range [off[i], off[i+1]) and the ranks' ranges
// inside it follow each other.
struct ClSide {
    const int* off;               // count + 1
    const int* bound;             // [i (C+1) + r]: first local position of rank r
    const int* sl_lo;             // [i C + r]: first slice of rank r; the next entry ends it
    const int4* slices;           // first row (rank-local), stream unit (rank-local), pairs | log2 T << 24, rows
    const int* base;              // [i C + r]: first stream unit of rank r
    const unsigned short* idx;    // slots gathered from the other side's vector
    const float* v32;             // scaled values
    const double* v64;
    const unsigned short* need;   // [position]: other ranks that gather this entry and not all of its rank's
    const unsigned short* slot;   // [C off[i] + r rows_i + local position]
    const int* ghost;             // [i]: slots a rank holds of this side's vector (largest rank)
    const int* bytes;             // [i C + r]: bytes of it that reach rank r from others in one phase
    const unsigned short* bulk;   // [i C + r]: ranks that take all of rank r's entries
};

// Vectors in the plan's order: scaled (the iteration) and original (KKT).
// col: x x0 c lo up one after another, ncol entries each; row: y y0 rl ru.
constexpr int kClColVecs = 5, kClRowVecs = 4;
struct ClVecs {
    double *col, *row;
    size_t ncol, nrow;
    double *xp, *yp;
    const double *dc, *oc, *ol, *ou, *dr, *orl, *oru;
};

struct ClArgs {
    ClSide col, row;
    ClVecs v;
    const int* list;    // instances in launch order
    const int* flags;   // [instance]: kCl*Shared
    int C, K, halpern, phase;
    double rho;
    DevState* st;       // [instance]
    const double *bnorm, *cnorm, *offset;  // [instance], or null: the state's norms and ctl.offset
    int lost;           // test of the bounded waits: rank 0 waits for so many bytes that nobody sends
    CtlArgs ctl;
};

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The cluster's hardware barrier (start and end of a chunk).
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// Stores v at the shared-memory address of rank r that corresponds to addr here.
__device__ __forceinline__ void cl_store(unsigned addr, unsigned r, double v) {
    asm volatile(
        "{\n.reg .u32 ra;\nmapa.shared::cluster.u32 ra, %0, %1;\nst.shared::cluster.f64 [ra], %2;\n}" ::"r"(addr), "r"(r),
        "d"(v)
        : "memory");
}
// The address of rank r's shared memory that corresponds to addr here.
__device__ __forceinline__ unsigned cl_map(unsigned addr, unsigned r) {
    unsigned m;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(addr), "r"(r));
    return m;
}
// Stores v at a mapped address without waiting; its arrival counts 8 bytes
// on the mapped barrier (of the same rank).
__device__ __forceinline__ void cl_send(unsigned addr, unsigned bar, double v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar));
}
// Copies `bytes` from this CTA's shared memory to a mapped address (multiples
// of 16, as both addresses); their arrival counts on the mapped barrier.
__device__ __forceinline__ void cl_send_bulk(unsigned dst, unsigned src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Makes this thread's shared-memory stores visible to the bulk copies.
__device__ __forceinline__ void cl_fence_bulk() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void cl_bar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// One thread: opens the barrier's phase for `bytes` arriving bytes.
__device__ __forceinline__ void cl_bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for a phase's bytes, at most kClWaitCycles; false when they did not
// come (they always do: the senders run on the same cluster), at once when
// another wait has failed.  A CTA whose wait failed ends the iteration, with
// what it owes the others in it, and the chunk: it opens no phase and sends
// nothing any more, so no barrier is re-armed in the middle of a phase and
// none counts more than three phases' bytes.  The ranks that wait for it give
// up in turn.  All meet at the check's cluster barrier, after which nobody
// sends, and a cluster with a failed rank stays kClSettleCycles more, so
// that copies in flight land in shared memory that is still theirs.
constexpr long long kClWaitCycles = 2000000000LL, kClSettleCycles = 2000000LL;
__device__ __forceinline__ bool cl_bar_wait(unsigned bar, unsigned parity, const volatile int* failed) {
    long long t0 = 0;
    for (;;) {
        unsigned ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        const long long t = clock64();
        if (t0 == 0) t0 = t;
        if (*failed || t - t0 > kClWaitCycles) return false;
    }
}

template <typename T>
struct ClPair;
template <>
struct ClPair<float> {
    using type = float2;
};
template <>
struct ClPair<double> {
    using type = double2;
};

// An array of the rank's: at a byte offset of the dynamic shared memory
// (RES: everything of the instance fits there), or behind a pointer to
// shared or global memory.
extern __shared__ __align__(16) unsigned char cl_smem[];

template <bool RES, typename T>
struct ClPtr {
    T* p;
    int off;
    __device__ __forceinline__ T& operator[](size_t i) const {
        if constexpr (RES) return reinterpret_cast<T*>(cl_smem + off)[unsigned(i)];
        else return p[i];
    }
    __device__ __forceinline__ void set(T* q, bool shared) {
        p = q;
        off = shared ? int(reinterpret_cast<const unsigned char*>(q) - cl_smem) : 0;
    }
};

// One side of this rank as the passes see it.  The struct lies in shared
// memory, so that a pass holds in registers only what it uses.
template <bool RES, typename TV>
struct ClRank {
    using V2 = typename ClPair<TV>::type;
    int n;                                // own rows of this side
    int ns;                               // slices
    int sl;                               // their byte offset in shared memory
    ClPtr<RES, const ushort2> idx;        // their stream, pair by pair
    ClPtr<RES, const V2> val;
    ClPtr<RES, double> own;               // own entries: vector k at own + k * stride
    int stride;
    ClPtr<RES, const unsigned short> need;  // [row]
    ClPtr<RES, const unsigned short> slot;  // [r * slot_stride + row]
    int slot_stride;
    int seg;                              // byte offset of this rank's own entries among the slots
    unsigned bulk;                        // ranks that take all of them
    unsigned seg_bytes;
    unsigned dst[kClRanksMax];            // where in rank r they go (mapped)
    unsigned ghosts[kClRanksMax];         // rank r's slots (mapped)
    unsigned bars[kClRanksMax];           // rank r's barrier (mapped)
    unsigned bar, bytes;                  // this rank's, and how many bytes a phase brings it
    size_t p0;                            // first position (global)
    ClPtr<false, const ushort2> idx_g;    // the stream in global memory, with the FP64 values (KKT)
    ClPtr<false, const double2> val64;
};

// Adds N pairs of this lane: the stream's loads, then the gathers.  g: byte
// offset of the gathered vector (an offset and not a pointer, so that the
// gathers are shared-memory loads).
template <bool RES>
using ClAt = std::conditional_t<RES, unsigned, size_t>;

template <int N, bool RES, typename V2>
__device__ __forceinline__ void cl_pairs(const ClPtr<RES, const ushort2>& idx, const ClPtr<RES, const V2>& val,
                                         ClAt<RES>& at, int g, double& a0, double& a1) {
    const double* gx = reinterpret_cast<const double*>(cl_smem + g);
    ushort2 c[N];
    V2 v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        c[j] = idx[at + j * 32];
        v[j] = val[at + j * 32];
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        a0 += double(v[j].x) * gx[c[j].x];
        a1 += double(v[j].y) * gx[c[j].y];
    }
    at += N * 32;
}

// One pass over a rank's slices.  ready() waits for the gathered vector; what
// does not depend on it is loaded before.  pre(row) fetches the epilogue's
// operands ahead of the sum; fin(row, sum, operands, first, step) applies
// the epilogue on each of the row's T lanes alike, first = the lane's number
// among them, step = T.
template <class Q, bool RES, typename V2, class Ready, class Pre, class Fin>
__device__ __forceinline__ void cl_pass(int sl, int ns, const ClPtr<RES, const ushort2> idx,
                                        const ClPtr<RES, const V2> val, int g, Ready ready, Pre pre, Fin fin) {
    const int lane = threadIdx.x & 31;
    const int4* slices = reinterpret_cast<const int4*>(cl_smem + sl);
    int s = threadIdx.x >> 5;
    const bool any = s < ns;
    int4 d = any ? slices[s] : make_int4(0, 0, 0, 0);
    Q q{};
    if (any) q = pre((lane >> (d.z >> 24)) < d.w ? d.x + (lane >> (d.z >> 24)) : d.x);
    bool waited = false;
    while (s < ns) {
        const int lt = d.z >> 24, row = d.x + (lane >> lt);
        const bool live = (lane >> lt) < d.w;
        int np = d.z & 0xffffff;
        if (np > 0 && !waited) {
            ready();
            waited = true;
        }
        ClAt<RES> at = ClAt<RES>(unsigned(d.y)) * 32 + lane;
        double a0 = 0.0, a1 = 0.0;
        for (; np >= 4; np -= 4) cl_pairs<4, RES, V2>(idx, val, at, g, a0, a1);
        if (np & 2) cl_pairs<2, RES, V2>(idx, val, at, g, a0, a1);
        if (np & 1) cl_pairs<1, RES, V2>(idx, val, at, g, a0, a1);
        double a = a0 + a1;
        for (int o = (1 << lt) >> 1; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (live) fin(row, a, q, lane & ((1 << lt) - 1), 1 << lt);
        s += kClWarps;
        if (s < ns) {
            d = slices[s];
            q = pre((lane >> (d.z >> 24)) < d.w ? d.x + (lane >> (d.z >> 24)) : d.x);
        }
    }
    if (threadIdx.x == 0 && !waited) ready();  // thread 0 opens the next phase later
    __syncwarp();  // a row's other lanes read what its first one wrote
}

// Publishes v as entry `row` of a side: into this rank's own segment, from
// where it reaches the ranks that take all of it (cl_flush), and to those of
// the ranks first, first + step, ... that gather this entry alone (need).
template <class R>
__device__ __forceinline__ void cl_push(const R& S, int row, unsigned need, double v, int first, int step, int C) {
    if (first == 0) reinterpret_cast<double*>(cl_smem + S.seg)[row] = v;
    if (!need) return;
    // bits 0, step, 2 step, ... (step divides 32), from `first` on
    unsigned m = need & ((0xffffffffu / ((1ull << step) - 1ull)) << first);
    while (m) {
        const int r = __ffs(int(m)) - 1;
        m &= m - 1;
        cl_send(S.ghosts[r] + 8u * S.slot[size_t(r * S.slot_stride + row)], S.bars[r], v);
    }
}

// After a pass: its own segment is complete for this CTA, and on its way to
// the ranks that take all of it.  Every thread calls it.
template <class R>
__device__ __forceinline__ void cl_flush(const R& S) {
    if (S.bulk) cl_fence_bulk();
    __syncthreads();
    // one copy per warp: a copy takes about 50 cycles to issue
    if ((threadIdx.x & 31) == 0)
        for (int r = int(threadIdx.x >> 5); r < kClRanksMax; r += kClWarps)
            if ((S.bulk >> r) & 1u)
                cl_send_bulk(S.dst[r], unsigned(__cvta_generic_to_shared(cl_smem)) + unsigned(S.seg), S.seg_bytes, S.bars[r]);
}

template <typename T>
__device__ __forceinline__ void cl_copy(T* dst, const T* src, size_t n) {
    for (size_t i = threadIdx.x; i < n; i += kClThreads) dst[i] = src[i];
}

// 16-byte copies of n bytes (n and both addresses multiples of 16).
__device__ __forceinline__ void cl_copy16(void* dst, const void* src, size_t bytes) {
    cl_copy(static_cast<uint4*>(dst), static_cast<const uint4*>(src), bytes / 16);
}

// What the whole CTA reads during a chunk, in shared memory.
template <bool RES, typename TV>
struct ClShared {
    ClRank<RES, TV> col, row;
    unsigned long long bar[2];  // arrivals of x-bar and of y
    double tau, sigma, isigma, rho;
    int failed;             // a wait ran out
    int stop;               // the same at the end of the last dual pass
    double2 w[kClWeights];  // Halpern weights (k + 1) / (k + 2), 1 / (k + 2) of the chunk's first iterations
    double warp[kClWarps][kClSums];
    double rank[kClRanksMax][kClSums];
    double fail[kClRanksMax];  // 1: a wait of that rank ran out
};

__device__ __forceinline__ double2 cl_weights(double k) { return make_double2((k + 1.0) / (k + 2.0), 1.0 / (k + 2.0)); }

// A phase of a side's vector: thread 0 opens it (every pass, having waited
// for the one before), then those who gather wait for its bytes.  A CTA
// barrier ends every pass (cl_flush), so no thread is two phases behind.
// No sender overwrites what a slower rank still gathers: an entry of A joins
// a row of one rank and a column of another, so whoever receives from a rank
// also sends to it, after its gathers, and a rank waits for all it receives
// before it sends again.  That also frees the segment the bulk copies read.
template <bool RES, typename TV>
__device__ __forceinline__ void cl_open(const ClRank<RES, TV>& R) {
    if (threadIdx.x == 0) cl_bar_expect(R.bar, R.bytes);
}
template <bool RES, typename TV>
__device__ __forceinline__ void cl_await(ClShared<RES, TV>& S, const ClRank<RES, TV>& R, unsigned parity) {
    if (!cl_bar_wait(R.bar, parity, &S.failed)) S.failed = 1;
}

// The primal step over this rank's columns (own: x x0 c lo up); adds the
// check's norms to s[0..1].
template <bool RES, typename TV, bool CHECK>
__device__ __forceinline__ void cl_primal(ClShared<RES, TV>& S, int ys, unsigned parity, double* xp, double2 w,
                                          bool halpern, int C, double (&s)[2]) {
    struct Q {
        double x, c, lo, up, x0;
        unsigned need;
    };
    const ClRank<RES, TV>& R = S.col;
    const auto own = R.own;
    const auto need = R.need;
    const int st = R.stride;
    const double tau = S.tau, rho = S.rho;
    cl_open(S.row);
    cl_pass<Q, RES, typename ClPair<TV>::type>(
        R.sl, R.ns, R.idx, R.val, ys, [&]() { cl_await(S, S.row, parity); },
        [&](int j) { return Q{own[j], own[j + 2 * size_t(st)], own[j + 3 * size_t(st)], own[j + 4 * size_t(st)], own[j + size_t(st)], need[j]}; },
        [&](int j, double aty, const Q& q, int first, int step) {
            const double x1 = clamp_box(q.x - tau * (q.c - aty), q.lo, q.up);
            cl_push(R, j, q.need, 2.0 * x1 - q.x, first, step, C);
            if (first) return;
            double xn = x1;
            if (halpern) xn = w.x * ((1.0 + rho) * x1 - rho * q.x) + w.y * q.x0;
            own[j] = xn;
            if (CHECK) {
                xp[j] = x1;
                const double d = q.x - x1, e = x1 - q.x0;
                s[0] += d * d;
                s[1] += e * e;
            }
        });
    cl_flush(R);
}

// The dual step over this rank's rows (own: y y0 rl ru).  A check's KKT pass
// gathers y+ itself, so a check sends that.
template <bool RES, typename TV, bool CHECK>
__device__ __forceinline__ void cl_dual(ClShared<RES, TV>& S, int xs, unsigned parity, double* yp, double2 w,
                                        bool halpern, int C, double (&s)[2]) {
    struct Q {
        double y, rl, ru, y0;
        unsigned need;
    };
    const ClRank<RES, TV>& R = S.row;
    const auto own = R.own;
    const auto need = R.need;
    const int st = R.stride;
    const double sigma = S.sigma, isigma = S.isigma, rho = S.rho;
    cl_open(S.col);
    cl_pass<Q, RES, typename ClPair<TV>::type>(
        R.sl, R.ns, R.idx, R.val, xs, [&]() { cl_await(S, S.col, parity); },
        [&](int i) { return Q{own[i], own[i + 2 * size_t(st)], own[i + 3 * size_t(st)], own[i + size_t(st)], need[i]}; },
        [&](int i, double ax, const Q& q, int first, int step) {
            const double pr = clamp_box(ax - q.y * isigma, q.rl, q.ru);
            const double y1 = q.y + sigma * (pr - ax);
            double yn = y1;
            if (halpern) yn = w.x * ((1.0 + rho) * y1 - rho * q.y) + w.y * q.y0;
            cl_push(R, i, q.need, CHECK ? y1 : yn, first, step, C);
            if (first) return;
            own[i] = yn;
            if (CHECK) {
                yp[i] = y1;
                const double d = q.y - y1, e = y1 - q.y0;
                s[0] += d * d;
                s[1] += e * e;
            }
        });
    // What the CTA goes by: thread 0 opens the phases, so its own waits count
    // here at once; a wait of another thread that ends later, at the latest
    // with the next iteration.  (A vote of all threads in both barriers took
    // 1 to 4% of an iteration, this 0.1 to 1.2%.)
    if (threadIdx.x == 0) S.stop = S.failed;
    cl_flush(R);
}

// The rest of a check, once per chunk and kept out of the iterations'
// registers: the KKT sums of (x+, y+) in the original space on the FP64
// values, the reduction over the cluster and the controller.  A CTA that a
// wait of its iterations failed in only reports that.
template <bool RES, typename TV>
__device__ __noinline__ void cl_check(const ClArgs& a, ClShared<RES, TV>& S, int xs, int ys, unsigned parity, unsigned rank,
                                      int inst, DevState* st, double sp0, double sp1, double sd0, double sd1) {
    const int C = a.C, tid = threadIdx.x;
    // every warp is past its last phases; xp and yp as this CTA wrote them
    if (__syncthreads_and(S.failed == 0)) {
        const double* xp = a.v.xp + S.col.p0;
        const double* yp = a.v.yp + S.row.p0;
        // y+ has come from every rank whose rows gather x-bar from here: x+ may take its place there
        cl_open(S.row);
        cl_await(S, S.row, parity);
        __syncthreads();
        cl_open(S.col);
        for (int j = tid; j < S.col.n; j += kClThreads) cl_push(S.col, j, S.col.need[j], xp[j], 0, 1, C);
        cl_flush(S.col);
        double sum[kClSums] = {sp0, sp1, sd0, sd1};
        {
            KktColEpi<double> e;
            e.dc = a.v.dc + S.col.p0;
            e.c = a.v.oc + S.col.p0;
            e.l = a.v.ol + S.col.p0;
            e.u = a.v.ou + S.col.p0;
            using Pre = typename KktColEpi<double>::Pre;
            // x+ was written in this launch: a plain load, not the read-only path
            cl_pass<Pre, false, double2>(
                S.col.sl, S.col.ns, S.col.idx_g, S.col.val64, ys, []() {},
                [&](int j) { return Pre{__ldg(e.dc + j), __ldg(e.c + j), __ldg(e.l + j), __ldg(e.u + j), xp[j]}; },
                [&](int j, double aty, const Pre& p, int first, int) {
                    if (!first) e.row(j, aty, p);
                });
#pragma unroll
            for (int q = 0; q < 4; ++q) sum[8 + q] = e.q[q];
        }
        {
            KktRowEpi<double> e;
            e.dr = a.v.dr + S.row.p0;
            e.rl = a.v.orl + S.row.p0;
            e.ru = a.v.oru + S.row.p0;
            using Pre = typename KktRowEpi<double>::Pre;
            cl_pass<Pre, false, double2>(
                S.row.sl, S.row.ns, S.row.idx_g, S.row.val64, xs, [&]() { cl_await(S, S.col, parity); },
                [&](int i) { return Pre{__ldg(e.dr + i), __ldg(e.rl + i), __ldg(e.ru + i), yp[i]}; },
                [&](int i, double ax, const Pre& p, int first, int) {
                    if (!first) e.row(i, ax, p);
                });
#pragma unroll
            for (int q = 0; q < 4; ++q) sum[4 + q] = e.q[q];
        }

        // sums: lanes, then warps, then ranks, in order (sum[7] is a maximum)
#pragma unroll
        for (int q = 0; q < kClSums; ++q) {
            const double v = q == 7 ? warp_max(sum[q]) : warp_sum(sum[q]);
            if ((tid & 31) == 0) S.warp[tid >> 5][q] = v;
        }
        __syncthreads();
        if (tid < kClSums) {
            double v = 0.0;
            for (int k = 0; k < kClWarps; ++k) v = tid == 7 ? fmax(v, S.warp[k][tid]) : v + S.warp[k][tid];
            cl_store(unsigned(__cvta_generic_to_shared(&S.rank[rank][tid])), 0, v);
        }
    }
    // every rank learns of a failure
    if (tid < C) cl_store(unsigned(__cvta_generic_to_shared(&S.fail[rank])), unsigned(tid), S.failed ? 1.0 : 0.0);
    cl_sync();
    bool failed = false;
    for (int r = 0; r < C; ++r) failed |= S.fail[r] != 0.0;
    if (rank == 0 && tid == 0) {
        if (failed) {
            st->done = 1;
            st->status = 14;  // NIR_STATUS_INTERNAL_ERROR
        } else {
            double t[kClSums];
            for (int q = 0; q < kClSums; ++q) {
                t[q] = 0.0;
                for (int r = 0; r < C; ++r) t[q] = q == 7 ? fmax(t[q], S.rank[r][q]) : t[q] + S.rank[r][q];
            }
            const CtlSums s{t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], t[10], t[11]};
            control_update(a.ctl, st, s, a.bnorm ? a.bnorm[inst] : st->bnorm, a.cnorm ? a.cnorm[inst] : st->cnorm,
                           a.offset ? a.offset[inst] : a.ctl.offset, a.ctl.hist);
        }
        __threadfence();
    }
    if (failed)
        for (const long long t0 = clock64(); clock64() - t0 < kClSettleCycles;) __nanosleep(1000);
    cl_sync();
}

template <bool RES, typename TV>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_chunk(const __grid_constant__ ClArgs a) {
    __shared__ ClShared<RES, TV> S;
    const int C = a.C, tid = threadIdx.x;
    const unsigned rank = cl_rank();
    const int inst = a.list[blockIdx.x / C];
    DevState* st = a.st + inst;
    // no CTA changes the state before the barriers below: all decide alike
    if (__ldcg(&st->done) || __ldcg(&st->phase) != a.phase) return;
    const int flags = RES ? kClOwnShared | kClPushShared | kClMatShared : a.flags[inst];
    const long long k_base = __ldcg(&st->k_base);
    const bool halpern = a.halpern != 0;
    if (tid == 0) {
        S.tau = __ldcg(&st->tau);
        S.sigma = __ldcg(&st->sigma);
        S.isigma = 1.0 / __ldcg(&st->sigma);
        S.rho = a.rho;
        S.failed = 0;
        S.col.bar = unsigned(__cvta_generic_to_shared(&S.bar[0]));
        S.row.bar = unsigned(__cvta_generic_to_shared(&S.bar[1]));
        cl_bar_init(S.col.bar);
        cl_bar_init(S.row.bar);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < kClWeights; i += kClThreads) S.w[i] = cl_weights(double(k_base + i));

    // ---- this rank's part of both sides in shared memory:
    // x-bar slots | y slots | slices | own entries | push tables | matrix
    unsigned char* top = cl_smem;
    auto take = [&](size_t bytes) {
        unsigned char* p = top;
        top += (bytes + 15) & ~size_t(15);
        return p;
    };
    const int gx = a.col.ghost[inst], gy = a.row.ghost[inst];
    double* gxs = reinterpret_cast<double*>(take(8 * size_t(gx)));
    double* gys = reinterpret_cast<double*>(take(8 * size_t(gy)));
    const int xs = 0, ys = int(reinterpret_cast<unsigned char*>(gys) - cl_smem);
    for (int i = tid; i < gx; i += kClThreads) gxs[i] = 0.0;
    for (int i = tid; i < gy; i += kClThreads) gys[i] = 0.0;
    const int bi = inst * (C + 1) + int(rank), ri = inst * C + int(rank);
    auto slices = [&](const ClSide& s, ClRank<RES, TV>& R, double* gathered) {
        const int lo = s.sl_lo[ri], ns = s.sl_lo[ri + 1] - lo;
        int4* d = reinterpret_cast<int4*>(take(16 * size_t(ns)));
        cl_copy(d, s.slices + lo, size_t(ns));
        if (tid == 0) {
            R.n = s.bound[bi + 1] - s.bound[bi];
            R.ns = ns;
            R.sl = int(reinterpret_cast<unsigned char*>(d) - cl_smem);
            R.p0 = size_t(s.off[inst]) + size_t(s.bound[bi]);
            R.bytes = unsigned(s.bytes[ri]) + (rank == 0 ? unsigned(a.lost) : 0u);
            R.bulk = s.bulk[ri];
            R.seg_bytes = 8u * unsigned((R.n + 1) & ~1);
        }
        // where the ranks keep this side (an empty rank has no segment)
        const int rows = s.off[inst + 1] - s.off[inst], b0 = s.bound[bi];
        const unsigned short* slot = s.slot + size_t(C) * s.off[inst] + b0;
        const bool some = s.bound[bi + 1] > b0;
        const unsigned base = unsigned(__cvta_generic_to_shared(gathered));
        if (tid < C) {
            R.ghosts[tid] = cl_map(base, unsigned(tid));
            R.bars[tid] = cl_map(unsigned(__cvta_generic_to_shared(&S.bar[&R == &S.row ? 1 : 0])), unsigned(tid));
            R.dst[tid] = R.ghosts[tid] + (some ? 8u * slot[size_t(tid) * rows] : 0u);
            if (tid == int(rank))
                R.seg = int(reinterpret_cast<unsigned char*>(gathered) - cl_smem) + (some ? 8 * int(slot[size_t(tid) * rows]) : 0);
        }
    };
    slices(a.col, S.col, gxs);
    slices(a.row, S.row, gys);
    __syncthreads();
    auto own = [&](ClRank<RES, TV>& R, double* v, size_t stride, int k) {
        double* src = v + R.p0;
        double* d = src;
        int ds = int(stride);
        if (flags & kClOwnShared) {
            ds = R.n;
            d = reinterpret_cast<double*>(take(8 * size_t(R.n) * size_t(k)));
            for (int q = 0; q < k; ++q) cl_copy(d + size_t(q) * R.n, src + size_t(q) * stride, size_t(R.n));
        }
        if (tid == 0) {
            R.own.set(d, (flags & kClOwnShared) != 0);
            R.stride = ds;
        }
    };
    own(S.col, a.v.col, a.v.ncol, kClColVecs);
    own(S.row, a.v.row, a.v.nrow, kClRowVecs);
    auto push_tables = [&](ClRank<RES, TV>& R, const ClSide& s) {
        const int off = s.off[inst], rows = s.off[inst + 1] - off;
        const unsigned short* need = s.need + R.p0;
        const unsigned short* slot = s.slot + size_t(C) * off + s.bound[bi];
        int stride = rows;
        if (flags & kClPushShared) {
            unsigned short* d = reinterpret_cast<unsigned short*>(take(2 * size_t(R.n) * size_t(C + 1)));
            cl_copy(d, need, size_t(R.n));
            for (int r = 0; r < C; ++r) cl_copy(d + size_t(R.n) * (r + 1), slot + size_t(r) * rows, size_t(R.n));
            need = d;
            slot = d + R.n;
            stride = R.n;
        }
        if (tid == 0) {
            R.need.set(need, (flags & kClPushShared) != 0);
            R.slot.set(slot, (flags & kClPushShared) != 0);
            R.slot_stride = stride;
        }
    };
    push_tables(S.col, a.col);
    push_tables(S.row, a.row);
    auto matrix = [&](ClRank<RES, TV>& R, const ClSide& s) {
        const int base = s.base[ri], units = s.base[ri + 1] - base;
        const unsigned short* idx = s.idx + size_t(base) * kClUnit;
        const TV* val;
        if constexpr (sizeof(TV) == 4) val = s.v32 + size_t(base) * kClUnit;
        else val = s.v64 + size_t(base) * kClUnit;
        if (tid == 0) {
            R.idx_g.set(reinterpret_cast<const ushort2*>(idx), false);
            R.val64.set(reinterpret_cast<const double2*>(s.v64 + size_t(base) * kClUnit), false);
        }
        const bool sh = (flags & kClMatShared) != 0;
        if (sh) {
            void* di = take(2 * kClUnit * size_t(units));
            cl_copy16(di, idx, 2 * kClUnit * size_t(units));
            void* dv = take(sizeof(TV) * kClUnit * size_t(units));
            cl_copy16(dv, val, sizeof(TV) * kClUnit * size_t(units));
            idx = static_cast<const unsigned short*>(di);
            val = static_cast<const TV*>(dv);
        }
        if (tid == 0) {
            R.idx.set(reinterpret_cast<const ushort2*>(idx), sh);
            R.val.set(reinterpret_cast<const typename ClPair<TV>::type*>(val), sh);
        }
    };
    matrix(S.col, a.col);
    matrix(S.row, a.row);
    cl_sync();  // every rank's slots and barriers are ready before anyone sends
    for (int i = tid; i < S.row.n; i += kClThreads) cl_push(S.row, i, S.row.need[i], S.row.own[i], 0, 1, C);
    cl_flush(S.row);

    // ---- the iterations: phase `it` of the y barrier brings the y they start
    // from, phase `it` of the x barrier x-bar
    const int K = a.K;
    double sp[2] = {0.0, 0.0}, sd[2] = {0.0, 0.0};
    for (int it = 0; it < K; ++it) {
        const double2 w = it < kClWeights ? S.w[it] : cl_weights(double(k_base + it));
        const unsigned par = unsigned(it) & 1u;
        if (it < K - 1) cl_primal<RES, TV, false>(S, ys, par, nullptr, w, halpern, C, sp);
        else cl_primal<RES, TV, true>(S, ys, par, a.v.xp + S.col.p0, w, halpern, C, sp);
        if (it < K - 1) cl_dual<RES, TV, false>(S, xs, par, nullptr, w, halpern, C, sd);
        else cl_dual<RES, TV, true>(S, xs, par, a.v.yp + S.row.p0, w, halpern, C, sd);
        if (S.stop) break;
    }
    cl_check<RES, TV>(a, S, xs, ys, unsigned(K) & 1u, rank, inst, st, sp[0], sp[1], sd[0], sd[1]);

    // ---- the iterate (and after a restart the anchor) for the next chunk
    const bool restart = __ldcg(&st->apply_restart) && !__ldcg(&st->done);
    auto finish = [&](const ClRank<RES, TV>& R, double* v, size_t stride, const double* plus) {
        for (int j = tid; j < R.n; j += kClThreads) {
            double* g = v + R.p0 + j;
            if (restart) {
                g[0] = plus[j];
                g[stride] = plus[j];
            } else if (flags & kClOwnShared) {
                g[0] = R.own[j];
            }
        }
    };
    finish(S.col, a.v.col, a.v.ncol, a.v.xp + S.col.p0);
    finish(S.row, a.v.row, a.v.nrow, a.v.yp + S.row.p0);
}

// ---------------------------------------------------------------- plan

// need[p] = the ranks of the other side whose rows gather entry p: row
// order[p] of this side's matrix lists exactly them.
__global__ void k_cl_need(int rows, const int* __restrict__ order, const int* __restrict__ rp,
                          const int* __restrict__ ci, const unsigned char* __restrict__ rank_other,
                          unsigned short* __restrict__ need) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= rows) return;
    const int r = order[p];
    unsigned m = 0;
    for (int k = rp[r]; k < rp[r + 1]; ++k) m |= 1u << rank_other[ci[k]];
    need[p] = (unsigned short)m;
}

// Slots of one side for rank r = b % C of instance b / C.  The entries of a
// source rank s that r gathers are numbered in position order; where they
// are one in kClBulkPart of s's entries or more, and for s = r, all of s's
// entries get slots, from an even one on, so that one bulk copy brings them.  The
// first kClZeroSlots are nobody's.  ghost[b] is the number of slots, bytes[b]
// what a phase brings from other ranks;
// all[b] collects the sources taken whole (bit s).
__global__ void __launch_bounds__(kBlock) k_cl_slots(int C, const int* __restrict__ off, const int* __restrict__ bound,
                                                     const unsigned short* __restrict__ need,
                                                     unsigned short* __restrict__ slot, int* __restrict__ ghost,
                                                     int* __restrict__ bytes, unsigned short* __restrict__ all) {
    __shared__ int sh[kWarps];
    const int i = blockIdx.x / C, r = blockIdx.x % C;
    const int p0 = off[i], n = off[i + 1] - p0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned short* out = slot + size_t(C) * p0 + size_t(r) * n;
    int carry = kClZeroSlots, come = 0;
    unsigned whole = 0;
    for (int s = 0; s < C; ++s) {
        const int b0 = bound[i * (C + 1) + s], b1 = bound[i * (C + 1) + s + 1];
        int cnt = 0;
        for (int p = b0 + int(threadIdx.x); p < b1; p += kBlock) cnt += (need[p0 + p] >> r) & 1;
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0) sh[w] = cnt;
        __syncthreads();
        int total = 0;
        for (int k = 0; k < kWarps; ++k) total += sh[k];
        __syncthreads();
        if (b1 > b0 && (s == r || kClBulkPart * total >= b1 - b0)) {
            carry = (carry + 1) & ~1;
            for (int p = b0 + int(threadIdx.x); p < b1; p += kBlock) out[p] = (unsigned short)(carry + p - b0);
            carry += (b1 - b0 + 1) & ~1;
            if (s != r) {
                come += 8 * ((b1 - b0 + 1) & ~1);
                whole |= 1u << s;
            }
            continue;
        }
        for (int b = b0; b < b1; b += kBlock) {
            const int p = b + int(threadIdx.x);
            const bool in = p < b1 && ((need[p0 + p] >> r) & 1);
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (lane == 0) sh[w] = __popc(m);
            __syncthreads();
            int before = carry;
            for (int k = 0; k < kWarps; ++k) {
                if (k < w) before += sh[k];
                carry += sh[k];
            }
            if (p < b1) out[p] = in ? (unsigned short)(before + __popc(m & ((1u << lane) - 1))) : (unsigned short)0xffff;
            __syncthreads();
        }
        come += 8 * total;
    }
    if (threadIdx.x == 0) {
        ghost[blockIdx.x] = carry;
        bytes[blockIdx.x] = come;
        all[blockIdx.x] = (unsigned short)whole;
    }
}

// bulk[b] = the ranks that take all entries of rank b % C, and need without
// them and without the entry's own rank.
__global__ void k_cl_bulk(int count, int C, const unsigned short* __restrict__ all, unsigned short* __restrict__ bulk) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count * C) return;
    const int i = b / C, s = b % C;
    unsigned m = 0;
    for (int r = 0; r < C; ++r) m |= ((unsigned(all[i * C + r]) >> s) & 1u) << r;
    bulk[b] = (unsigned short)m;
}
__global__ void k_cl_single(int rows, int C, const int* __restrict__ order, const unsigned char* __restrict__ rank,
                            const int* __restrict__ inst_of, const unsigned short* __restrict__ bulk,
                            unsigned short* __restrict__ need) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= rows) return;
    const int r = order[p], i = inst_of ? inst_of[r] : 0, k = rank[r];
    need[p] = (unsigned short)(need[p] & ~(unsigned(bulk[i * C + k]) | (1u << k)));
}

// A slice's entry (lane, step) as its place in the CSR arrays, or -1 for padding.
__device__ __forceinline__ int cl_source(const int4 d, int lane, int step, int p_first, const int* __restrict__ order,
                                         const int* __restrict__ rp) {
    const int lt = d.z >> 24, rl = lane >> lt;
    if (rl >= d.w) return -1;
    const int r = order[p_first + d.x + rl];
    const int e = (lane & ((1 << lt) - 1)) + (step << lt);
    return e < rp[r + 1] - rp[r] ? rp[r] + e : -1;
}

// One warp per slice: the slots its entries gather (slot 0, which holds zero,
// in the padding, whose values are 0).
__global__ void k_cl_fill_idx(int ns, int C, const int4* __restrict__ slices, const int* __restrict__ owner,
                              ClSide side, ClSide other, const int* __restrict__ order, const int* __restrict__ rp,
                              const int* __restrict__ ci, const int* __restrict__ pos_other,
                              unsigned short* __restrict__ idx) {
    const int s = int((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (s >= ns) return;
    const int4 d = slices[s];
    const int b = owner[s], i = b / C, r = b % C;
    const int first = side.off[i] + side.bound[i * (C + 1) + r];
    const int ooff = other.off[i], orows = other.off[i + 1] - ooff;
    const unsigned short* sl = other.slot + size_t(C) * ooff + size_t(r) * orows;
    unsigned short* out = idx + (size_t(side.base[b]) + size_t(d.y)) * kClUnit;
    const int steps = 2 * (d.z & 0xffffff);
    for (int k = 0; k < steps; ++k) {
        const int src = cl_source(d, lane, k, first, order, rp);
        out[(k >> 1) * kClUnit + 2 * lane + (k & 1)] = src < 0 ? (unsigned short)0 : sl[pos_other[ci[src]] - ooff];
    }
}

__global__ void k_cl_fill_vals(int ns, int C, const int4* __restrict__ slices, const int* __restrict__ owner,
                               ClSide side, const int* __restrict__ order, const int* __restrict__ rp,
                               const double* __restrict__ s64, const float* __restrict__ s32,
                               double* __restrict__ v64, float* __restrict__ v32) {
    const int s = int((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (s >= ns) return;
    const int4 d = slices[s];
    const int b = owner[s], i = b / C, r = b % C;
    const int first = side.off[i] + side.bound[i * (C + 1) + r];
    const size_t at = (size_t(side.base[b]) + size_t(d.y)) * kClUnit;
    const int steps = 2 * (d.z & 0xffffff);
    for (int k = 0; k < steps; ++k) {
        const int src = cl_source(d, lane, k, first, order, rp);
        const size_t o = at + (k >> 1) * kClUnit + 2 * lane + (k & 1);
        v64[o] = src < 0 ? 0.0 : s64[src];
        v32[o] = src < 0 ? 0.0f : s32[src];
    }
}

// out_k[p] = in_k[order[p]] for up to eight vectors of one side.
struct ClMove {
    const double* in[8];
    double* out[8];
};

__global__ void k_cl_gather(int rows, int nv, const int* __restrict__ order, ClMove mv) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= rows) return;
    const int r = order[p];
    for (int k = 0; k < nv; ++k) mv.out[k][p] = mv.in[k][r];
}

// out[order[p]] = in[p] for the instances the clusters solved (member null: all).
__global__ void k_cl_scatter(int rows, const int* __restrict__ order, const int* __restrict__ inst_of,
                             const unsigned char* __restrict__ member, const double* __restrict__ in,
                             double* __restrict__ out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= rows) return;
    const int r = order[p];
    if (member && !member[inst_of[r]]) return;
    out[r] = in[p];
}

}  // namespace nir
