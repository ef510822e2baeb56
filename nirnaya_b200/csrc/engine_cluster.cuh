// Host side of the cluster path (k_cluster.cuh): plans, their buffers, the
// choice of the cluster size, and the launches.  Included by engine.cu
// before the solves that use it.
#pragma once

// A plan of one handle for clusters of C CTAs: one LP, or the instances of a
// batch.  It depends on the matrix structure only; the values and vectors
// are moved into its order by every solve.
struct ClusterPlan {
    int C = 0, count = 0;
    struct Side {
        nir::ClHostSide h;
        int rows = 0;
        int *order = nullptr, *pos = nullptr, *bound = nullptr, *sl_lo = nullptr, *base = nullptr, *owner = nullptr;
        int4* slices = nullptr;
        unsigned char* rank = nullptr;
        unsigned short *idx = nullptr, *need = nullptr, *slot = nullptr;
        float* v32 = nullptr;
        double* v64 = nullptr;
        int *ghost = nullptr, *ghost_rank = nullptr, *bytes = nullptr;
        unsigned short *all = nullptr, *bulk = nullptr;
        std::vector<int> ghosts;  // [i]: largest rank
        std::vector<int> come;    // [i C + r]: bytes a phase brings from other ranks
        double* vec = nullptr;    // the side's vectors in the plan's order, `rows` entries each:
                                  // col x x0 c lo up xp dc oc ol ou, row y y0 rl ru yp dr orl oru
        double* v(int k) const { return vec + size_t(k) * size_t(rows); }
    } row, col;
    const int *d_row_off = nullptr, *d_col_off = nullptr;  // instance offsets on the device
    std::vector<int> row_off, col_off;
    std::vector<unsigned char> member;  // [i]: solved by a cluster
    int members = 0;
    unsigned char* d_member = nullptr;
    int* d_list = nullptr;
    int* d_flags[2] = {};   // kCl*Shared per instance, for FP32 and FP64 values
    size_t smem[2] = {};    // dynamic shared memory of a launch
    bool resident[2] = {true, true};  // every member has all of it in shared memory
    long long values_of = -1;  // the scaling whose values the streams hold
    DevArena mem;
    ~ClusterPlan() { mem.clear(); }
};

namespace {

static_assert(nir::kClPlanWarps == nir::kClWarps, "the plan deals slices to the kernel's warps");

// Dynamic shared memory a CTA may use: 227 KB less the static sums.
constexpr size_t kClSmemMax = 220 * 1024;

template <typename T>
T* cl_alloc(ClusterPlan& P, size_t count) {
    return static_cast<T*>(P.mem.alloc(count * sizeof(T)));
}

template <typename T>
T* cl_upload(nir_pdhg* h, ClusterPlan& P, const std::vector<T>& v) {
    T* p = cl_alloc<T>(P, v.size());
    if (!v.empty()) NIR_CUDA(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, h->stream));
    return p;
}

// What the kernel sees of one side.
nir::ClSide cl_side(const ClusterPlan::Side& s, const int* off) {
    return nir::ClSide{off,   s.bound, s.sl_lo, s.slices, s.base, s.idx, s.v32, s.v64, s.need, s.slot, s.ghost, s.bytes, s.bulk};
}

// Shared memory of instance i for values of `vb` bytes, in the kernel's
// order, taking what fits; the flags say what was taken.  0 when the
// gathered entries and the slices alone do not fit, or a slot number does
// not fit 16 bits.
size_t cl_instance_smem(const ClusterPlan& P, int i, int vb, int* flags) {
    const int C = P.C;
    auto up16 = [](size_t b) { return (b + 15) & ~size_t(15); };
    const size_t gx = size_t(P.col.ghosts[size_t(i)]), gy = size_t(P.row.ghosts[size_t(i)]);
    if (gx > 0xffff || gy > 0xffff) return 0;
    size_t base = 0, own = 0, push = 0, mat = 0;
    for (int r = 0; r < C; ++r) {
        size_t b = up16(8 * gx) + up16(8 * gy), o = 0, p = 0, m = 0;
        for (const ClusterPlan::Side* s : {&P.col, &P.row}) {
            const size_t k = size_t(i) * C + r, kb = size_t(i) * (C + 1) + r;
            const size_t n = size_t(s->h.bound[kb + 1] - s->h.bound[kb]);
            const size_t units = size_t(s->h.base[k + 1] - s->h.base[k]);
            b += 16 * size_t(s->h.sl_lo[k + 1] - s->h.sl_lo[k]);
            o += up16(8 * n * size_t(s == &P.col ? nir::kClColVecs : nir::kClRowVecs));
            p += up16(2 * n * size_t(C + 1));
            m += units * nir::kClUnit * size_t(2 + vb);
        }
        base = std::max(base, b);
        own = std::max(own, o);
        push = std::max(push, p);
        mat = std::max(mat, m);
    }
    if (base > kClSmemMax) return 0;
    *flags = 0;
    size_t s = base;
    const std::pair<int, size_t> parts[3] = {{nir::kClOwnShared, own}, {nir::kClPushShared, push}, {nir::kClMatShared, mat}};
    for (auto& q : parts)
        if (s + q.second <= kClSmemMax) {
            s += q.second;
            *flags |= q.first;
        }
    return std::max<size_t>(s, 16);
}

// Builds the plan for clusters of C CTAs on the handle's matrix; instance i
// owns rows [row_off[i], row_off[i+1]) and columns likewise (the offsets are
// on the device too, as the instance of every row and column; null for one).
// Null when no instance fits.
std::unique_ptr<ClusterPlan> cl_build(nir_pdhg* h, int C, const std::vector<int>& row_off,
                                      const std::vector<int>& col_off, const int* d_row_off, const int* d_col_off,
                                      const int* d_row_inst, const int* d_col_inst) {
    auto up = std::make_unique<ClusterPlan>();
    ClusterPlan& P = *up;
    cudaStream_t s = h->stream;
    P.C = C;
    P.count = int(row_off.size()) - 1;
    P.row_off = row_off;
    P.col_off = col_off;
    P.d_row_off = d_row_off;
    P.d_col_off = d_col_off;
    {
        size_t total = 0;
        for (ClusterPlan::Side* t : {&P.row, &P.col}) {
            const bool is_row = t == &P.row;
            const Orient& o = is_row ? h->A : h->At;
            t->rows = o.rows;
            nir::cl_build_side(is_row ? row_off : col_off, o.h_rp, C, t->h);
            total += size_t(o.rows) * size_t(4 + 4 + 1 + 2 + 2 * C) + t->h.slices.size() * 20 + size_t(P.count) * C * 40;
        }
        P.mem.reserve(total + 64 * DevArena::kAlign);
        for (ClusterPlan::Side* t : {&P.row, &P.col}) {
            const bool is_row = t == &P.row;
            const Orient& o = is_row ? h->A : h->At;
            t->order = cl_upload(h, P, t->h.order);
            t->pos = cl_upload(h, P, t->h.pos);
            t->rank = cl_upload(h, P, t->h.rank);
            t->bound = cl_upload(h, P, t->h.bound);
            t->sl_lo = cl_upload(h, P, t->h.sl_lo);
            t->base = cl_upload(h, P, t->h.base);
            t->slices = cl_upload(h, P, t->h.slices);
            t->owner = cl_upload(h, P, t->h.owner);
            t->need = cl_alloc<unsigned short>(P, size_t(o.rows));
            t->slot = cl_alloc<unsigned short>(P, size_t(o.rows) * C);
            t->ghost_rank = cl_alloc<int>(P, size_t(P.count) * C);
            t->bytes = cl_alloc<int>(P, size_t(P.count) * C);
            t->all = cl_alloc<unsigned short>(P, size_t(P.count) * C);
            t->bulk = cl_alloc<unsigned short>(P, size_t(P.count) * C);
        }
        std::vector<int> gr(size_t(P.count) * C);
        for (ClusterPlan::Side* t : {&P.row, &P.col}) {
            const bool is_row = t == &P.row;
            const Orient& o = is_row ? h->A : h->At;
            // entry p of y is gathered by the ranks of the columns in row p, and x-bar by those of the rows
            const ClusterPlan::Side& other = is_row ? P.col : P.row;
            nir::k_cl_need<<<grid_for(o.rows), nir::kBlock, 0, s>>>(o.rows, t->order, o.rp, o.ci, other.rank, t->need);
            nir::k_cl_slots<<<P.count * C, nir::kBlock, 0, s>>>(C, is_row ? d_row_off : d_col_off, t->bound, t->need,
                                                                t->slot, t->ghost_rank, t->bytes, t->all);
            nir::k_cl_bulk<<<grid_for(P.count * (long long)C), nir::kBlock, 0, s>>>(P.count, C, t->all, t->bulk);
            nir::k_cl_single<<<grid_for(o.rows), nir::kBlock, 0, s>>>(o.rows, C, t->order, t->rank,
                                                                      is_row ? d_row_inst : d_col_inst, t->bulk, t->need);
            NIR_LAUNCHED();
            d2h(h, gr.data(), t->ghost_rank, gr.size() * sizeof(int));
            t->come.resize(gr.size());
            d2h(h, t->come.data(), t->bytes, t->come.size() * sizeof(int));
            t->ghosts.assign(size_t(P.count), nir::kClZeroSlots);  // the padding's index
            for (int i = 0; i < P.count; ++i)
                for (int r = 0; r < C; ++r) t->ghosts[size_t(i)] = std::max(t->ghosts[size_t(i)], gr[size_t(i) * C + r]);
            t->ghost = cl_upload(h, P, t->ghosts);
        }
        // the instances that fit, by falling work
        P.member.assign(size_t(P.count), 0);
        std::vector<int> list, flags[2];
        for (int q = 0; q < 2; ++q) flags[q].assign(size_t(P.count), 0);
        for (int i = 0; i < P.count; ++i) {
            size_t b[2];
            for (int q = 0; q < 2; ++q) b[q] = cl_instance_smem(P, i, q ? 8 : 4, &flags[q][size_t(i)]);
            if (!b[0] || !b[1]) continue;
            P.member[size_t(i)] = 1;
            for (int q = 0; q < 2; ++q) {
                P.smem[q] = std::max(P.smem[q], b[q]);
                P.resident[q] = P.resident[q] && flags[q][size_t(i)] ==
                                                     (nir::kClOwnShared | nir::kClPushShared | nir::kClMatShared);
            }
            list.push_back(i);
        }
        auto nnz_of = [&](int i) { return h->A.h_rp[size_t(row_off[size_t(i) + 1])] - h->A.h_rp[size_t(row_off[size_t(i)])]; };
        std::stable_sort(list.begin(), list.end(), [&](int a, int b) { return nnz_of(a) > nnz_of(b); });
        P.members = int(list.size());
        if (P.members == 0) {
            NIR_CUDA(cudaStreamSynchronize(s));
            return nullptr;
        }
        P.d_list = cl_upload(h, P, list);
        P.d_member = cl_upload(h, P, P.member);
        for (int q = 0; q < 2; ++q) P.d_flags[q] = cl_upload(h, P, flags[q]);
        size_t streams = 0;
        for (ClusterPlan::Side* t : {&P.row, &P.col})
            streams += size_t(t->h.base.back()) * nir::kClUnit * 14 + size_t(t->rows) * 80 + 4 * DevArena::kAlign;
        P.mem.reserve(streams);
        for (ClusterPlan::Side* t : {&P.row, &P.col}) {
            const size_t e = size_t(t->h.base.back()) * nir::kClUnit;
            t->idx = cl_alloc<unsigned short>(P, e);
            t->v32 = cl_alloc<float>(P, e);
            t->v64 = cl_alloc<double>(P, e);
            t->vec = cl_alloc<double>(P, size_t(t->rows) * 10);
        }
        for (int t = 0; t < 2; ++t) {
            const Orient& o = t ? h->At : h->A;
            ClusterPlan::Side& me = t ? P.col : P.row;
            ClusterPlan::Side& ot = t ? P.row : P.col;
            const int ns = int(me.h.slices.size());
            nir::k_cl_fill_idx<<<grid_for(ns * 32LL), nir::kBlock, 0, s>>>(
                ns, C, me.slices, me.owner, cl_side(me, t ? d_col_off : d_row_off),
                cl_side(ot, t ? d_row_off : d_col_off), me.order, o.rp, o.ci, ot.pos, me.idx);
            NIR_LAUNCHED();
        }
        NIR_CUDA(cudaStreamSynchronize(s));  // the uploads read the vectors above
    }
    return up;
}

// The scaled values (after a preconditioning), once per scaling, and the
// vectors, iterate and anchor of this solve, in the plan's order.
void cl_load(nir_pdhg* h, ClusterPlan& P) {
    cudaStream_t s = h->stream;
    if (P.values_of != h->scaled.version) {
        for (int t = 0; t < 2; ++t) {
            const Orient& o = t ? h->At : h->A;
            ClusterPlan::Side& me = t ? P.col : P.row;
            const int ns = int(me.h.slices.size());
            nir::k_cl_fill_vals<<<grid_for(ns * 32LL), nir::kBlock, 0, s>>>(
                ns, P.C, me.slices, me.owner, cl_side(me, t ? P.d_col_off : P.d_row_off), me.order, o.rp, o.v64, o.v32,
                me.v64, me.v32);
            NIR_LAUNCHED();
        }
        P.values_of = h->scaled.version;
        h->launches += 2;
    }
    auto move = [&](ClusterPlan::Side& t, std::initializer_list<std::pair<const double*, int>> what) {
        nir::ClMove mv{};
        int k = 0;
        for (auto& w : what) {
            mv.in[k] = w.first;
            mv.out[k] = t.v(w.second);
            ++k;
        }
        nir::k_cl_gather<<<grid_for(t.rows), nir::kBlock, 0, s>>>(t.rows, k, t.order, mv);
        NIR_LAUNCHED();
        h->launches += 1;
    };
    move(P.col, {{h->x64, 0}, {h->x064, 1}, {h->c64, 2}, {h->l64, 3}, {h->u64, 4}, {h->dc, 6}});
    move(P.col, {{h->c, 7}, {h->l, 8}, {h->u, 9}});
    move(P.row, {{h->y64, 0}, {h->y064, 1}, {h->rl64, 2}, {h->ru64, 3}, {h->dr, 5}, {h->rl, 6}, {h->ru, 7}});
}

// x+ and y+ back into the handle's order.
void cl_store_out(nir_pdhg* h, ClusterPlan& P, const int* col_inst, const int* row_inst) {
    const unsigned char* mem = col_inst ? P.d_member : nullptr;
    nir::k_cl_scatter<<<grid_for(P.col.rows), nir::kBlock, 0, h->stream>>>(P.col.rows, P.col.order, col_inst, mem,
                                                                          P.col.v(5), h->xp64);
    nir::k_cl_scatter<<<grid_for(P.row.rows), nir::kBlock, 0, h->stream>>>(P.row.rows, P.row.order, row_inst, mem,
                                                                          P.row.v(4), h->yp64);
    NIR_LAUNCHED();
    h->launches += 2;
}

// Once per kernel and device, before any capture.
template <bool RES, typename TV>
void cl_prepare_kernel() {
    auto* k = nir::k_cluster_chunk<RES, TV>;
    NIR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kClSmemMax)));
    NIR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

// One chunk of every instance the plan solves.  st: the states, one per
// instance; the norms and offsets by instance, or null for one LP.
template <typename TV>
void cl_launch(nir_pdhg* h, ClusterPlan& P, const nir::CtlArgs& ctl, int K, int halpern, int phase, double rho,
               nir::DevState* st, const double* bnorm, const double* cnorm, const double* offset, bool wait_test) {
    const int q = sizeof(TV) == 8 ? 1 : 0;
    nir::ClArgs a{};
    a.col = cl_side(P.col, P.d_col_off);
    a.row = cl_side(P.row, P.d_row_off);
    const ClusterPlan::Side &c = P.col, &r = P.row;
    a.v = nir::ClVecs{c.vec,  r.vec,  size_t(c.rows), size_t(r.rows), c.v(5), r.v(4), c.v(6),
                      c.v(7), c.v(8), c.v(9),         r.v(5),         r.v(6), r.v(7)};
    a.list = P.d_list;
    a.flags = P.d_flags[q];
    a.C = P.C;
    a.K = K;
    a.halpern = halpern;
    a.phase = phase;
    a.rho = rho;
    a.st = st;
    a.bnorm = bnorm;
    a.cnorm = cnorm;
    a.offset = offset;
    a.lost = wait_test ? 8 : 0;
    a.ctl = ctl;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(P.members) * unsigned(P.C));
    cfg.blockDim = dim3(nir::kClThreads);
    cfg.dynamicSmemBytes = P.smem[q];
    cfg.stream = h->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = unsigned(P.C);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    NIR_CUDA(cudaLaunchKernelEx(&cfg, P.resident[q] ? nir::k_cluster_chunk<true, TV> : nir::k_cluster_chunk<false, TV>, a));
    NIR_LAUNCHED();
    h->launches += 1;
}

// Clusters of C CTAs the device holds at once with all the dynamic shared
// memory a plan may use (after cl_prepare_kernels; the kernels' registers and
// static memory are alike): 0 where a GPC has fewer than C SMs for the process.
int cl_resident(int C) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(C) * 148u);
    cfg.blockDim = dim3(nir::kClThreads);
    cfg.dynamicSmemBytes = kClSmemMax;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = unsigned(C);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, nir::k_cluster_chunk<false, float>, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}

// nir_pdhg_params.persistent: clusters, one of whose waits cannot end.
constexpr int kClWaitTest = 3;

// The solves a cluster can run: the default iteration in FP64 arithmetic.
// A caller that fixes a layout, asks for the persistent kernel, for FP32
// iterates, for single launches or their timing, or for a fresh FP64 phase
// gets the per-launch kernels.
bool cl_takes(const nir_pdhg* h, const nir_pdhg_params& p) {
    return p.spmv_block_nnz == 0 && (p.persistent == 0 || p.persistent == kClWaitTest) && p.use_graphs && !h->profiling &&
           p.precision != NIR_PREC_FP32 && (p.precision == NIR_PREC_FP64 || p.polish_fresh == 2);
}

// NIR_PDHG_CLUSTER in the environment: the cluster size (1, 2, 4, 8, 16), 0
// for never; -1 when unset.
int cl_forced() {
    const char* e = std::getenv("NIR_PDHG_CLUSTER");
    if (!e) return -1;
    const int v = std::atoi(e);
    return (v == 1 || v == 2 || v == 4 || v == 8 || v == 16) ? v : 0;
}

// What an iteration costs, in microseconds, as measured on B200 for LPs of
// 1,200 to 500,000 nonzeros on clusters of 1 to 16: the latency of two
// passes, the gathers of an SM (0.35 per 1,000 nonzeros, and more the more
// ranks wait for the slowest) and the entries that come from other ranks
// (0.6 for 6,500 on the 2,000 x 5,000 LP, 1.9 for 9,800, 3.9 for 16,400).
// Against it the two launches of the per-launch kernels while the LP lies
// in L2.
double cl_time(double nnz, double entries, int C) {
    const double per = 0.35 + 0.04 * std::log2(double(C)), k = 1e-3 * entries;
    return (C >= 16 ? 2.9 : 2.4) + 1e-3 * per * nnz / C + (C > 1 ? k * (0.04 + 0.0125 * k) : 0.0);
}
double cl_launch_time(double nnz) { return 5.3 + 7e-6 * nnz; }
// Clusters must be this much faster by the estimate.
constexpr double kClMargin = 0.95;

void cl_prepare_kernels() {
    cl_prepare_kernel<false, float>();
    cl_prepare_kernel<false, double>();
    cl_prepare_kernel<true, float>();
    cl_prepare_kernel<true, double>();
}

// Entries a phase pair brings instance i's busiest rank from other ranks.
double cl_arrivals(const ClusterPlan& P, int i) {
    int mx = 0;
    for (int r = 0; r < P.C; ++r) {
        const size_t k = size_t(i) * P.C + r;
        mx = std::max(mx, P.col.come[k] + P.row.come[k]);
    }
    return mx / 8.0;
}

// The plan a single LP's solve runs on, or null for the per-launch kernels.
// The cluster is as large as shortens an iteration: 16 CTAs, fewer on an LP
// whose rows do not fill them or where the device holds none of 16.  Built
// where clusters are faster even with nothing to exchange (below about
// 85,000 nonzeros), kept where they still are with what the plan exchanges:
// 2.5 against 4.3 us an iteration on a 60 x 150 LP, 4.6 against 5.9 on a
// random 2,000 x 5,000 one of 40,000 nonzeros, 3.4 against 4.4 on a
// multiperiod one of 15,000, but 6.0 against 5.6 on one of 126,000 and 9.5
// against 5.6 on a blending LP of 100,000 whose ranks need nearly all
// entries.
ClusterPlan* cl_single(nir_pdhg* h, const nir_pdhg_params& p) {
    if (!cl_takes(h, p) || h->m < 1 || h->n < 1) return nullptr;
    if (h->cluster_size < 0) {
        h->cluster_size = 0;
        const int f = cl_forced();
        const double nnz = double(h->nnz);
        int C = f >= 0 ? f : (nnz < 3000 ? 4 : (nnz < 10000 ? 8 : 16));
        if (f < 0 && cl_time(nnz, 0.0, C) >= kClMargin * cl_launch_time(nnz)) C = 0;
        if (C > 0) {
            cl_prepare_kernels();
            const int held = nir::cl_size_held(C, cl_resident);
            // a size that the caller fixed is not replaced
            const bool ok = held == C || (f < 0 && held > 0 && cl_time(nnz, 0.0, held) < kClMargin * cl_launch_time(nnz));
            C = ok ? held : 0;
        }
        if (C > 0) {
            one_instance(h);
            std::unique_ptr<ClusterPlan> P = nir::cl_if_memory(
                [&] { return cl_build(h, C, {0, h->m}, {0, h->n}, h->one_row, h->one_col, nullptr, nullptr); });
            if (P && (f >= 0 || cl_time(nnz, cl_arrivals(*P, 0), C) < kClMargin * cl_launch_time(nnz))) {
                h->cluster = std::move(P);
                h->cluster_size = C;
            }
        }
    }
    return h->cluster.get();
}

// The plan a batch runs on, or null: the cluster size with the shortest
// iteration of the whole batch by the times above, the instances dealt to
// as many clusters as the device holds; the next larger one while an
// instance does not fit, or there is no memory for the plan.  A plan may
// leave out instances that fit no cluster; the per-launch kernels then run
// those.
std::unique_ptr<ClusterPlan> cl_batch(nir_pdhg* h, const std::vector<int>& row_off, const std::vector<int>& col_off,
                                      const int* d_row_off, const int* d_col_off, const int* d_row_inst,
                                      const int* d_col_inst) {
    const int f = cl_forced(), count = int(row_off.size()) - 1;
    if (f == 0 || h->m < 1 || h->n < 1) return nullptr;
    cl_prepare_kernels();
    const int sizes[5] = {1, 2, 4, 8, 16};
    int first = 0;
    if (f > 0) {
        while (sizes[first] != f) ++first;
    } else {
        double best = 1e300;
        for (int k = 0; k < 5; ++k) {
            const int slots = cl_resident(sizes[k]);
            if (slots < 1) continue;
            double sum = 0.0, mx = 0.0;
            for (int i = 0; i < count; ++i) {
                const double nnz = double(h->A.h_rp[size_t(row_off[size_t(i) + 1])] - h->A.h_rp[size_t(row_off[size_t(i)])]);
                const double entries = double(row_off[size_t(i) + 1] - row_off[size_t(i)]) +
                                       double(col_off[size_t(i) + 1] - col_off[size_t(i)]);
                const double t = cl_time(nnz, 0.5 * entries, sizes[k]);
                sum += t;
                mx = std::max(mx, t);
            }
            const double t = sum / slots + 0.5 * mx;
            if (t < best) {
                best = t;
                first = k;
            }
        }
    }
    std::unique_ptr<ClusterPlan> best;
    for (int k = first; k < 5; ++k) {
        std::unique_ptr<ClusterPlan> P;
        if (cl_resident(sizes[k]) > 0)
            P = nir::cl_if_memory([&] {
                return cl_build(h, sizes[k], row_off, col_off, d_row_off, d_col_off, d_row_inst, d_col_inst);
            });
        if (P && (!best || P->members > best->members)) best = std::move(P);
        if (f > 0 || (best && best->members == count)) break;
    }
    return best;
}

void launch_cluster_chunk(nir_pdhg* h, ClusterPlan& P, const SolveCfg& cfg, int phase, bool fp64_values) {
    nir::CtlArgs ca = control_args(cfg, phase, h->hist);
    ca.offset = h->offset;
    if (fp64_values)
        cl_launch<double>(h, P, ca, cfg.K, cfg.halpern, phase, cfg.p.reflection, h->st, nullptr, nullptr, nullptr,
                          cfg.barrier_test != 0);
    else
        cl_launch<float>(h, P, ca, cfg.K, cfg.halpern, phase, cfg.p.reflection, h->st, nullptr, nullptr, nullptr,
                         cfg.barrier_test != 0);
    nir::k_snap<<<1, 32, 0, h->stream>>>(h->st, h->snap.ring, h->snap.d_seq);
    NIR_LAUNCHED();
    h->launches += 1;
}

}  // namespace
