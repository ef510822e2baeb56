// Kernels of NIR_ALGO_REFERENCE: the reference PDHG loop
// (src/gpu/pdhg_solver.hpp:33-105) in FP64 with the reference's exact
// arithmetic.  Every sum runs in the reference's order on one thread
// (CscMatrix::spmv adds a row's terms in ascending column order, the
// transpose adds a column's terms in ascending row order,
// src/core/csc_matrix.hpp:99-120), and every product and sum is a separate
// correctly rounded operation (__dmul_rn/__dadd_rn: no contraction into
// FMA, as the reference is compiled without it).  The results are
// bit-identical to the reference's.
#pragma once

#include "dev_common.cuh"
#include "row_blocks.hpp"

namespace nir {

// y[r] = sum_k v[k] * x[ci[k]] over row r, sequentially from +0.0.
__global__ void k_ref_spmv(int rows, const int* __restrict__ rp, const int* __restrict__ ci,
                           const double* __restrict__ v, const double* __restrict__ x, double* __restrict__ y) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    double s = 0.0;
    for (int k = rp[r]; k < rp[r + 1]; ++k) s = __dadd_rn(s, __dmul_rn(v[k], x[ci[k]]));
    y[r] = s;
}

// Power-iteration norm, src/gpu/pdhg_solver.hpp:38-41: u_j^2 added in index
// order, then norm_est = sqrt(max(1e-12, n2)).  One CTA: the sum is one
// chain, so one thread carries it and the other warps keep the squares ready
// in shared memory, a tile ahead (5,000 terms: 195 us with the loads on the
// chain, 40 without).
constexpr int kRefTile = kBlock - 32;
__global__ void __launch_bounds__(kBlock) k_ref_norm(int n, const double* __restrict__ u, DevState* st) {
    __shared__ double sq[2][kRefTile];
    if (blockIdx.x != 0) return;
    auto fill = [&](int base, int b) {
        const int k = int(threadIdx.x) - 32;
        if (k < 0) return;
        const double v = base + k < n ? u[base + k] : 0.0;
        sq[b][k] = __dmul_rn(v, v);
    };
    double n2 = 0.0;
    fill(0, 0);
    __syncthreads();
    for (int base = 0, t = 0; base < n; base += kRefTile, ++t) {
        const int b = t & 1;
        if (base + kRefTile < n) fill(base + kRefTile, b ^ 1);
        if (threadIdx.x == 0) {
            // n2 >= 0, so the zeros past the end change nothing
#pragma unroll 8
            for (int k = 0; k < kRefTile; ++k) n2 = __dadd_rn(n2, sq[b][k]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) st->ref_norm_est = __dsqrt_rn(smax(1e-12, n2));
}

__global__ void k_ref_div(int n, double* __restrict__ u, const DevState* __restrict__ st) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) u[j] = __ddiv_rn(u[j], st->ref_norm_est);
}

// Fixed steps, src/gpu/pdhg_solver.hpp:43-45.
__global__ void k_ref_steps(DevState* st) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    double sigma_max = __dsqrt_rn(st->ref_norm_est);
    double s = __ddiv_rn(0.85, smax(1e-6, sigma_max));
    st->tau = s;
    st->sigma = s;
}

// Box-midpoint start, src/gpu/pdhg_solver.hpp:47-57.
__global__ void k_ref_init(int n, int m, const double* __restrict__ lo, const double* __restrict__ up,
                           double* __restrict__ x, double* __restrict__ y) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        double l = lo[t], u = up[t], v = 0.0;
        if (fin_bound(l) && fin_bound(u)) v = __dmul_rn(0.5, __dadd_rn(l, u));
        else if (fin_bound(l)) v = smax(0.0, l);
        else if (fin_bound(u)) v = smin(0.0, u);
        x[t] = v;
    }
    if (t < m) y[t] = 0.0;
}

// Primal step, src/gpu/pdhg_solver.hpp:69-78, one thread per column j
// (row j of the stored transpose).
__global__ void k_ref_primal(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                             const double* __restrict__ v, const double* __restrict__ y,
                             const double* __restrict__ cost, const double* __restrict__ lo,
                             const double* __restrict__ up, double* __restrict__ x, double* __restrict__ xbar,
                             const DevState* __restrict__ st, int i_in_chunk) {
    if (st->done || st->iter + i_in_chunk >= st->max_iters) return;
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double s = 0.0;
    for (int k = rp[j]; k < rp[j + 1]; ++k) s = __dadd_rn(s, __dmul_rn(v[k], y[ci[k]]));
    const double tau = st->tau;
    double xj = x[j];
    double cand = __dsub_rn(xj, __dmul_rn(tau, __dsub_rn(cost[j], s)));
    if (fin_bound(lo[j])) cand = smax(lo[j], cand);
    if (fin_bound(up[j])) cand = smin(up[j], cand);
    xbar[j] = __dsub_rn(__dmul_rn(2.0, cand), xj);
    x[j] = cand;
}

// Dual step and the row-violation maximum, src/gpu/pdhg_solver.hpp:80-95,
// one thread per row.  Each block writes its violation maximum to part[].
__global__ void k_ref_dual(int m, const int* __restrict__ rp, const int* __restrict__ ci,
                           const double* __restrict__ v, const double* __restrict__ xbar,
                           const double* __restrict__ rlo, const double* __restrict__ rup, double* __restrict__ y,
                           double* __restrict__ part, const DevState* __restrict__ st, int i_in_chunk) {
    __shared__ double sh[kWarps];
    if (st->done || st->iter + i_in_chunk >= st->max_iters) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double viol = 0.0;
    if (i < m) {
        double a = 0.0;
        for (int k = rp[i]; k < rp[i + 1]; ++k) a = __dadd_rn(a, __dmul_rn(v[k], xbar[ci[k]]));
        const double sigma = st->sigma;
        double yi = y[i];
        double r = __dsub_rn(a, __ddiv_rn(yi, sigma));
        double lo = rlo[i], hi = rup[i];
        if (fin_bound(lo)) r = smax(lo, r);
        if (fin_bound(hi)) r = smin(hi, r);
        y[i] = __dadd_rn(yi, __dmul_rn(sigma, __dsub_rn(r, a)));
        if (fin_bound(lo)) viol = smax(viol, __dsub_rn(lo, a));
        if (fin_bound(hi)) viol = smax(viol, __dsub_rn(a, hi));
    }
    // max is order-independent, so the tree gives the reference's value
    double bm = block_max(viol, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bm;
}

// ---- the same steps over warp row blocks (row_blocks.hpp)
//
// With a thread per row a warp's loads of 32 rows scatter over as many cache
// lines, and every term waits for its loads.  Over row blocks a warp reads
// the block's entries with consecutive lanes, gathers and multiplies them
// all at once, and leaves the rounded products in shared memory; each row's
// products are then added in their order by the row's own lane.  The bits
// are the same; only the additions are left on the chain.  A row longer than
// the block capacity is added by one lane, 256 products at a time.

// One warp's block: fin(row, sum) on the row's lane.
template <class Fin>
__device__ __forceinline__ void ref_block(int2 d0, int2 d1, int cap, const int* __restrict__ rp,
                                          const int* __restrict__ ci, const double* __restrict__ val,
                                          const double* __restrict__ x, double* s_prod, Fin fin) {
    const int lane = threadIdx.x & 31;
    const int r0 = d0.x, p0 = d0.y, nrows = d1.x - d0.x, nnzb = d1.y - d0.y;
    const int r = r0 + lane;
    int ra = 0, re = 0;
    if (nnzb <= cap && lane < nrows) {
        ra = max(__ldg(rp + r) - p0, 0);
        re = min(__ldg(rp + r + 1) - p0, nnzb);
    }
    double s = 0.0;
    for (int base = 0; base < nnzb; base += kWarpCapMax) {
        int c[kWarpU];
        double v[kWarpU];
#pragma unroll
        for (int q = 0; q < kWarpU; ++q) {
            const int k = base + lane + 32 * q;
            c[q] = k < nnzb ? __ldg(ci + p0 + k) : 0;
            v[q] = k < nnzb ? __ldg(val + p0 + k) : 0.0;
        }
        if (base == 0) pdl_wait();
#pragma unroll
        for (int q = 0; q < kWarpU; ++q) {
            const int k = base + lane + 32 * q;
            if (k < nnzb) s_prod[lane + 32 * q] = __dmul_rn(v[q], __ldca(x + c[q]));
        }
        __syncwarp();
        if (nnzb <= cap) {
            for (int k = ra; k < re; ++k) s = __dadd_rn(s, s_prod[k]);
        } else if (lane == 0) {
            const int n = min(kWarpCapMax, nnzb - base);
#pragma unroll 4
            for (int k = 0; k < n; ++k) s = __dadd_rn(s, s_prod[k]);
        }
        __syncwarp();
    }
    if (nnzb == 0) pdl_wait();
    if (lane < nrows) fin(r, s);
}

__device__ __forceinline__ bool ref_over(const DevState* st, int i_in_chunk) {
    return st->done || st->iter + i_in_chunk >= st->max_iters;
}

// Primal step, src/gpu/pdhg_solver.hpp:69-78.
__global__ void __launch_bounds__(kBlock) k_refb_primal(const int2* __restrict__ blk, int nblk, int cap,
                                                        const int* __restrict__ rp, const int* __restrict__ ci,
                                                        const double* __restrict__ v, const double* __restrict__ y,
                                                        const double* __restrict__ cost, const double* __restrict__ lo,
                                                        const double* __restrict__ up, double* __restrict__ x,
                                                        double* __restrict__ xbar, const DevState* __restrict__ st,
                                                        int i_in_chunk) {
    __shared__ double prod[kWarps][kWarpCapMax];
    pdl_release();
    const int w = threadIdx.x >> 5, b = blockIdx.x * kWarps + w;
    // the first kernel of a chunk is launched after the one that wrote the state
    if (b >= nblk || ref_over(st, i_in_chunk)) {
        pdl_wait();
        return;
    }
    const double tau = st->tau;
    ref_block(blk[b], blk[b + 1], cap, rp, ci, v, y, prod[w], [&](int j, double s) {
        const double xj = x[j], l = lo[j], u = up[j];
        double cand = __dsub_rn(xj, __dmul_rn(tau, __dsub_rn(cost[j], s)));
        if (fin_bound(l)) cand = smax(l, cand);
        if (fin_bound(u)) cand = smin(u, cand);
        xbar[j] = __dsub_rn(__dmul_rn(2.0, cand), xj);
        x[j] = cand;
    });
}

// Dual step, src/gpu/pdhg_solver.hpp:80-95; TEST: also each CTA's violation
// maximum to part[] (the stop test reads it every 32nd iteration only).
template <bool TEST>
__global__ void __launch_bounds__(kBlock) k_refb_dual(const int2* __restrict__ blk, int nblk, int cap,
                                                      const int* __restrict__ rp, const int* __restrict__ ci,
                                                      const double* __restrict__ v, const double* __restrict__ xbar,
                                                      const double* __restrict__ rlo, const double* __restrict__ rup,
                                                      double* __restrict__ y, double* __restrict__ part,
                                                      const DevState* __restrict__ st, int i_in_chunk) {
    __shared__ double prod[kWarps][kWarpCapMax];
    __shared__ double sh[kWarps];
    pdl_release();
    const int w = threadIdx.x >> 5, b = blockIdx.x * kWarps + w;
    if (ref_over(st, i_in_chunk)) {
        pdl_wait();
        return;
    }
    double viol = 0.0;
    if (b < nblk) {
        const double sigma = st->sigma;
        ref_block(blk[b], blk[b + 1], cap, rp, ci, v, xbar, prod[w], [&](int i, double a) {
            const double yi = y[i], lo = rlo[i], hi = rup[i];
            double r = __dsub_rn(a, __ddiv_rn(yi, sigma));
            if (fin_bound(lo)) r = smax(lo, r);
            if (fin_bound(hi)) r = smin(hi, r);
            y[i] = __dadd_rn(yi, __dmul_rn(sigma, __dsub_rn(r, a)));
            if (TEST) {
                if (fin_bound(lo)) viol = smax(viol, __dsub_rn(lo, a));
                if (fin_bound(hi)) viol = smax(viol, __dsub_rn(a, hi));
            }
        });
    } else {
        pdl_wait();
    }
    if (TEST) {
        const double bm = block_max(viol, sh);
        if (threadIdx.x == 0) part[blockIdx.x] = bm;
    }
}

// The stop test after a chunk's first iteration (chunks start at multiples
// of 32, their length) and the end of a chunk: k_ref_stop's outcomes with
// two launches a chunk instead of one an iteration.
__global__ void k_refb_test(const double* __restrict__ part, int nblk, DevState* st) {
    __shared__ double sh[kWarps];
    const long long it = st->iter;
    if (st->done || it >= st->max_iters || it <= 20) return;
    const double mx = block_max_array(part, nblk, sh);
    if (threadIdx.x == 0 && mx <= 1e-6) {
        st->done = 1;
        st->ref_stopped = 1;
        st->status = 0;
        st->ref_iterations = it + 1;
    }
}
__global__ void k_refb_end(DevState* st, int K) {
    if (threadIdx.x != 0 || st->done) return;
    if (st->iter + K >= st->max_iters) {
        st->done = 1;
        st->status = 6;  // NIR_STATUS_ITERATION_LIMIT
        st->ref_iterations = st->max_iters;
        return;
    }
    st->iter += K;
    st->ref_iterations = st->iter;
}

// Stop test after iteration `it`, src/gpu/pdhg_solver.hpp:97-100, and the
// iteration count of PdhgResult (iterations = it + 1 at a stop, max_iters
// at the cap).  Launched after every dual step; the last one of a chunk of
// K iterations advances st->iter.
__global__ void k_ref_stop(const double* __restrict__ part, int nblk, DevState* st, int i_in_chunk, int K) {
    __shared__ double sh[kWarps];
    if (st->done) return;
    const long long it = st->iter + i_in_chunk;
    if (it >= st->max_iters) return;
    const bool test = (it > 20) && ((it & 31) == 0);
    double mx = 0.0;
    if (test) mx = block_max_array(part, nblk, sh);
    if (threadIdx.x != 0) return;
    if (test && mx <= 1e-6) {
        st->done = 1;
        st->ref_stopped = 1;
        st->status = 0;
        st->ref_iterations = it + 1;
        return;
    }
    if (it + 1 >= st->max_iters) {
        st->done = 1;
        st->status = 6;  // NIR_STATUS_ITERATION_LIMIT
        st->ref_iterations = st->max_iters;
        return;
    }
    if (i_in_chunk == K - 1) {
        st->iter += K;
        st->ref_iterations = st->iter;
    }
}

}  // namespace nir
