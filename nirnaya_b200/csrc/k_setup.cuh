// Setup kernels: CSC -> CSR transpose on the device, diagonal
// preconditioning (Ruiz l-inf passes + one Pock-Chambolle alpha=1 pass,
// factors rounded to powers of two so scaling is exact), the power
// iteration for ||A||_2 and the scaled problem vectors.
#pragma once

#include "dev_common.cuh"
#include "k_verify.cuh"

namespace nir {

// col_of[k] = column of CSC entry k (one thread per column).
__global__ void k_expand_cols(int n, const long long* __restrict__ start, int* __restrict__ col_of) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    for (long long k = start[j]; k < start[j + 1]; ++k) col_of[k] = j;
}

__global__ void k_iota(long long n, int* __restrict__ v) {
    long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k < n) v[k] = int(k);
}

// row_ptr[i] = first position of key >= i in the sorted row keys.
__global__ void k_row_ptr_from_sorted(int m, long long nnz, const int* __restrict__ keys, int* __restrict__ rp) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > m) return;
    long long lo = 0, hi = nnz;
    while (lo < hi) {
        long long mid = (lo + hi) >> 1;
        if (keys[mid] < i) lo = mid + 1;
        else hi = mid;
    }
    rp[i] = int(lo);
}

__global__ void k_gather_csr(long long nnz, const int* __restrict__ perm, const int* __restrict__ col_of,
                             const double* __restrict__ v_in, int* __restrict__ ci, double* __restrict__ v_out) {
    long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (p >= nnz) return;
    int k = perm[p];
    ci[p] = col_of[k];
    v_out[p] = v_in[k];
}

__global__ void k_offsets_to_int(int n1, const long long* __restrict__ in, int* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n1) out[i] = int(in[i]);
}

// Sanitise bounds: anything the reference does not treat as a finite bound
// (src/core/types.hpp:49-51) becomes -inf (lower) or +inf (upper).
__global__ void k_sanitize_bounds(int n, const double* __restrict__ lo_in, const double* __restrict__ up_in,
                                  double* __restrict__ lo, double* __restrict__ up) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double l = lo_in[j], u = up_in[j];
    lo[j] = fin_bound(l) ? l : -INFINITY;
    up[j] = fin_bound(u) ? u : INFINITY;
}

// ---------------------------------------------------------------- scaling

// One warp per row: out[r] = max (mode 0) or sum (mode 1) over the row of
// |v| * d_row[r] * d_col[ci].  Deterministic shuffle tree.
__global__ void k_row_stat(int rows, const int* __restrict__ rp, const int* __restrict__ ci,
                           const double* __restrict__ v, const double* d_row, const double* d_col, int mode,
                           double* out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    pdl_release();
    pdl_wait();
    if (warp >= rows) return;
    const double dr = d_row[warp];
    double acc = 0.0;
    for (int k = rp[warp] + lane; k < rp[warp + 1]; k += 32) {
        double a = fabs(v[k]) * dr * d_col[ci[k]];
        acc = mode == 0 ? fmax(acc, a) : acc + a;
    }
    acc = mode == 0 ? warp_max(acc) : warp_sum(acc);
    if (lane == 0) out[warp] = acc;
}

// The same maximum with T lanes per row, for rows too short to fill a warp
// (a maximum does not depend on the order; the sum of mode 1 keeps the warp's
// tree, because its last bit can decide the rounding to a power of two).
// 16M nonzeros in rows of 10 and 25: 130 us a pass against 330 with a warp
// per row.
template <int T>
__global__ void k_row_max(int rows, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
                          const double* d_row, const double* d_col, double* out) {
    const int r = int((blockIdx.x * (long long)blockDim.x + threadIdx.x) / T), t = threadIdx.x % T;
    double acc = 0.0;
    pdl_release();
    int k = 0, e = 0;
    if (r < rows) {
        k = rp[r] + t;
        e = rp[r + 1];
    }
    pdl_wait();
    if (r < rows) {
        const double dr = d_row[r];
#pragma unroll 4
        for (; k < e; k += T) acc = fmax(acc, fabs(v[k]) * dr * d_col[ci[k]]);
    }
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) acc = fmax(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    if (r < rows && t == 0) out[r] = acc;
}

// d[i] /= sqrt(stat[i]) where stat > 0.
__global__ void k_apply_stat(int n, const double* stat, double* d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_release();
    pdl_wait();
    if (i >= n) return;
    double s = stat[i];
    if (s > 0.0 && isfinite(s)) d[i] /= sqrt(s);
}

// Nearest power of two (in the log sense), exponent clamped to +-60.
__global__ void k_round_pow2(int n, double* __restrict__ d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = d[i];
    if (!(v > 0.0) || !isfinite(v)) {
        d[i] = 1.0;
        return;
    }
    int e;
    double f = frexp(v, &e);  // v = f * 2^e, f in [0.5, 1)
    int k = (f >= 0.70710678118654752440) ? e : e - 1;
    k = k > 60 ? 60 : (k < -60 ? -60 : k);
    d[i] = ldexp(1.0, k);
}

// Scaled values of one orientation: v = (orig * dr_i) * dc_j with i the row
// of A and j the column of A, identical bits in both orientations.
__global__ void k_scale_values(int rows, const int* __restrict__ rp, const int* __restrict__ ci,
                               const double* __restrict__ orig, const double* __restrict__ d_this,
                               const double* __restrict__ d_other, int this_is_row_of_A, double* __restrict__ v64,
                               float* __restrict__ v32) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= rows) return;
    const double dt = d_this[warp];
    for (int k = rp[warp] + lane; k < rp[warp + 1]; k += 32) {
        const double dother = d_other[ci[k]];
        const double s = this_is_row_of_A ? (orig[k] * dt) * dother : (orig[k] * dother) * dt;
        v64[k] = s;
        v32[k] = float(s);
    }
}

// Scaled vectors: c^ = c*dc, l^ = l/dc, u^ = u/dc (columns);
// rl^ = rl*dr, ru^ = ru*dr (rows).  Infinite bounds stay infinite.
__global__ void k_scale_vectors(int n, int m, const double* __restrict__ c, const double* __restrict__ l,
                                const double* __restrict__ u, const double* __restrict__ rl,
                                const double* __restrict__ ru, const double* __restrict__ dc,
                                const double* __restrict__ dr, double* __restrict__ c64, double* __restrict__ l64,
                                double* __restrict__ u64, double* __restrict__ rl64, double* __restrict__ ru64,
                                float* __restrict__ c32, float* __restrict__ l32, float* __restrict__ u32,
                                float* __restrict__ rl32, float* __restrict__ ru32) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        double d = dc[t];
        double cc = c[t] * d, ll = l[t] / d, uu = u[t] / d;
        c64[t] = cc;
        l64[t] = ll;
        u64[t] = uu;
        c32[t] = float(cc);
        l32[t] = float(ll);
        u32[t] = float(uu);
    }
    if (t < m) {
        double d = dr[t];
        double a = rl[t] * d, b = ru[t] * d;
        rl64[t] = a;
        ru64[t] = b;
        rl32[t] = float(a);
        ru32[t] = float(b);
    }
}

// ---------------------------------------------------------------- power iteration

// Deterministic pseudo-random start in [0.5, 1.5) (splitmix64 of the index).
__device__ __forceinline__ double power_start_value(unsigned long long j) {
    unsigned long long z = j * 0x9e3779b97f4a7c15ULL + 0x632be59bd9b4e019ULL;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    z ^= z >> 31;
    return 0.5 + double(z >> 11) * 0x1.0p-53;
}

__global__ void k_power_start(int n, double* __restrict__ u) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    u[j] = power_start_value(j);
}

// Batch start: each instance's columns from its own index 0, so an
// instance's estimate does not depend on the batch around it.
__global__ void k_power_start_batch(int n, const int* __restrict__ col_inst, const int* __restrict__ col_off,
                                    double* __restrict__ u) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    u[j] = power_start_value(j - col_off[col_inst[j]]);
}

// FP64 SpMV of the power iteration with T lanes per row: y = A x / norm of
// the row's instance (norm null: 1; a zero norm gives 0).  T near a quarter
// of the mean row length: with a warp per row, rows of 10 entries left two
// thirds of the lanes idle (16M nonzeros: 220 us a product, 75 with 4 and 8
// lanes).  The division stands for a pass that scaled x.
// The kernels of a round, as those of the Ruiz passes, start while the ones
// before them end: set-up of a 120 x 300 LP 1.56 -> 1.22 ms, of a multiperiod
// one of 200,000 nonzeros 1.71 -> 1.09.
template <int T>
__global__ void k_power_spmv(int rows, const int* __restrict__ rp, const int* __restrict__ ci,
                             const double* __restrict__ v, const double* x, const double* norm,
                             const int* __restrict__ inst_of, double* y) {
    const int r = int((blockIdx.x * (long long)blockDim.x + threadIdx.x) / T), t = threadIdx.x % T;
    double acc = 0.0;
    pdl_release();
    int k = 0, e = 0;
    if (r < rows) {
        k = rp[r] + t;
        e = rp[r + 1];
    }
    pdl_wait();
#pragma unroll 4
    for (; k < e; k += T) acc += v[k] * x[ci[k]];
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (r < rows && t == 0) {
        if (norm) {
            const double d = norm[inst_of ? inst_of[r] : 0];
            acc = d > 0.0 ? acc / d : 0.0;
        }
        y[r] = acc;
    }
}

// Norms of an instance's part of w, in two steps: G CTAs per instance leave
// partial sums of squares, then one warp per instance adds them in a fixed
// order.
__global__ void k_seg_sumsq(int G, const int* __restrict__ off, const double* w, double* part) {
    __shared__ double sh[kWarps];
    pdl_release();
    pdl_wait();
    const int i = blockIdx.x / G, g = blockIdx.x % G;
    double s = 0.0;
    for (int j = off[i] + g * kBlock + int(threadIdx.x); j < off[i + 1]; j += G * kBlock) s += w[j] * w[j];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}
__global__ void k_seg_norm(int count, int G, const double* part, double* norm) {
    pdl_release();
    pdl_wait();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= count) return;
    double s = 0.0;
    for (int g = lane; g < G; g += 32) s += part[i * G + g];
    s = warp_sum(s);
    if (lane == 0) norm[i] = sqrt(s);
}

// ---------------------------------------------------------------- double-double sums

// Sums in double-double over an instance's entries (the reference's dd_real
// steps, k_verify.cuh): the objective c'x + offset of Model::eval_objective
// (src/model/model.hpp:73-98) and the norms of b and c, given and scaled.
// Each thread adds its entries, then the threads, then the G CTAs of an
// instance; the order differs from a loop's, the rounding is 2^-104 relative
// to the terms either way.  On the host these sums took 16 ms of a 256-
// iteration solve of 16M nonzeros, with another 18 MB copied back for them.
__device__ inline vfy::DD dd_warp(vfy::DD d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double h = __shfl_down_sync(0xffffffffu, d.hi, o), l = __shfl_down_sync(0xffffffffu, d.lo, o);
        vfy::add_dd(d, h, l);
    }
    return d;
}
// The CTA's sum in thread 0.
__device__ inline vfy::DD dd_block(vfy::DD d, vfy::DD* sh /* kWarps */) {
    d = dd_warp(d);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 1; k < kWarps; ++k) vfy::add_dd(d, sh[k].hi, sh[k].lo);
    return d;
}

constexpr int kDdNorms = 4;  // c, c scaled, b, b scaled (b_i: the larger finite bound of row i in magnitude)

__global__ void __launch_bounds__(kBlock) k_dd_norms(int G, const int* __restrict__ row_off, const int* __restrict__ col_off,
                                                     const double* __restrict__ c, const double* __restrict__ dc,
                                                     const double* __restrict__ rl, const double* __restrict__ ru,
                                                     const double* __restrict__ dr, vfy::DD* __restrict__ part) {
    __shared__ vfy::DD sh[kWarps];
    const int i = blockIdx.x / G, g = blockIdx.x % G;
    vfy::DD s[kDdNorms] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    for (int j = col_off[i] + g * kBlock + int(threadIdx.x); j < col_off[i + 1]; j += G * kBlock) {
        const double a = c[j], b = vfy::mul(a, dc[j]);
        vfy::add_prod(s[0], a, a);
        vfy::add_prod(s[1], b, b);
    }
    for (int r = row_off[i] + g * kBlock + int(threadIdx.x); r < row_off[i + 1]; r += G * kBlock) {
        double a = 0.0;
        if (isfinite(rl[r])) a = fabs(rl[r]);
        if (isfinite(ru[r])) a = fmax(a, fabs(ru[r]));
        const double b = vfy::mul(a, dr[r]);
        vfy::add_prod(s[2], a, a);
        vfy::add_prod(s[3], b, b);
    }
#pragma unroll
    for (int q = 0; q < kDdNorms; ++q) {
        const vfy::DD d = dd_block(s[q], sh);
        if (threadIdx.x == 0) part[blockIdx.x * kDdNorms + q] = d;
    }
}

__global__ void __launch_bounds__(kBlock) k_dd_objective(int G, const int* __restrict__ col_off,
                                                         const double* __restrict__ c, const double* __restrict__ x,
                                                         vfy::DD* __restrict__ part) {
    __shared__ vfy::DD sh[kWarps];
    const int i = blockIdx.x / G, g = blockIdx.x % G;
    vfy::DD s{0.0, 0.0};
    for (int j = col_off[i] + g * kBlock + int(threadIdx.x); j < col_off[i + 1]; j += G * kBlock)
        if (c[j] != 0.0 && x[j] != 0.0) vfy::add_prod(s, c[j], x[j]);
    const vfy::DD d = dd_block(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = d;
}

// out[i Q + q] = base[i] (or 0) plus the G partial sums, in order.
__global__ void k_dd_finish(int count, int G, int Q, const vfy::DD* __restrict__ part, const double* __restrict__ base,
                            double* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count * Q) return;
    const int i = t / Q, q = t % Q;
    vfy::DD s{base ? base[i] : 0.0, 0.0};
#pragma unroll 8
    for (int g = 0; g < G; ++g) {
        const vfy::DD p = part[(size_t(i) * G + g) * Q + q];
        vfy::add_dd(s, p.hi, p.lo);
    }
    out[t] = vfy::add(s.hi, s.lo);
}

// ---------------------------------------------------------------- iterate setup

// x^ = clamp(x_init / dc (or 0), l^, u^); y^ = y_init / dr (or 0); both
// also copied into the anchors and converted to FP32.
__global__ void k_init_iterates(int n, int m, const double* __restrict__ x_in, const double* __restrict__ y_in,
                                const double* __restrict__ dc, const double* __restrict__ dr,
                                const double* __restrict__ l64, const double* __restrict__ u64,
                                double* __restrict__ x64, double* __restrict__ x064, double* __restrict__ y64,
                                double* __restrict__ y064, float* __restrict__ x32, float* __restrict__ x032,
                                float* __restrict__ y32, float* __restrict__ y032, const float* __restrict__ l32,
                                const float* __restrict__ u32) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        double v = x_in ? x_in[t] / dc[t] : 0.0;
        double v64 = clamp_box(v, l64[t], u64[t]);
        x64[t] = v64;
        x064[t] = v64;
        float v32 = clamp_box(float(v), l32[t], u32[t]);
        x32[t] = v32;
        x032[t] = v32;
    }
    if (t < m) {
        double v = y_in ? y_in[t] / dr[t] : 0.0;
        y64[t] = v;
        y064[t] = v;
        y32[t] = float(v);
        y032[t] = float(v);
    }
}

// FP32 -> FP64 hand-over for the polish phase: iterate and anchor become
// the last evaluated point (x+, y+), clamped to the FP64 box.
__global__ void k_promote(int n, int m, const float* __restrict__ xp32, const float* __restrict__ yp32,
                          const double* __restrict__ l64, const double* __restrict__ u64, double* __restrict__ x64,
                          double* __restrict__ x064, double* __restrict__ xp64, double* __restrict__ y64,
                          double* __restrict__ y064, double* __restrict__ yp64) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        double v = clamp_box(double(xp32[t]), l64[t], u64[t]);
        x64[t] = v;
        x064[t] = v;
        xp64[t] = v;
    }
    if (t < m) {
        double v = double(yp32[t]);
        y64[t] = v;
        y064[t] = v;
        yp64[t] = v;
    }
}

// Fresh start of the FP64 polish at the last evaluated point: iterate and
// anchor become (x+, y+).
__global__ void k_restart_at(int n, int m, const double* __restrict__ xp, const double* __restrict__ yp,
                             double* __restrict__ x, double* __restrict__ x0, double* __restrict__ y,
                             double* __restrict__ y0) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        x[t] = xp[t];
        x0[t] = xp[t];
    }
    if (t < m) {
        y[t] = yp[t];
        y0[t] = yp[t];
    }
}

// Original-space output: x = dc * x^, y = dr * y^.
template <typename T>
__global__ void k_unscale_out(int n, int m, const T* __restrict__ xp, const T* __restrict__ yp,
                              const double* __restrict__ dc, const double* __restrict__ dr, double* __restrict__ xo,
                              double* __restrict__ yo) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) xo[t] = double(xp[t]) * dc[t];
    if (t < m) yo[t] = double(yp[t]) * dr[t];
}

__global__ void k_to_float(long long n, const double* __restrict__ a, float* __restrict__ b) {
    long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k < n) b[k] = float(a[k]);
}

__global__ void k_to_double(long long n, const float* __restrict__ a, double* __restrict__ b) {
    long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k < n) b[k] = double(a[k]);
}

__global__ void k_fill(long long n, double v, double* __restrict__ a) {
    long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k < n) a[k] = v;
}

// Compact status record written to host-mapped memory at the end of
// every launch chunk, read by the host after the chunk's event.
struct HostSnap {
    long long seq;
    long long iter;
    int done, status, phase, restarts;
    double kkt, kp, kd, kg, pobj, dobj, max_rel_row, omega, res;
    long long ref_iterations;
    int ref_stopped, pad;
};

constexpr int kSnapRing = 64;

// One thread.
__device__ inline void write_snap(const DevState* st, HostSnap* ring, long long* seq) {
    long long s = *seq + 1;
    *seq = s;
    HostSnap h;
    h.seq = s;
    h.iter = st->iter;
    h.done = st->done;
    h.status = st->status;
    h.phase = st->phase;
    h.restarts = st->restarts;
    h.kkt = st->kkt;
    h.kp = st->kp;
    h.kd = st->kd;
    h.kg = st->kg;
    h.pobj = st->pobj;
    h.dobj = st->dobj;
    h.max_rel_row = st->max_rel_row;
    h.omega = st->omega;
    h.res = st->res;
    h.ref_iterations = st->ref_iterations;
    h.ref_stopped = st->ref_stopped;
    h.pad = 0;
    ring[s % kSnapRing] = h;
    __threadfence_system();
}

__global__ void k_snap(const DevState* st, HostSnap* ring, long long* seq) {
    if (threadIdx.x == 0 && blockIdx.x == 0) write_snap(st, ring, seq);
}

}  // namespace nir
