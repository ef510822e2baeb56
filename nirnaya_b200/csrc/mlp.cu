// Warm-start network: hand-written BF16 tensor-core GEMMs (tcgen05, FP32
// accumulation), fused epilogues, Adam, all on one stream.
// C ABI: include/nir_mlp.h.
//
// GEMM.  C[M x N] = sum_k A(m, k) * B(n, k).  Each operand is stored either
// K-major (element (r, k) at P[r * ld + k]) or MN-major (at P[k * ld + r]);
// the three products of a dense layer use all three combinations:
//   forward   Y  = X * W^T      A = X  K-major,  B = W  K-major
//   input grad dX = dY * W      A = dY K-major,  B = W  MN-major
//   weight grad dW = dY^T * X   A = dY MN-major, B = X  MN-major
// A CTA computes a tile of 128 rows and 64 or 128 columns: TMA brings the
// operands into shared memory stage by stage, 64 of K each, one thread issues
// tcgen05.mma on them, the FP32 accumulators lie in tensor memory, and 8
// warps finish the tile (bias, ReLU, mask) and store it.
// A product with few output tiles and a long K is a sum of splits of K, added
// in order (deterministic): a CTA keeps an accumulator for each, or the CTAs
// of a thread-block cluster compute them side by side and add them through
// each other's shared memory, or as many CTAs as there are splits leave them
// in a workspace, where another kernel adds them.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <random>
#include <stdexcept>
#include <string>
#include <vector>

#include "grown.hpp"
#include "mapped_host.hpp"
#include "nir_mlp.h"

namespace {

thread_local std::string g_err;

#define MLP_CUDA(call)                                                                              \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess)                                                                      \
            throw std::runtime_error(std::string(#call) + ": " + cudaGetErrorString(e_));           \
    } while (0)
#define MLP_LAUNCHED() MLP_CUDA(cudaGetLastError())

using bf16 = __nv_bfloat16;

constexpr int BM = 128, BN = 128, BK = 32;  // BM x BN: the tiles the splits of K are counted by

enum Epi : int { EPI_BIAS_RELU_BF16 = 0, EPI_BIAS_F32 = 1, EPI_MASK_BF16 = 2, EPI_F32 = 3 };

struct GemmArgs {
    const bf16* A;
    int lda;
    const bf16* B;
    int ldb;
    int M, N, K;
    int kps;           // K range per split (multiple of BK)
    int splits;        // partial sums of kps each, added in order
    int epi;
    const float* bias;
    bf16* out_bf;
    float* out_f;
    int ldc;
    const bf16* mask;  // EPI_MASK_BF16: multiply by (mask > 0)
    int ldm;
    bool wide;         // rows of whole, aligned groups of 8 columns
};

// Programmatic dependent launch: with the launch attribute a kernel starts
// while the one before still runs and waits for it before it reads what
// that wrote; without it both do nothing.
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The epilogue of one element, and of 8 neighbouring columns (col a multiple
// of 8), which are read and stored together where the rows allow it.
__device__ __forceinline__ void epilogue1(const GemmArgs& g, int row, int col, float v) {
    const size_t o = (size_t)row * g.ldc + col;
    switch (g.epi) {
        case EPI_BIAS_RELU_BF16: g.out_bf[o] = __float2bfloat16_rn(fmaxf(v + g.bias[col], 0.f)); break;
        case EPI_BIAS_F32: g.out_f[o] = v + g.bias[col]; break;
        case EPI_MASK_BF16:
            g.out_bf[o] = __float2bfloat16_rn(__bfloat162float(g.mask[(size_t)row * g.ldm + col]) > 0.f ? v : 0.f);
            break;
        default: g.out_f[o] = v; break;
    }
}
__device__ __forceinline__ void epilogue8(const GemmArgs& g, int row, int col, const float (&in)[8]) {
    if (!g.wide) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (col + j < g.N) epilogue1(g, row, col + j, in[j]);
        return;
    }
    const size_t o = (size_t)row * g.ldc + col;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = in[j];
    if (g.epi == EPI_BIAS_RELU_BF16 || g.epi == EPI_BIAS_F32) {
        const float4* b = reinterpret_cast<const float4*>(g.bias + col);
        const float4 b0 = b[0], b1 = b[1];
        v[0] += b0.x, v[1] += b0.y, v[2] += b0.z, v[3] += b0.w;
        v[4] += b1.x, v[5] += b1.y, v[6] += b1.z, v[7] += b1.w;
    }
    if (g.epi == EPI_BIAS_F32 || g.epi == EPI_F32) {
        float4* q = reinterpret_cast<float4*>(g.out_f + o);
        q[0] = make_float4(v[0], v[1], v[2], v[3]);
        q[1] = make_float4(v[4], v[5], v[6], v[7]);
        return;
    }
    union Pack {
        uint4 q;
        bf16 e[8];
        __device__ Pack() {}
    } out, m;
    if (g.epi == EPI_MASK_BF16) {
        m.q = *reinterpret_cast<const uint4*>(g.mask + (size_t)row * g.ldm + col);
#pragma unroll
        for (int j = 0; j < 8; ++j) out.e[j] = __float2bfloat16_rn(__bfloat162float(m.e[j]) > 0.f ? v[j] : 0.f);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) out.e[j] = __float2bfloat16_rn(fmaxf(v[j], 0.f));
    }
    *reinterpret_cast<uint4*>(g.out_bf + o) = out.q;
}

// ---- the GEMM kernel
//
// A CTA of 8 warps computes a 128 x TN tile in tensor memory, 64 of K a
// stage.  One thread has the operands brought into shared memory by TMA, in
// the 128-byte swizzle that the tensor core reads, several stages ahead;
// another issues each stage's tcgen05.mma (K = 16 each, in order).  A CTA
// computes G.accs splits one after another, each in its own accumulator, and
// adds them in order as it reads them; or (G.rank_bits > 0) the CTAs of a
// cluster share the tile: in each round a rank computes one split and leaves
// it in shared memory, where the stages were, and every rank adds its share
// of the tile's rows over the splits in order, reading the other ranks'
// shared memory; or (G.parts) each split of a tile has a CTA of its own, which
// leaves it in the workspace as rows of a taller product, for k_add_splits.
// Neither the tile nor the ranks decide the order of any sum.
// One launch takes a group of independent products (the weight gradients of
// all layers).
// Small products are bound by their latency (load, multiply, read back,
// store), large ones by the loads: with 128 x 128 tiles a stage's 32 KB from
// L2 take longer than its 256 cycles of multiplication.  In TFLOP/s, with
// mma.sync on 128 x 128 tiles and splits added by another kernel before:
// 8192^3 280 -> 1290, 4096^3 327 -> 1110, 65536 x 512 x 512 222 -> 490,
// 8192 x 512 x 512 75 -> 420, 1024 x 512 x 512 29 -> 80.
constexpr int GROUP_MAX = 17;  // layers
constexpr int RANK_BITS_MAX = 4;
constexpr int STAGES_MAX = 6;
constexpr int SK = 64;         // K of a stage
constexpr int TMEM_COLUMNS = 512;  // of an SM
// A wait ends after so many tries (about 30 ms), one for loads after another
// wait has failed sooner.
constexpr int WAIT_TRIES = 1 << 20, DRAIN_TRIES = 1 << 12;

template <int TN>
struct GTile {
    static constexpr int threads = 256;
    static constexpr int bytes_a = 128 * SK * 2, bytes_b = TN * SK * 2;
    static constexpr int stage = bytes_a + bytes_b;      // 24 or 32 KB
    static constexpr int ld = TN + 4;                    // floats per row of the finished tile
    // dynamic shared memory, from a multiple of 1024: the stages, or the tile
    static constexpr int tile = 128 * ld * 4;
    static int smem(int stages) { return std::max(stages * stage, tile) + 1024; }
};

struct GemmOne {
    alignas(64) CUtensorMap a, b;
    GemmArgs g;
};
template <int MAX>
struct GemmGroupOf {
    GemmOne g[MAX];
    int first[MAX + 1];  // first tile of each product
    int count;
    int rank_bits;       // 2^rank_bits CTAs per tile, a cluster
    int parts;           // splits per tile that CTAs leave in the workspace, or 0 (then rank_bits = 0, accs = 1)
    int accs;            // splits that a CTA computes one after another, each in its own accumulator (one CTA per tile)
    int stages;          // at most STAGES_MAX
    uint32_t tmem;       // columns of tensor memory for them, a power of two
    uint32_t lost;       // test of the bounded waits: bytes of every stage that nobody loads
    int* fault;          // set if a wait of the kernel gives up
};
// Weight gradients come in groups, the other products one by one (the
// arguments of a launch are copied by the host).
template <bool AK, bool BKM>
using GemmGroup = GemmGroupOf<(!AK && !BKM) ? GROUP_MAX : 1>;

// A stage's operand: K-major ROWS rows of 64 k (128 bytes); MN-major 64
// K-rows of 64 rows (128 bytes), 64 ROWS after 64 ROWS.
template <int ROWS, bool KMAJ>
__device__ __forceinline__ void load_operand(uint32_t dst, const CUtensorMap* map, int r0, int k0, uint32_t bar) {
#pragma unroll
    for (int i = 0; i < (KMAJ ? 1 : ROWS / 64); ++i)
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
            "[%4];" ::"r"(dst + i * (SK * 128)),
            "l"(map), "r"(KMAJ ? k0 : r0 + i * 64), "r"(KMAJ ? r0 : k0), "r"(bar)
            : "memory");
}

// Shared-memory descriptor of an operand at `addr` in the 128-byte swizzle:
// groups of 8 rows (K-major) or 8 K-rows (MN-major) 1024 bytes apart; MN-major
// the next 64 rows after SK K-rows.
template <bool KMAJ>
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    const uint64_t lead = KMAJ ? 1 : (SK * 128) >> 4;
    return uint64_t((addr >> 4) & 0x3fff) | (lead << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
           (uint64_t(2) << 61);
}

__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, int tries = WAIT_TRIES) {
    for (int i = 0; i < tries; ++i) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// 8 floats of a rank's shared memory, added to v.
__device__ __forceinline__ void add_rank8(uint32_t addr, int rank, float (&v)[8]) {
    uint32_t a;
    float w[8];
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3])
                 : "r"(a)
                 : "memory");
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7])
                 : "r"(a + 16)
                 : "memory");
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += w[j];
}

// Arrives at `bar` when this thread's multiplications so far are done.
__device__ __forceinline__ void mma_arrive(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 16 columns of this warp's 32 rows of tensor memory.
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

template <int TN, bool AK, bool BKM>
__global__ void __launch_bounds__(256, 2) k_gemm(const __grid_constant__ GemmGroup<AK, BKM> G) {
    using L = GTile<TN>;
    const int S = G.stages;
    constexpr int GROUPS = TN / 8;                 // 8-column groups of a row
    constexpr int SUMS = 128 * GROUPS / 2 / 256;   // groups that a thread adds, for two ranks
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint32_t tmem_at;
    __shared__ int gave_up;  // a wait of the multiplying thread ran out
    __shared__ __align__(8) unsigned long long bars[2 * STAGES_MAX + 1];  // stage full, stage free, round multiplied
    pdl_release();
    const uint32_t sb = (static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + 1023u) & ~1023u;
    const uint32_t full = static_cast<uint32_t>(__cvta_generic_to_shared(bars)), free = full + 8 * STAGES_MAX,
                   all = free + 8 * STAGES_MAX;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&tmem_at))),
                     "r"(G.tmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    } else if (tid == 32) {
        gave_up = 0;
        for (int i = 0; i <= 2 * STAGES_MAX; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + i * 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    int ranks = 1 << G.rank_bits, tile = int(blockIdx.x) >> G.rank_bits, rank = int(blockIdx.x) & (ranks - 1);
    if (G.parts) {
        ranks = G.parts;
        tile = int(blockIdx.x) / ranks;
        rank = int(blockIdx.x) % ranks;
    }
    int p = 0;
    while (p + 1 < G.count && tile >= G.first[p + 1]) ++p;
    const GemmOne& o = G.g[p];
    const GemmArgs& g = o.g;
    const int tn = (g.N + TN - 1) / TN, t = tile - G.first[p];
    const int m0 = (t / tn) * 128, n0 = (t % tn) * TN;
    const bool split = G.rank_bits > 0 && g.splits > 1;  // over the ranks
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_at;
    // BF16 operands (K-major or MN-major), FP32 accumulator, 128 x TN
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (AK ? 0u : 1u << 15) | (BKM ? 0u : 1u << 16) |
                               (uint32_t(TN / 8) << 17) | (8u << 24);
    constexpr uint32_t step_a = AK ? 32 : 2048, step_b = BKM ? 32 : 2048;  // 16 of K
    bool ok = true;
    int bad = 0;           // gave_up
    int rounds = 0;        // multiplied so far
    const uint32_t expect = uint32_t(L::stage) + G.lost;  // bytes of a stage
    int s = 0, phase = 0;  // of the loading and of the multiplying thread: the next stage, and how often all were passed
    float sum[SUMS][8];
#pragma unroll
    for (int i = 0; i < SUMS; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[i][j] = 0.f;
    pdl_wait();  // the operands come from the kernels before

    for (int round = 0; round < g.splits; round += ranks * G.accs) {
        // this CTA's splits of the round, their stages one after another
        const int z0 = round + rank * G.accs, z1 = min(z0 + G.accs, g.splits);
        if (tid == 32) {
            for (int z = z0; z < z1; ++z)
                for (int k = z * g.kps; k < min(g.K, (z + 1) * g.kps); k += SK) {
                    if (phase > 0) ok = ok && bar_wait(free + s * 8, (phase - 1) & 1);
                    if (!ok) break;
                    const uint32_t at = sb + s * L::stage;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + s * 8),
                                 "r"(expect)
                                 : "memory");
                    load_operand<128, AK>(at, &o.a, m0, k, full + s * 8);
                    load_operand<TN, BKM>(at + L::bytes_a, &o.b, n0, k, full + s * 8);
                    if (++s == S) s = 0, ++phase;
                }
        } else if (tid == 0 && z1 > z0) {
            for (int z = z0; z < z1; ++z) {
                const int kbeg = z * g.kps, kend = min(g.K, kbeg + g.kps);
                const uint32_t acc = tmem + (z - z0) * TN;
                for (int k = kbeg; k < kend; k += SK) {
                    ok = ok && bar_wait(full + s * 8, phase & 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t at = sb + s * L::stage;
                    const uint64_t da = smem_desc<AK>(at), db = smem_desc<BKM>(at + L::bytes_a);
                    // whole steps of BK, zero-filled past the end of K
                    const int steps = min(SK, (kend - k + BK - 1) / BK * BK) / 16;
#pragma unroll
                    for (int q = 0; q < SK / 16; ++q)
                        if (q < steps)
                            asm volatile(
                                "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(acc),
                                "l"(da + ((q * step_a) >> 4)), "l"(db + ((q * step_b) >> 4)), "r"(idesc),
                                "r"(uint32_t(k > kbeg || q > 0))
                                : "memory");
                    mma_arrive(free + s * 8);
                    if (++s == S) s = 0, ++phase;
                }
            }
            mma_arrive(all);
        }
        __syncwarp();
        if (z1 > z0) {
            ok = bar_wait(all, rounds & 1) && ok;
            ++rounds;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (tid == 0 && !ok) gave_up = 1;
        __syncthreads();  // the finished tile lies where the stages were
        bad |= gave_up;
        if (z1 > z0) {
            // warp w holds rows 32 (w % 4).. and half of the columns
            const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * (TN / 2);
            const uint32_t to = sb + uint32_t(r * L::ld + c0) * 4u;
            const uint32_t from = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(c0);
#pragma unroll
            for (int c = 0; c < TN / 2; c += 16) {
                float v[16];
                tmem_ld16(from + c, v);
                if (G.accs > 1 && g.splits > 1) {  // add this CTA's splits in order
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = 0.f + v[j];
                    for (int z = 1; z < g.splits; ++z) {
                        float w[16];
                        tmem_ld16(from + z * TN + c, w);
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] += w[j];
                    }
                }
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + (c + j) * 4), "f"(v[j]),
                                 "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3])
                                 : "memory");
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (!split) {
            __syncthreads();
            const int part = G.parts ? rank * g.M : 0;  // first row of this split in the workspace
            for (int e = tid; e < ((G.parts ? z1 > z0 : rank == 0) ? 128 * GROUPS : 0); e += 256) {
                const int r = e / GROUPS, c = 8 * (e % GROUPS);
                if (m0 + r >= g.M || n0 + c >= g.N) continue;
                float v[8];
                const uint32_t at = sb + uint32_t(r * L::ld + c) * 4u;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                             : "r"(at)
                             : "memory");
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                             : "r"(at + 16)
                             : "memory");
                epilogue8(g, part + m0 + r, n0 + c, v);
            }
        } else {
            cluster_arrive();
            cluster_wait();
            const int have = min(ranks, g.splits - round);
            const int per = 128 >> G.rank_bits, mine = per * GROUPS;
#pragma unroll
            for (int i = 0; i < SUMS; ++i) {
                const int e = tid + i * 256;
                if (e < mine) {
                    const uint32_t at = sb + uint32_t((rank * per + e / GROUPS) * L::ld + 8 * (e % GROUPS)) * 4u;
#pragma unroll 4
                    for (int q = 0; q < have; ++q) add_rank8(at, q, sum[i]);
                }
            }
            // no rank leaves or fills its stages while another reads its tile
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            cluster_arrive();
            if (round + ranks >= g.splits) {
#pragma unroll
                for (int i = 0; i < SUMS; ++i) {
                    const int e = tid + i * 256;
                    const int r = rank * per + e / GROUPS, c = 8 * (e % GROUPS);
                    if (e < mine && m0 + r < g.M && n0 + c < g.N) epilogue8(g, m0 + r, n0 + c, sum[i]);
                }
            }
            cluster_wait();
        }
    }
    // given up: the loads that were started land while this CTA is there
    if (tid == 32 && bad)
        for (int j = 0; j < S; ++j)
            if (j < s || phase > 0) bar_wait(full + j * 8, (j < s ? phase : phase - 1) & 1, DRAIN_TRIES);
    if (!ok) *G.fault = 1;
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(G.tmem));
}

// C of each product from its splits in the workspace, one element per thread.
struct AddTable {
    GemmArgs g[GROUP_MAX];
    const float* ws[GROUP_MAX];  // splits x M x N
    int first[GROUP_MAX + 1];    // first CTA of each product
    int count;
};
__global__ void __launch_bounds__(256) k_add_splits(const __grid_constant__ AddTable t) {
    pdl_release();
    int p = 0;
    while (p + 1 < t.count && int(blockIdx.x) >= t.first[p + 1]) ++p;
    const GemmArgs& g = t.g[p];
    const size_t n = (size_t)g.M * g.N, i = (size_t)(int(blockIdx.x) - t.first[p]) * 256 + threadIdx.x;
    pdl_wait();
    if (i >= n) return;
    const float* ws = t.ws[p] + i;
    float v = 0.f;
#pragma unroll 16
    for (int z = 0; z < g.splits; ++z) v += ws[(size_t)z * n];
    epilogue1(g, int(i / g.N), int(i % g.N), v);
}

// ------------------------------------------------------------ elementwise

__global__ void k_to_bf16(size_t n, const float* __restrict__ a, bf16* __restrict__ b) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        b[i] = __float2bfloat16_rn(a[i]);
}

// out[i] = shift[i] + scale[i] * clamp(pred[i * ld + col], lo, hi), FP64
// (r0 = the first sample of this chunk; pred holds the chunk's rows).  The
// product and the sum are rounded separately (no fused multiply-add), the
// clamp passes a NaN through, and a missing scale or shift is no operation,
// so the result is the host's numpy expression bit for bit.
__global__ void k_affine_out(int rows, int r0, const float* __restrict__ pred, int ld, int col, double lo, double hi,
                             const double* __restrict__ scale, const double* __restrict__ shift,
                             double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    const int g = r0 + i;
    double p = double(pred[(size_t)i * ld + col]);
    p = (p < lo) ? lo : ((p > hi) ? hi : p);
    const double v = scale ? __dmul_rn(scale[g], p) : p;
    out[g] = shift ? __dadd_rn(shift[g], v) : v;
}

template <typename T>
__global__ void k_gather_rows(const int* __restrict__ idx, int rows, int cols, const T* __restrict__ src,
                              T* __restrict__ dst) {
    const size_t total = (size_t)rows * cols;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int r = int(i / cols), c = int(i % cols);
        dst[i] = src[(size_t)idx[r] * cols + c];
    }
}

__device__ __forceinline__ float block_sum_f(float v, float* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    float t = 0.f;
    if (threadIdx.x == 0)
        for (int i = 0; i < int(blockDim.x >> 5); ++i) t += sh[i];
    __syncthreads();
    return t;
}

// dY = scale * w * (pred - target) (BF16) and per-block sums of w*(pred-target)^2.
// (pred is still being written when an early launch starts: not restrict.)
__global__ void k_loss(int rows, int cols, const float* pred, const float* __restrict__ tgt,
                       const float* __restrict__ w, float scale, bf16* __restrict__ dy, float* __restrict__ part) {
    __shared__ float sh[32];
    const size_t total = (size_t)rows * cols;
    float s = 0.f;
    pdl_release();
    pdl_wait();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const float wc = w[i % cols];
        const float d = pred[i] - tgt[i];
        s += wc * d * d;
        dy[i] = __float2bfloat16_rn(scale * (wc * d));
    }
    s = block_sum_f(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// out[slot] = mul * the sum of the slot's n partials, one CTA per slot (all
// steps of an epoch at once).
__global__ void k_sum_partials(int n, const float* __restrict__ part, float mul, float* __restrict__ out) {
    __shared__ float sh[32];
    const float* p = part + (size_t)blockIdx.x * n;
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += p[i];
    s = block_sum_f(s, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = s * mul;
}

// db[c] = sum over rows of dY[r][c] in two deterministic passes: chunk z
// of kColChunkRows rows -> part[z][c] (rows in order), then the chunks in
// order.
constexpr int kColChunkRows = 128;

// The chunks of every layer in one launch.
struct ColsumTable {
    const bf16* dy[GROUP_MAX];
    float* part[GROUP_MAX];
    int cols[GROUP_MAX];
    int first[GROUP_MAX + 1];  // first CTA of each layer
    int count, rows;
};
// A CTA takes 64 columns of a chunk: all threads load it, then a thread per
// column adds its 128 values in order out of shared memory.
constexpr int kColsumCols = 64;
__global__ void __launch_bounds__(256) k_colsum_part(const __grid_constant__ ColsumTable t) {
    __shared__ __align__(16) bf16 sh[kColChunkRows][kColsumCols];
    pdl_release();
    int l = 0;
    while (l + 1 < t.count && int(blockIdx.x) >= t.first[l + 1]) ++l;
    const int cols = t.cols[l], cb = (cols + kColsumCols - 1) / kColsumCols, b = int(blockIdx.x) - t.first[l];
    const int c0 = (b % cb) * kColsumCols, z = b / cb;
    const int r0 = z * kColChunkRows, n = min(t.rows - r0, kColChunkRows);
    pdl_wait();
    // 8 columns (16 bytes) at a time; cols is a multiple of 8
    for (int i = threadIdx.x; i < n * (kColsumCols / 8); i += 256) {
        const int r = i / (kColsumCols / 8), c = 8 * (i % (kColsumCols / 8));
        if (c0 + c < cols)
            *reinterpret_cast<uint4*>(&sh[r][c]) =
                *reinterpret_cast<const uint4*>(t.dy[l] + (size_t)(r0 + r) * cols + c0 + c);
    }
    __syncthreads();
    const int c = threadIdx.x;
    if (c >= kColsumCols || c0 + c >= cols) return;
    float s = 0.f;
#pragma unroll 16
    for (int r = 0; r < n; ++r) s += __bfloat162float(sh[r][c]);
    t.part[l][(size_t)z * cols + c0 + c] = s;
}

// (part: not restrict, k_adam starts while it is written)
__device__ __forceinline__ float colsum_total(int chunks, int cols, int c, const float* part) {
    float s = 0.f;
    for (int z = 0; z < chunks; ++z) s += part[(size_t)z * cols + c];
    return s;
}

__global__ void k_colsum_final(int chunks, int cols, const float* __restrict__ part, float* __restrict__ db) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < cols) db[c] = colsum_total(chunks, cols, c, part);
}

// Adam over the weights and biases of every layer in one launch, one element
// per thread; a bias' gradient is added up from its chunks here.
struct AdamTable {
    struct Layer {
        float *w, *gw, *mw, *vw, *b, *gb, *mb, *vb;
        bf16* wb;
        const float* part;
        int nw, nb;
    } l[GROUP_MAX];
    int first[GROUP_MAX + 1];  // first CTA of each layer
    int count, chunks;
    const float2* bc;  // the step's bias corrections
    float lr, b1, b2, eps;
};
__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ AdamTable t) {
    pdl_release();
    int l = 0;
    while (l + 1 < t.count && int(blockIdx.x) >= t.first[l + 1]) ++l;
    const AdamTable::Layer& y = t.l[l];
    const int i = (int(blockIdx.x) - t.first[l]) * 256 + int(threadIdx.x);
    pdl_wait();
    if (i >= y.nw + y.nb) return;
    const bool weight = i < y.nw;
    const int j = weight ? i : i - y.nw;
    float* m = weight ? y.mw : y.mb;
    float* v = weight ? y.vw : y.vb;
    float* w = weight ? y.w : y.b;
    float gi;
    if (weight) {
        gi = y.gw[j];
    } else {
        gi = colsum_total(t.chunks, y.nb, j, y.part);
        y.gb[j] = gi;
    }
    // the roundings are spelled out, so that they do not depend on what the
    // compiler contracts here
    const float mi = __fmaf_rn(1.f - t.b1, gi, __fmul_rn(t.b1, m[j]));
    const float vi = __fmaf_rn(__fmul_rn(1.f - t.b2, gi), gi, __fmul_rn(t.b2, v[j]));
    m[j] = mi;
    v[j] = vi;
    const float2 bc = __ldg(t.bc);
    const float wi = w[j] - t.lr * (mi / bc.x) / (sqrtf(vi / bc.y) + t.eps);
    w[j] = wi;
    if (weight) y.wb[j] = __float2bfloat16_rn(wi);
}

// Uniform(-a, a) from a counter hash (splitmix64) of (seed, index).
__global__ void k_init_uniform(size_t n, uint64_t seed, float a, float* __restrict__ w, bf16* __restrict__ wb) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        uint64_t z = seed + 0x9e3779b97f4a7c15ULL * (i + 1);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
        z ^= z >> 31;
        const float u = float(z >> 40) * (1.0f / 16777216.0f);  // [0, 1)
        const float x = (2.f * u - 1.f) * a;
        w[i] = x;
        if (wb) wb[i] = __float2bfloat16_rn(x);
    }
}

unsigned grid1d(size_t n, int cap = 148 * 16) {
    size_t b = (n + 255) / 256;
    return unsigned(std::max<size_t>(1, std::min<size_t>(b, cap)));
}

}  // namespace

// ------------------------------------------------------------ the handle

namespace {
// A flag for each handle in host memory, which a kernel sets when one of its
// waits gives up: the host reads it after a synchronisation at no cost.
nir::MappedBlocks& fault_flags() {
    static auto* const flags = new nir::MappedBlocks(sizeof(int));  // outlives every handle
    return *flags;
}
}  // namespace

struct nir_mlp {
    nir_mlp_config cfg{};
    int device = 0;
    int sms = 148;
    cudaStream_t stream = nullptr;
    std::vector<int> dims;  // d_in, width x depth, d_out
    struct Layer {
        int in = 0, out = 0;
        float *W = nullptr, *b = nullptr, *gW = nullptr, *gb = nullptr;
        float *mW = nullptr, *vW = nullptr, *mb = nullptr, *vb = nullptr;
        bf16* Wb = nullptr;
    };
    std::vector<Layer> layers;
    float* outw = nullptr;  // per-output loss weights
    float outw_sum = 0.f;
    // activations of a forward pass
    nir::Grown<float> ws;  // splits of products (k_add_splits)
    nir::Grown<bf16> x;
    std::vector<nir::Grown<bf16>> act;  // hidden outputs
    nir::Grown<float> pred;
    // buffers of a backward pass
    nir::Grown<float> tgt;
    nir::Grown<bf16> dy;
    std::vector<nir::Grown<bf16>> grad;  // masked gradients at the hidden outputs
    nir::Grown<float> colsum_ws;         // every layer's chunks, one after another
    nir::Grown<float> part;              // loss partials, loss_blocks() per step
    nir::Grown<float> losses;            // loss per step
    nir::Grown<bf16> ep_x;               // a piece of the epoch's samples in its order
    nir::Grown<float> ep_y;
    nir::Grown<float2> bc;               // Adam's bias corrections of the epoch's steps
    // training set
    int n_data = 0;
    nir::Grown<bf16> data_x;
    nir::Grown<float> data_y;
    nir::Grown<int> perm;
    int64_t adam_t = 0;
    double us_per_step = 0.0, flops_per_step = 0.0;
    nir::Grown<float> stage;  // FP32 staging of uploaded rows
    // output map of nir_mlp_predict_device_affine
    bool gemm_ready[8] = {};  // GEMM kernels prepared for launches
    int* fault = nullptr;     // mapped host memory, set if a wait inside a GEMM gives up
    bool wait_test = false;   // the next products' waits cannot end (nir_mlp_wait_test)
    int aff_n = 0, aff_col = 0;
    double aff_lo = 0.0, aff_hi = 0.0;
    double *aff_scale = nullptr, *aff_shift = nullptr, *aff_out = nullptr;
    std::vector<void*> allocs;

    template <typename T>
    T* alloc(size_t n) {
        void* p = nullptr;
        MLP_CUDA(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
        MLP_CUDA(cudaMemsetAsync(p, 0, std::max<size_t>(n, 1) * sizeof(T), stream));
        allocs.push_back(p);
        return static_cast<T*>(p);
    }
    void release(void* p) {
        for (auto& q : allocs)
            if (q == p) {
                cudaFree(q);
                q = nullptr;
            }
    }
    ~nir_mlp() {
        cudaSetDevice(device);
        if (stream) cudaStreamSynchronize(stream);
        if (fault) fault_flags().give(device, fault);
        for (void* p : allocs)
            if (p) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

void check_mult8(int v, const char* what) {
    if (v <= 0 || v % 8 != 0) throw std::invalid_argument(std::string(what) + " must be a positive multiple of 8");
}

// Arguments of C = op(A) op(B)^T with the given storage (see the file
// header): the splits of K depend on the sizes alone, so the order of the
// sums does not depend on the kernel that takes the product.
GemmArgs gemm_args(const nir_mlp* h, bool a_kmaj, bool b_kmaj, const bf16* A, int lda, const bf16* B, int ldb, int M,
                   int N, int K, int epi, const float* bias, bf16* out_bf, float* out_f, int ldc, const bf16* mask,
                   int ldm) {
    if (K % 8 != 0 || (!a_kmaj && M % 8 != 0) || (!b_kmaj && N % 8 != 0) || lda % 8 != 0 || ldb % 8 != 0)
        throw std::invalid_argument("gemm: contiguous extents must be multiples of 8");
    GemmArgs g{};
    g.A = A;
    g.lda = lda;
    g.B = B;
    g.ldb = ldb;
    g.M = M;
    g.N = N;
    g.K = K;
    g.epi = epi;
    g.bias = bias;
    g.out_bf = out_bf;
    g.out_f = out_f;
    g.ldc = ldc;
    g.mask = mask;
    g.ldm = ldm;
    auto aligned = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; };
    g.wide = (N | ldc | ldm) % 8 == 0 && aligned(bias) && aligned(out_bf) && aligned(out_f) && aligned(mask);
    const int tm = (M + BM - 1) / BM, tn = (N + BN - 1) / BN;
    const int KT = (K + BK - 1) / BK;
    int splits = 1;
    const int want = 2 * h->sms;
    if (tm * tn < want && KT >= 16) splits = std::min(KT / 8, (want + tm * tn - 1) / (tm * tn));
    splits = std::max(splits, 1);
    g.kps = ((KT + splits - 1) / splits) * BK;
    g.splits = (K + g.kps - 1) / g.kps;
    return g;
}

template <typename... P, typename... A>
void launch_early(nir_mlp* h, void (*k)(P...), dim3 grid, int threads, size_t smem, int cluster, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(unsigned(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = h->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = unsigned(cluster);
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    MLP_CUDA(cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...));
}

// The tensor map of an operand of `rows` rows for stages of `tile` of them.
CUtensorMap operand_map(const bf16* P, int ld, int rows, int K, bool kmaj, int tile) {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        MLP_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q));
        if (!f) throw std::runtime_error("the driver has no cuTensorMapEncodeTiled");
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    }();
    CUtensorMap m;
    const cuuint64_t dims[2] = {cuuint64_t(kmaj ? K : rows), cuuint64_t(kmaj ? rows : K)};
    // (the stride of a single row is not used, but checked)
    const cuuint64_t strides[1] = {dims[1] > 1 ? cuuint64_t(ld) * sizeof(bf16) : (dims[0] + 7) / 8 * 16};
    const cuuint32_t box[2] = {64, cuuint32_t(kmaj ? tile : SK)}, one[2] = {1, 1};
    if (encode(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(P), dims, strides, box, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        throw std::invalid_argument("an operand's rows must start at multiples of 16 bytes");
    return m;
}

// How a launch is cut: 128 x tn tiles, of 2^bits or of `parts` CTAs each.
struct GemmPlan {
    double time = 1e300;
    int tn = 64, bits = 0, parts = 0, stages = 0;
    uint32_t tmem = 0;
};
// Estimated time (us) of a group, from runs over M 128..65536, N 16..8192 and
// K 64..52000.  A CTA's start, first load and epilogue take 4 (tn = 64) or 5
// us, a stage of 64 of K 0.4 us with 64 columns; with 128 it takes 0.36 us,
// and 0.5 where two CTAs share an SM.  Splits that one CTA takes one after
// another cost nothing more (1024 x 512 x 512 in two splits: 6.7 us), but
// more CTAs share the stages (512 x 512 x 1024 in four: 9.7 us by one CTA a
// tile, 7.5 by four).  An exchange between the CTAs of a cluster takes 1.5 to
// 2.5 us with an SM for each, 5 to 8 where they share SMs, and the round
// after it loads anew.  Two CTAs fit on an SM unless their tensor memory or
// their stages do not; clusters of 16 fill about half of the SMs, and those
// of 8 and more find an SM for each CTA only while half of the SMs do.
// With few tiles and a long K clusters leave SMs idle and take many rounds;
// a CTA for each split does not, for a second kernel of 2 us and the splits'
// way through L2 (1.4 us per million of them, and 0.04 for each one a sum is
// deep): 256 x 512 x 52000 in 37 splits takes 31 us, 77 at best by clusters,
// 128 x 128 x 65536 in 256 splits 25 against 128, 512 x 512 x 4096 in 16 15
// against 24; but 512 x 512 x 1024 in four 9.2 against 7.6, 2048 x 1024 x
// 16384 in three 109 against 97 by one CTA a tile.
GemmPlan gemm_plan(const nir_mlp* h, const GemmArgs* gs, int count, int splits, int tn, int bits, bool parts) {
    const int ranks = parts ? splits : 1 << bits;
    long long ctas = 0;
    for (int i = 0; i < count; ++i) ctas += (long long)((gs[i].M + 127) / 128) * ((gs[i].N + tn - 1) / tn) * ranks;
    GemmPlan p;
    p.tn = tn;
    p.bits = bits;
    p.parts = parts ? splits : 0;
    p.tmem = tn;
    while (bits == 0 && !parts && p.tmem < uint32_t(tn * splits)) p.tmem *= 2;
    const int slots = bits == RANK_BITS_MAX || 2 * p.tmem > TMEM_COLUMNS ? h->sms : 2 * h->sms;
    // one CTA to an SM, with all of its memory
    const bool alone = ctas <= (bits >= 3 ? h->sms / 2 : h->sms) || 2 * p.tmem > TMEM_COLUMNS;
    p.stages = alone ? 6 : tn == 64 ? 4 : 3;
    const double there = double(std::min<long long>(ctas, slots));
    const double stage = tn == 64 ? 0.4 : alone ? 0.36 : 0.5;
    const double swap = alone ? (tn == 64 ? 0.8 + 0.3 * bits + 0.004 * there : 1.5 + 0.6 * bits + 0.005 * there)
                              : (tn == 64 ? 2.3 + 0.5 * bits + 0.012 * there : 3.0 + 1.5 * bits + 0.03 * there);
    const double again = !alone ? 0.0 : tn == 64 ? 1.0 : 1.8;
    double longest = 0.0, add = 0.0;
    for (int i = 0; i < count; ++i) {
        const double split = (std::min(gs[i].kps, gs[i].K) + SK - 1) / SK * stage;
        const int rounds = (gs[i].splits + ranks - 1) / ranks;
        if (parts) {
            longest = std::max(longest, split);
            add += 1.4e-6 * double(gs[i].splits) * gs[i].M * gs[i].N;
            continue;
        }
        longest = std::max(longest, bits ? rounds * (split + swap) + (rounds - 1) * again : gs[i].splits * split);
    }
    p.time = double((ctas + slots - 1) / slots) * ((tn == 64 ? 4.0 : 5.0) + longest);
    if (parts) p.time += 2.0 + 0.04 * splits + add;
    return p;
}

// Once per handle and kernel that it uses: what a launch may ask for.
template <int TN, bool AK, bool BKM>
void prepare_gemm(nir_mlp* h) {
    bool& ready = h->gemm_ready[(TN == 128) * 4 + AK * 2 + BKM];
    if (ready) return;
    MLP_CUDA(cudaFuncSetAttribute(k_gemm<TN, AK, BKM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  GTile<TN>::smem(STAGES_MAX)));
    MLP_CUDA(cudaFuncSetAttribute(k_gemm<TN, AK, BKM>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    ready = true;
}

// Floats of a product's splits in the workspace, whole 256-byte lines.
size_t parts_len(const GemmArgs& g) { return ((size_t)g.splits * g.M * g.N + 63) / 64 * 64; }

template <int TN, bool AK, bool BKM>
void launch_tiles(nir_mlp* h, const GemmArgs* gs, int count, int splits, const GemmPlan& plan) {
    prepare_gemm<TN, AK, BKM>(h);
    GemmGroup<AK, BKM> G{};
    int tiles = 0;
    for (int i = 0; i < count; ++i) {
        G.g[i].g = gs[i];
        G.g[i].a = operand_map(gs[i].A, gs[i].lda, gs[i].M, gs[i].K, AK, 128);
        G.g[i].b = operand_map(gs[i].B, gs[i].ldb, gs[i].N, gs[i].K, BKM, TN);
        G.first[i] = tiles;
        tiles += ((gs[i].M + 127) / 128) * ((gs[i].N + TN - 1) / TN);
    }
    G.first[count] = tiles;
    G.count = count;
    G.fault = h->fault;
    G.lost = h->wait_test ? 16 : 0;
    G.rank_bits = plan.bits;
    G.parts = plan.parts;
    G.accs = plan.bits || plan.parts ? 1 : splits;
    G.tmem = plan.tmem;
    G.stages = plan.stages;
    if (plan.parts) {
        size_t floats = 0;
        for (int i = 0; i < count; ++i) floats += parts_len(gs[i]);
        float* ws = h->ws.ensure(*h, floats);
        AddTable t;
        t.count = count;
        t.first[0] = 0;
        for (int i = 0; i < count; ++i) {
            const GemmArgs& g = gs[i];
            t.g[i] = g;
            t.ws[i] = ws;
            t.first[i + 1] = t.first[i] + int(((size_t)g.M * g.N + 255) / 256);
            GemmArgs& q = G.g[i].g;
            q.epi = EPI_F32;
            q.out_f = ws;
            q.ldc = g.N;
            q.wide = g.N % 8 == 0;
            ws += parts_len(g);
        }
        launch_early(h, k_gemm<TN, AK, BKM>, dim3(unsigned(tiles * plan.parts)), GTile<TN>::threads,
                     GTile<TN>::smem(G.stages), 1, G);
        launch_early(h, k_add_splits, dim3(unsigned(t.first[count])), 256, 0, 1, t);
    } else {
        launch_early(h, k_gemm<TN, AK, BKM>, dim3(unsigned(tiles) << G.rank_bits), GTile<TN>::threads,
                     GTile<TN>::smem(G.stages), 1 << G.rank_bits, G);
    }
    MLP_LAUNCHED();
}

// Independent products of one storage kind in one launch.
template <bool AK, bool BKM>
void launch_gemm(nir_mlp* h, const GemmArgs* gs, int count) {
    int splits = 1;
    for (int i = 0; i < count; ++i) splits = std::max(splits, gs[i].splits);
    GemmPlan best;
    for (int tn : {64, 128})
        for (int bits = splits * tn > TMEM_COLUMNS; bits == 0 || (bits <= RANK_BITS_MAX && (1 << bits) < 2 * splits);
             ++bits) {
            const GemmPlan p = gemm_plan(h, gs, count, splits, tn, bits, false);
            if (p.time < best.time) best = p;
        }
    if (splits > 1)
        for (int tn : {64, 128}) {
            const GemmPlan p = gemm_plan(h, gs, count, splits, tn, 0, true);
            if (p.time < best.time) best = p;
        }
    if (best.tn == 64) launch_tiles<64, AK, BKM>(h, gs, count, splits, best);
    else launch_tiles<128, AK, BKM>(h, gs, count, splits, best);
}

void gemm(nir_mlp* h, bool a_kmaj, bool b_kmaj, const bf16* A, int lda, const bf16* B, int ldb, int M, int N, int K,
          int epi, const float* bias, bf16* out_bf, float* out_f, int ldc, const bf16* mask, int ldm) {
    if (M <= 0 || N <= 0) return;
    const GemmArgs g =
        gemm_args(h, a_kmaj, b_kmaj, A, lda, B, ldb, M, N, K, epi, bias, out_bf, out_f, ldc, mask, ldm);
    if (a_kmaj && b_kmaj) launch_gemm<true, true>(h, &g, 1);
    else if (a_kmaj && !b_kmaj) launch_gemm<true, false>(h, &g, 1);
    else if (!a_kmaj && !b_kmaj) launch_gemm<false, false>(h, &g, 1);
    else launch_gemm<false, true>(h, &g, 1);
}

// Waits for the stream; an error if a kernel could not finish its work.
void finish(nir_mlp* h) {
    MLP_CUDA(cudaStreamSynchronize(h->stream));
    if (h->fault && *reinterpret_cast<volatile int*>(h->fault)) {
        *h->fault = 0;
        throw std::runtime_error("a wait inside a GEMM kernel gave up");
    }
}

void ensure_rows(nir_mlp* h, int rows) {
    h->x.ensure(*h, (size_t)rows * h->cfg.d_in);
    h->act.resize(size_t(h->cfg.depth));
    for (auto& a : h->act) a.ensure(*h, (size_t)rows * h->cfg.width);
    h->pred.ensure(*h, (size_t)rows * h->cfg.d_out);
}

// The buffers of a backward pass over `rows` samples (a forward pass alone
// needs none of them).
void ensure_backward(nir_mlp* h, int rows) {
    h->tgt.ensure(*h, (size_t)rows * h->cfg.d_out);
    h->dy.ensure(*h, (size_t)rows * h->cfg.d_out);
    h->grad.resize(size_t(h->cfg.depth));
    for (auto& g : h->grad) g.ensure(*h, (size_t)rows * h->cfg.width);
    size_t cols = 0;
    for (auto& ly : h->layers) cols += (size_t)ly.out;
    h->colsum_ws.ensure(*h, (size_t)((rows + kColChunkRows - 1) / kColChunkRows) * cols);
}

void forward(nir_mlp* h, int rows, const bf16* in) {
    const int L = int(h->layers.size());
    for (int l = 0; l < L; ++l) {
        auto& ly = h->layers[l];
        if (l + 1 < L) {
            gemm(h, true, true, in, ly.in, ly.Wb, ly.in, rows, ly.out, ly.in, EPI_BIAS_RELU_BF16, ly.b, h->act[l].p,
                 nullptr, ly.out, nullptr, 0);
            in = h->act[l].p;
        } else {
            gemm(h, true, true, in, ly.in, ly.Wb, ly.in, rows, ly.out, ly.in, EPI_BIAS_F32, ly.b, nullptr, h->pred.p,
                 ly.out, nullptr, 0);
        }
    }
}

unsigned loss_blocks(const nir_mlp* h, int rows) { return grid1d((size_t)rows * h->cfg.d_out, 1024); }

// The losses of `steps` steps of `rows` samples from their partials.
void finish_losses(nir_mlp* h, int rows, int steps) {
    const float denom = float(rows) * std::max(h->outw_sum, 1.f);
    k_sum_partials<<<unsigned(steps), 256, 0, h->stream>>>(int(loss_blocks(h, rows)), h->part.p, 1.f / denom, h->losses.p);
    MLP_LAUNCHED();
}

// The column sums of every layer's output gradient, chunk by chunk.
int colsum_chunks(int rows) { return (rows + kColChunkRows - 1) / kColChunkRows; }
float* colsum_of(nir_mlp* h, int rows, int l) {
    size_t o = 0;
    for (int k = 0; k < l; ++k) o += (size_t)h->layers[k].out;
    return h->colsum_ws.p + o * (size_t)colsum_chunks(rows);
}

// Loss partials (of step `slot`) and dY, the gradients down the layers, then
// every layer's weight gradient in one launch and every bias' column sums in
// another: they depend on nothing after them, and a step's launches, not its
// arithmetic, are what it spends its time on (1024 samples of 16 -> 3 x 512
// -> 8: 258 us with 40 launches, 68 us with 11).
void backward(nir_mlp* h, int rows, const bf16* x, const float* tgt, int slot) {
    const int dout = h->cfg.d_out;
    const float denom = float(rows) * std::max(h->outw_sum, 1.f);
    const unsigned gb = loss_blocks(h, rows);
    launch_early(h, k_loss, dim3(gb), 256, 0, 1, rows, dout, (const float*)h->pred.p, tgt, (const float*)h->outw,
                 2.f / denom, h->dy.p, h->part.p + (size_t)slot * gb);
    const int L = int(h->layers.size());
    auto grad_of = [&](int l) { return l == L - 1 ? h->dy.p : h->grad[l].p; };
    for (int l = L - 1; l > 0; --l) {
        auto& ly = h->layers[l];
        // d(in) = g W, masked by the ReLU of the layer below
        gemm(h, true, false, grad_of(l), ly.out, ly.Wb, ly.in, rows, ly.in, ly.out, EPI_MASK_BF16, nullptr, h->grad[l - 1].p,
             nullptr, ly.in, h->act[l - 1].p, ly.in);
    }
    GemmArgs gs[GROUP_MAX];
    ColsumTable ct{};
    for (int l = 0; l < L; ++l) {
        auto& ly = h->layers[l];
        const bf16* in = (l == 0) ? x : h->act[l - 1].p;
        // dW = g^T in   (out x in), contraction over the rows
        gs[l] = gemm_args(h, false, false, grad_of(l), ly.out, in, ly.in, ly.out, ly.in, rows, EPI_F32, nullptr, nullptr,
                          ly.gW, ly.in, nullptr, 0);
        ct.dy[l] = grad_of(l);
        ct.part[l] = colsum_of(h, rows, l);
        ct.cols[l] = ly.out;
        ct.first[l + 1] = ct.first[l] + colsum_chunks(rows) * ((ly.out + kColsumCols - 1) / kColsumCols);
    }
    launch_gemm<false, false>(h, gs, L);
    ct.count = L;
    ct.rows = rows;
    launch_early(h, k_colsum_part, dim3(unsigned(ct.first[L])), 256, 0, 1, ct);
    MLP_LAUNCHED();
}

void adam(nir_mlp* h, int rows, int slot) {
    AdamTable t{};
    const int L = int(h->layers.size());
    for (int l = 0; l < L; ++l) {
        auto& y = h->layers[l];
        const int nw = y.in * y.out;
        t.l[l] = AdamTable::Layer{y.W, y.gW, y.mW, y.vW, y.b, y.gb, y.mb, y.vb, y.Wb, colsum_of(h, rows, l), nw, y.out};
        t.first[l + 1] = t.first[l] + (nw + y.out + 255) / 256;
    }
    t.count = L;
    t.chunks = colsum_chunks(rows);
    t.bc = h->bc.p + slot;
    t.lr = h->cfg.lr;
    t.b1 = h->cfg.beta1;
    t.b2 = h->cfg.beta2;
    t.eps = h->cfg.eps;
    launch_early(h, k_adam, dim3(unsigned(t.first[L])), 256, 0, 1, t);
    MLP_LAUNCHED();
}

// Host FP32 rows -> device BF16, through a staging buffer that grows on
// demand and is kept (no allocation per call once it is large enough).
void upload_rows(nir_mlp* h, const float* x, int rows, bf16* dst, int cols) {
    const size_t len = (size_t)rows * cols;
    float* const stage = h->stage.ensure(*h, len);
    MLP_CUDA(cudaMemcpyAsync(stage, x, len * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    k_to_bf16<<<grid1d(len), 256, 0, h->stream>>>(len, stage, dst);
    MLP_LAUNCHED();
    finish(h);
}

// An epoch's samples are gathered into its order in pieces of at most this
// size (one step at least): a copy of the whole set would take its memory a
// second time, and a piece that stays in L2 costs two launches in 100 steps.
constexpr size_t kPieceBytes = size_t(32) << 20;

int fail(const std::exception& e, bool input) {
    g_err = e.what();
    return input ? 2 : 3;
}

}  // namespace

extern "C" {

const char* nir_mlp_last_error(void) { return g_err.c_str(); }

int nir_mlp_create(const nir_mlp_config* cfg, int device, nir_mlp** out) {
    if (!cfg || !out) {
        g_err = "null argument";
        return 2;
    }
    *out = nullptr;
    auto h = std::make_unique<nir_mlp>();
    try {
        check_mult8(cfg->d_in, "d_in");
        check_mult8(cfg->width, "width");
        check_mult8(cfg->d_out, "d_out");
        if (cfg->depth < 1 || cfg->depth > 16) throw std::invalid_argument("depth must be in [1, 16]");
        h->cfg = *cfg;
        h->device = device;
        MLP_CUDA(cudaSetDevice(device));
        MLP_CUDA(cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device));
        MLP_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
        h->dims.push_back(cfg->d_in);
        for (int i = 0; i < cfg->depth; ++i) h->dims.push_back(cfg->width);
        h->dims.push_back(cfg->d_out);
        for (size_t l = 0; l + 1 < h->dims.size(); ++l) {
            nir_mlp::Layer ly;
            ly.in = h->dims[l];
            ly.out = h->dims[l + 1];
            const size_t nw = (size_t)ly.in * ly.out;
            ly.W = h->alloc<float>(nw);
            ly.Wb = h->alloc<bf16>(nw);
            ly.gW = h->alloc<float>(nw);
            ly.mW = h->alloc<float>(nw);
            ly.vW = h->alloc<float>(nw);
            ly.b = h->alloc<float>(ly.out);
            ly.gb = h->alloc<float>(ly.out);
            ly.mb = h->alloc<float>(ly.out);
            ly.vb = h->alloc<float>(ly.out);
            // He-uniform for ReLU layers, smaller for the linear output
            const bool last = (l + 2 == h->dims.size());
            const float a = (last ? 0.5f : 1.f) * std::sqrt(6.f / float(ly.in));
            k_init_uniform<<<grid1d(nw), 256, 0, h->stream>>>(nw, cfg->seed * 1315423911ULL + l, a, ly.W, ly.Wb);
            MLP_LAUNCHED();
            h->layers.push_back(ly);
        }
        void* flag = nullptr;
        MLP_CUDA(fault_flags().take(device, &flag));
        h->fault = static_cast<int*>(flag);
        *h->fault = 0;
        h->outw = h->alloc<float>(cfg->d_out);
        std::vector<float> ones(cfg->d_out, 1.f);
        MLP_CUDA(cudaMemcpyAsync(h->outw, ones.data(), ones.size() * sizeof(float), cudaMemcpyHostToDevice, h->stream));
        h->outw_sum = float(cfg->d_out);
        h->losses.ensure(*h, 1024);
        finish(h.get());
    } catch (const std::invalid_argument& e) {
        return fail(e, true);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    *out = h.release();
    return 0;
}

void nir_mlp_free(nir_mlp* h) { delete h; }

int64_t nir_mlp_param_count(const nir_mlp* h) {
    if (!h) return -1;
    int64_t n = 0;
    for (auto& ly : h->layers) n += (int64_t)ly.in * ly.out + ly.out;
    return n;
}

int nir_mlp_get_params(nir_mlp* h, float* out) {
    if (!h || !out) return 2;
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        size_t o = 0;
        for (auto& ly : h->layers) {
            const size_t nw = (size_t)ly.in * ly.out;
            MLP_CUDA(cudaMemcpyAsync(out + o, ly.W, nw * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
            o += nw;
            MLP_CUDA(cudaMemcpyAsync(out + o, ly.b, ly.out * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
            o += ly.out;
        }
        finish(h);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_set_params(nir_mlp* h, const float* in) {
    if (!h || !in) return 2;
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        size_t o = 0;
        for (auto& ly : h->layers) {
            const size_t nw = (size_t)ly.in * ly.out;
            MLP_CUDA(cudaMemcpyAsync(ly.W, in + o, nw * sizeof(float), cudaMemcpyHostToDevice, h->stream));
            k_to_bf16<<<grid1d(nw), 256, 0, h->stream>>>(nw, ly.W, ly.Wb);
            MLP_LAUNCHED();
            o += nw;
            MLP_CUDA(cudaMemcpyAsync(ly.b, in + o, ly.out * sizeof(float), cudaMemcpyHostToDevice, h->stream));
            o += ly.out;
            MLP_CUDA(cudaMemsetAsync(ly.mW, 0, nw * sizeof(float), h->stream));
            MLP_CUDA(cudaMemsetAsync(ly.vW, 0, nw * sizeof(float), h->stream));
            MLP_CUDA(cudaMemsetAsync(ly.mb, 0, ly.out * sizeof(float), h->stream));
            MLP_CUDA(cudaMemsetAsync(ly.vb, 0, ly.out * sizeof(float), h->stream));
        }
        h->adam_t = 0;
        finish(h);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_set_output_weights(nir_mlp* h, const float* w) {
    if (!h || !w) return 2;
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        double s = 0.0;
        for (int i = 0; i < h->cfg.d_out; ++i) {
            if (!(w[i] >= 0.f)) throw std::invalid_argument("output weights must be >= 0");
            s += w[i];
        }
        MLP_CUDA(cudaMemcpyAsync(h->outw, w, h->cfg.d_out * sizeof(float), cudaMemcpyHostToDevice, h->stream));
        finish(h);
        h->outw_sum = float(s);
    } catch (const std::invalid_argument& e) {
        return fail(e, true);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_set_data(nir_mlp* h, const float* x, const float* targets, int32_t n) {
    if (!h || !x || !targets || n < 1) {
        g_err = "invalid arguments";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        const int din = h->cfg.d_in, dout = h->cfg.d_out;
        h->n_data = 0;  // none until the new one is complete
        h->data_x.renew(*h, (size_t)n * din);
        h->data_y.renew(*h, (size_t)n * dout);
        h->perm.renew(*h, size_t(n));
        // in slices so that the FP32 staging buffer stays small
        const int slice = std::max(1, int((size_t(256) << 20) / (sizeof(float) * din)));
        for (int r = 0; r < n; r += slice) {
            const int k = std::min(slice, n - r);
            upload_rows(h, x + (size_t)r * din, k, h->data_x.p + (size_t)r * din, din);
        }
        MLP_CUDA(cudaMemcpyAsync(h->data_y.p, targets, (size_t)n * dout * sizeof(float), cudaMemcpyHostToDevice,
                                 h->stream));
        finish(h);
        h->n_data = n;
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_train(nir_mlp* h, int32_t epochs, int32_t batch, float* epoch_loss) {
    if (!h || epochs < 0 || batch < 8 || batch % 8 != 0) {
        g_err = "invalid arguments (batch must be a positive multiple of 8)";
        return 2;
    }
    if (h->n_data < batch) {
        g_err = "training set smaller than one batch";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        ensure_rows(h, batch);
        ensure_backward(h, batch);
        const int steps = h->n_data / batch;
        h->losses.ensure(*h, size_t(steps));
        h->part.ensure(*h, (size_t)steps * loss_blocks(h, batch));
        const size_t per_step = (size_t)batch * (h->cfg.d_in * sizeof(bf16) + h->cfg.d_out * sizeof(float));
        const int piece = int(std::min<size_t>(size_t(steps), std::max<size_t>(1, kPieceBytes / per_step)));  // steps
        h->ep_x.ensure(*h, (size_t)piece * batch * h->cfg.d_in);
        h->ep_y.ensure(*h, (size_t)piece * batch * h->cfg.d_out);
        std::mt19937_64 rng(h->cfg.seed ^ 0x5bd1e995ULL ^ (uint64_t)h->adam_t);
        std::vector<int> perm(h->n_data);
        std::vector<float> lossv(steps);
        std::vector<float2> bcv(steps);
        h->bc.ensure(*h, size_t(steps));
        cudaEvent_t e0, e1;
        MLP_CUDA(cudaEventCreate(&e0));
        MLP_CUDA(cudaEventCreate(&e1));
        double total_ms = 0.0;
        long long total_steps = 0;
        for (int ep = 0; ep < epochs; ++ep) {
            for (int i = 0; i < h->n_data; ++i) perm[i] = i;
            std::shuffle(perm.begin(), perm.end(), rng);
            MLP_CUDA(cudaMemcpyAsync(h->perm.p, perm.data(), perm.size() * sizeof(int), cudaMemcpyHostToDevice,
                                     h->stream));
            MLP_CUDA(cudaEventRecord(e0, h->stream));
            for (int s = 0; s < steps; ++s) {
                h->adam_t += 1;
                bcv[size_t(s)] = make_float2(1.f - std::pow(h->cfg.beta1, float(h->adam_t)),
                                             1.f - std::pow(h->cfg.beta2, float(h->adam_t)));
            }
            MLP_CUDA(cudaMemcpyAsync(h->bc.p, bcv.data(), bcv.size() * sizeof(float2), cudaMemcpyHostToDevice, h->stream));
            for (int s0 = 0; s0 < steps; s0 += piece) {
                // the piece's samples in the epoch's order, at once
                const int k = std::min(piece, steps - s0), rows = k * batch;
                const int* idx = h->perm.p + (size_t)s0 * batch;
                k_gather_rows<bf16><<<grid1d((size_t)rows * h->cfg.d_in), 256, 0, h->stream>>>(
                    idx, rows, h->cfg.d_in, h->data_x.p, h->ep_x.p);
                k_gather_rows<float><<<grid1d((size_t)rows * h->cfg.d_out), 256, 0, h->stream>>>(
                    idx, rows, h->cfg.d_out, h->data_y.p, h->ep_y.p);
                MLP_LAUNCHED();
                for (int s = 0; s < k; ++s) {
                    const bf16* x = h->ep_x.p + (size_t)s * batch * h->cfg.d_in;
                    forward(h, batch, x);
                    backward(h, batch, x, h->ep_y.p + (size_t)s * batch * h->cfg.d_out, s0 + s);
                    adam(h, batch, s0 + s);
                }
            }
            finish_losses(h, batch, steps);
            MLP_CUDA(cudaEventRecord(e1, h->stream));
            MLP_CUDA(cudaMemcpyAsync(lossv.data(), h->losses.p, steps * sizeof(float), cudaMemcpyDeviceToHost,
                                     h->stream));
            finish(h);
            float ms = 0.f;
            MLP_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            total_ms += ms;
            total_steps += steps;
            if (epoch_loss) {
                double m = 0.0;
                for (float v : lossv) m += v;
                epoch_loss[ep] = float(m / steps);
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (total_steps > 0) h->us_per_step = 1000.0 * total_ms / double(total_steps);
        double f = 0.0;
        for (auto& ly : h->layers) f += 2.0 * double(batch) * ly.in * ly.out;
        // forward, weight gradient, input gradient (none for the first layer)
        h->flops_per_step = 3.0 * f - 2.0 * double(batch) * h->layers[0].in * h->layers[0].out;
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_predict(nir_mlp* h, const float* x, int32_t n, float* y) {
    if (!h || !x || !y || n < 8 || n % 8 != 0) {
        g_err = "invalid arguments (n must be a positive multiple of 8)";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        // one chunk for a whole family member's variables (70,000 at the
        // 20,000 x 50,000 blending size): fewer uploads and synchronisations
        const int chunk = std::min(n, 65536);
        ensure_rows(h, chunk);
        for (int r = 0; r < n; r += chunk) {
            const int k = std::min(chunk, n - r);  // a multiple of 8
            upload_rows(h, x + (size_t)r * h->cfg.d_in, k, h->x.p, h->cfg.d_in);
            forward(h, k, h->x.p);
            MLP_CUDA(cudaMemcpyAsync(y + (size_t)r * h->cfg.d_out, h->pred.p, (size_t)k * h->cfg.d_out * sizeof(float),
                                     cudaMemcpyDeviceToHost, h->stream));
            finish(h);
        }
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_predict_device(nir_mlp* h, const float* x_dev, int32_t n, float* y) {
    if (!h || !x_dev || !y || n < 8 || n % 8 != 0) {
        g_err = "invalid arguments (n must be a positive multiple of 8)";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        const int chunk = std::min(n, 65536);
        ensure_rows(h, chunk);
        for (int r = 0; r < n; r += chunk) {
            const int k = std::min(chunk, n - r);
            const size_t len = (size_t)k * h->cfg.d_in;
            k_to_bf16<<<grid1d(len), 256, 0, h->stream>>>(len, x_dev + (size_t)r * h->cfg.d_in, h->x.p);
            MLP_LAUNCHED();
            forward(h, k, h->x.p);
            MLP_CUDA(cudaMemcpyAsync(y + (size_t)r * h->cfg.d_out, h->pred.p, (size_t)k * h->cfg.d_out * sizeof(float),
                                     cudaMemcpyDeviceToHost, h->stream));
            finish(h);
        }
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_set_affine(nir_mlp* h, int32_t n, int32_t col, double lo, double hi, const double* scale,
                       const double* shift) {
    if (!h || n < 8 || n % 8 != 0 || col < 0 || col >= h->cfg.d_out || !(lo <= hi)) {
        g_err = "invalid arguments (n a positive multiple of 8, 0 <= col < d_out, lo <= hi)";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        for (double** q : {&h->aff_scale, &h->aff_shift, &h->aff_out}) {
            if (*q) h->release(*q);
            *q = nullptr;
        }
        h->aff_out = h->alloc<double>(size_t(n));
        if (scale) {
            h->aff_scale = h->alloc<double>(size_t(n));
            MLP_CUDA(cudaMemcpyAsync(h->aff_scale, scale, size_t(n) * sizeof(double), cudaMemcpyHostToDevice,
                                     h->stream));
        }
        if (shift) {
            h->aff_shift = h->alloc<double>(size_t(n));
            MLP_CUDA(cudaMemcpyAsync(h->aff_shift, shift, size_t(n) * sizeof(double), cudaMemcpyHostToDevice,
                                     h->stream));
        }
        finish(h);
        h->aff_n = n;
        h->aff_col = col;
        h->aff_lo = lo;
        h->aff_hi = hi;
    } catch (const std::exception& e) {
        h->aff_n = 0;
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_predict_device_affine(nir_mlp* h, const float* x_dev, int32_t n, const double** out_dev) {
    if (!h || !x_dev || !out_dev || n < 8 || n % 8 != 0 || n != h->aff_n) {
        g_err = "invalid arguments (n must be the n of nir_mlp_set_affine)";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        const int chunk = std::min(n, 65536);
        ensure_rows(h, chunk);
        for (int r = 0; r < n; r += chunk) {
            const int k = std::min(chunk, n - r);
            const size_t len = (size_t)k * h->cfg.d_in;
            k_to_bf16<<<grid1d(len), 256, 0, h->stream>>>(len, x_dev + (size_t)r * h->cfg.d_in, h->x.p);
            MLP_LAUNCHED();
            forward(h, k, h->x.p);
            k_affine_out<<<unsigned((k + 255) / 256), 256, 0, h->stream>>>(k, r, h->pred.p, h->cfg.d_out, h->aff_col,
                                                                          h->aff_lo, h->aff_hi, h->aff_scale,
                                                                          h->aff_shift, h->aff_out);
            MLP_LAUNCHED();
        }
        finish(h);
        *out_dev = h->aff_out;
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_gradients(nir_mlp* h, const float* x, const float* targets, int32_t n, float* loss, float* grads) {
    if (!h || !x || !targets || n < 8 || n % 8 != 0 || n > 4096) {
        g_err = "invalid arguments (n must be a multiple of 8 in [8, 4096])";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        ensure_rows(h, n);
        ensure_backward(h, n);
        h->losses.ensure(*h, 1);
        h->part.ensure(*h, loss_blocks(h, n));
        upload_rows(h, x, n, h->x.p, h->cfg.d_in);
        MLP_CUDA(cudaMemcpyAsync(h->tgt.p, targets, (size_t)n * h->cfg.d_out * sizeof(float), cudaMemcpyHostToDevice,
                                 h->stream));
        forward(h, n, h->x.p);
        backward(h, n, h->x.p, h->tgt.p, 0);
        finish_losses(h, n, 1);
        for (size_t l = 0; l < h->layers.size(); ++l)
            k_colsum_final<<<(h->layers[l].out + 255) / 256, 256, 0, h->stream>>>(
                colsum_chunks(n), h->layers[l].out, colsum_of(h, n, int(l)), h->layers[l].gb);
        MLP_LAUNCHED();
        float lv = 0.f;
        MLP_CUDA(cudaMemcpyAsync(&lv, h->losses.p, sizeof(float), cudaMemcpyDeviceToHost, h->stream));
        if (grads) {
            size_t o = 0;
            for (auto& ly : h->layers) {
                const size_t nw = (size_t)ly.in * ly.out;
                MLP_CUDA(cudaMemcpyAsync(grads + o, ly.gW, nw * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
                o += nw;
                MLP_CUDA(cudaMemcpyAsync(grads + o, ly.gb, ly.out * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
                o += ly.out;
            }
        }
        finish(h);
        if (loss) *loss = lv;
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_gemm_check(nir_mlp* h, int a_kmaj, int b_kmaj, int32_t M, int32_t N, int32_t K, const float* A,
                       int32_t lda, const float* B, int32_t ldb, float* C) {
    if (!h || !A || !B || !C || M < 1 || N < 1 || K < 1) {
        g_err = "invalid arguments";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        const size_t na = a_kmaj ? (size_t)M * lda : (size_t)K * lda;
        const size_t nb = b_kmaj ? (size_t)N * ldb : (size_t)K * ldb;
        if ((a_kmaj && lda < K) || (!a_kmaj && lda < M) || (b_kmaj && ldb < K) || (!b_kmaj && ldb < N))
            throw std::invalid_argument("leading dimension too small");
        bf16* da = h->alloc<bf16>(na);
        bf16* db = h->alloc<bf16>(nb);
        float* dc = h->alloc<float>((size_t)M * N);
        upload_rows(h, A, 1, da, int(na));
        upload_rows(h, B, 1, db, int(nb));
        gemm(h, a_kmaj != 0, b_kmaj != 0, da, lda, db, ldb, M, N, K, EPI_F32, nullptr, nullptr, dc, N, nullptr, 0);
        MLP_CUDA(cudaMemcpyAsync(C, dc, (size_t)M * N * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
        finish(h);
        h->release(da);
        h->release(db);
        h->release(dc);
    } catch (const std::invalid_argument& e) {
        return fail(e, true);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_wait_test(nir_mlp* h, int32_t M, int32_t N, int32_t K) {
    if (!h || M < 8 || N < 8 || K < 8 || M % 8 || N % 8 || K % 8) {
        g_err = "invalid arguments";
        return 2;
    }
    std::vector<float> a, b, c;
    try {
        a.resize((size_t)M * K);
        b.resize((size_t)N * K);
        c.resize((size_t)M * N);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    h->wait_test = true;
    const int rc = nir_mlp_gemm_check(h, 1, 1, M, N, K, a.data(), K, b.data(), K, c.data());
    h->wait_test = false;
    return rc;
}

int nir_mlp_gemm_time(nir_mlp* h, int32_t M, int32_t N, int32_t K, int32_t reps, double* us) {
    if (!h || !us || M < 8 || N < 8 || K < 8 || M % 8 || N % 8 || K % 8 || reps < 1) {
        g_err = "invalid arguments";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        bf16* a = h->alloc<bf16>((size_t)M * K);
        bf16* b = h->alloc<bf16>((size_t)N * K);
        bf16* c = h->alloc<bf16>((size_t)M * N);
        float* bias = h->alloc<float>(N);
        cudaEvent_t e0, e1;
        MLP_CUDA(cudaEventCreate(&e0));
        MLP_CUDA(cudaEventCreate(&e1));
        gemm(h, true, true, a, K, b, K, M, N, K, EPI_BIAS_RELU_BF16, bias, c, nullptr, N, nullptr, 0);  // warm-up
        MLP_CUDA(cudaEventRecord(e0, h->stream));
        for (int r = 0; r < reps; ++r)
            gemm(h, true, true, a, K, b, K, M, N, K, EPI_BIAS_RELU_BF16, bias, c, nullptr, N, nullptr, 0);
        MLP_CUDA(cudaEventRecord(e1, h->stream));
        MLP_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        MLP_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        *us = 1000.0 * ms / reps;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        h->release(a);
        h->release(b);
        h->release(c);
        h->release(bias);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

int nir_mlp_step_stats(nir_mlp* h, double* us_per_step, double* flops_per_step) {
    if (!h) return 2;
    if (us_per_step) *us_per_step = h->us_per_step;
    if (flops_per_step) *flops_per_step = h->flops_per_step;
    return 0;
}

}  // extern "C"

// ---------------------------------------------------------------- blending-family features

namespace {

__global__ void k_blend_cols(int n, int nf, const float* __restrict__ tmpl, const double* __restrict__ g,
                             const double* __restrict__ f, const double* __restrict__ cost0,
                             const double* __restrict__ atybar, const double* __restrict__ dem_w, double cscale,
                             const long long* __restrict__ rp, const int* __restrict__ ci,
                             const double* __restrict__ val, float* __restrict__ out) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const float* t = tmpl + (size_t)j * nf;
    float* o = out + (size_t)j * nf;
    for (int k = 0; k < nf; ++k) o[k] = t[k];
    const double gj = g[j];
    const double c = cost0[j] * gj;
    double dp = 0.0;
    for (long long q = rp[j]; q < rp[j + 1]; ++q) dp += val[q] * (f[ci[q]] - 1.0);
    o[0] = float((gj - 1.0) / 0.1);
    o[1] = float(c / cscale);
    o[2] = float((c - atybar[j]) / cscale);
    o[6] = float(dp / fmax(dem_w[j], 1e-12) / 0.2);
}

__global__ void k_blend_rows(int m, int nd, int nf, const float* __restrict__ tmpl, const double* __restrict__ f,
                             const double* __restrict__ g, const double* __restrict__ rowlo0,
                             const double* __restrict__ rowup, const double* __restrict__ axbar,
                             const double* __restrict__ bscale, const double* __restrict__ row_abs,
                             const long long* __restrict__ rp, const int* __restrict__ ci,
                             const double* __restrict__ val, float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const float* t = tmpl + (size_t)i * nf;
    float* o = out + (size_t)i * nf;
    for (int k = 0; k < nf; ++k) o[k] = t[k];
    const double lo = (i < nd) ? rowlo0[i] * f[i] : rowlo0[i];
    const double up = rowup[i];
    double gp = 0.0;
    for (long long q = rp[i]; q < rp[i + 1]; ++q) gp += val[q] * (g[ci[q]] - 1.0);
    if (i < nd) o[1] = float((f[i] - 1.0) / 0.2);
    o[4] = float((isfinite(lo) ? axbar[i] - lo : 0.0) / bscale[i]);
    o[5] = float((isfinite(up) ? up - axbar[i] : 0.0) / bscale[i]);
    o[6] = float(gp / fmax(row_abs[i], 1e-12) / 0.1);
}

}  // namespace

struct nir_blend_features {
    int device = 0;
    cudaStream_t stream = nullptr;
    int n = 0, m = 0, nd = 0, nf = 0;
    double cscale = 1.0;
    std::vector<void*> allocs;
    float *col_t = nullptr, *row_t = nullptr, *col_out = nullptr, *row_out = nullptr;
    double *cost0 = nullptr, *atybar = nullptr, *dem_w = nullptr, *dem_val = nullptr;
    double *rowlo0 = nullptr, *rowup = nullptr, *axbar = nullptr, *bscale = nullptr, *row_abs = nullptr,
           *abs_val = nullptr;
    long long *dem_rp = nullptr, *abs_rp = nullptr;
    int *dem_ci = nullptr, *abs_ci = nullptr;
    double *f = nullptr, *g = nullptr;

    template <typename T>
    T* upload(const T* src, size_t count) {
        void* p = nullptr;
        MLP_CUDA(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
        allocs.push_back(p);
        if (src && count) MLP_CUDA(cudaMemcpy(p, src, count * sizeof(T), cudaMemcpyHostToDevice));
        return static_cast<T*>(p);
    }
    ~nir_blend_features() {
        cudaSetDevice(device);
        if (stream) cudaStreamSynchronize(stream);
        for (void* p : allocs) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }
};

extern "C" {

int nir_blend_features_create(const nir_blend_feature_data* d, int32_t device, nir_blend_features** out) {
    if (!d || !out || d->n < 0 || d->m < 0 || d->nd < 0 || d->nd > d->m || d->nf < 7 || !d->col_template ||
        !d->row_template || !d->cost0 || !d->atybar || !d->dem_w || !d->dem_rp || !d->rowlo0 || !d->rowup ||
        !d->axbar || !d->bscale || !d->row_abs || !d->abs_rp) {
        g_err = "invalid blending-feature data";
        return 2;
    }
    *out = nullptr;
    auto h = std::make_unique<nir_blend_features>();
    try {
        const long long dn = d->dem_rp[d->n], an = d->abs_rp[d->m];
        if (dn < 0 || an < 0 || (dn > 0 && (!d->dem_ci || !d->dem_val)) || (an > 0 && (!d->abs_ci || !d->abs_val)))
            throw std::invalid_argument("invalid feature operators");
        for (long long q = 0; q < dn; ++q)
            if (d->dem_ci[q] < 0 || d->dem_ci[q] >= d->nd) throw std::invalid_argument("demand index out of range");
        for (long long q = 0; q < an; ++q)
            if (d->abs_ci[q] < 0 || d->abs_ci[q] >= d->n) throw std::invalid_argument("column index out of range");
        h->device = device;
        MLP_CUDA(cudaSetDevice(device));
        MLP_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
        h->n = d->n;
        h->m = d->m;
        h->nd = d->nd;
        h->nf = d->nf;
        h->cscale = d->cscale;
        const size_t n = size_t(d->n), m = size_t(d->m), nf = size_t(d->nf);
        h->col_t = h->upload(d->col_template, n * nf);
        h->row_t = h->upload(d->row_template, m * nf);
        h->col_out = h->upload<float>(nullptr, n * nf);
        h->row_out = h->upload<float>(nullptr, m * nf);
        h->cost0 = h->upload(d->cost0, n);
        h->atybar = h->upload(d->atybar, n);
        h->dem_w = h->upload(d->dem_w, n);
        h->rowlo0 = h->upload(d->rowlo0, m);
        h->rowup = h->upload(d->rowup, m);
        h->axbar = h->upload(d->axbar, m);
        h->bscale = h->upload(d->bscale, m);
        h->row_abs = h->upload(d->row_abs, m);
        static_assert(sizeof(long long) == sizeof(int64_t), "64-bit offsets");
        h->dem_rp = h->upload(reinterpret_cast<const long long*>(d->dem_rp), n + 1);
        h->dem_ci = h->upload(d->dem_ci, size_t(dn));
        h->dem_val = h->upload(d->dem_val, size_t(dn));
        h->abs_rp = h->upload(reinterpret_cast<const long long*>(d->abs_rp), m + 1);
        h->abs_ci = h->upload(d->abs_ci, size_t(an));
        h->abs_val = h->upload(d->abs_val, size_t(an));
        h->f = h->upload<double>(nullptr, std::max<size_t>(size_t(d->nd), 1));
        h->g = h->upload<double>(nullptr, n);
    } catch (const std::invalid_argument& e) {
        return fail(e, true);
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    *out = h.release();
    return 0;
}

int nir_blend_features_build(nir_blend_features* h, const double* f, const double* g, const float** col_dev,
                             const float** row_dev) {
    if (!h || (!f && h->nd > 0) || (!g && h->n > 0) || !col_dev || !row_dev) {
        g_err = "invalid arguments";
        return 2;
    }
    try {
        MLP_CUDA(cudaSetDevice(h->device));
        cudaStream_t s = h->stream;
        if (h->nd) MLP_CUDA(cudaMemcpyAsync(h->f, f, size_t(h->nd) * sizeof(double), cudaMemcpyHostToDevice, s));
        if (h->n) MLP_CUDA(cudaMemcpyAsync(h->g, g, size_t(h->n) * sizeof(double), cudaMemcpyHostToDevice, s));
        if (h->n)
            k_blend_cols<<<unsigned((h->n + 255) / 256), 256, 0, s>>>(h->n, h->nf, h->col_t, h->g, h->f, h->cost0,
                                                                     h->atybar, h->dem_w, h->cscale, h->dem_rp,
                                                                     h->dem_ci, h->dem_val, h->col_out);
        if (h->m)
            k_blend_rows<<<unsigned((h->m + 255) / 256), 256, 0, s>>>(h->m, h->nd, h->nf, h->row_t, h->f, h->g,
                                                                     h->rowlo0, h->rowup, h->axbar, h->bscale,
                                                                     h->row_abs, h->abs_rp, h->abs_ci, h->abs_val,
                                                                     h->row_out);
        MLP_LAUNCHED();
        MLP_CUDA(cudaStreamSynchronize(s));
        *col_dev = h->col_out;
        *row_dev = h->row_out;
    } catch (const std::exception& e) {
        return fail(e, false);
    }
    return 0;
}

void nir_blend_features_free(nir_blend_features* h) { delete h; }

}  // extern "C"
