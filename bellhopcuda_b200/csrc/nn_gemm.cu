// BF16 GEMM on the 5th-generation tensor cores (sm_100a) for the TL surrogate.
//
//   C[M, N] = epilogue(A[M, K] * B[N, K]^T)      A, B row-major bf16 (K-major)
//
// Either operand may instead be stored as its transpose, [K, M] or [K, N]
// (MN-major): the tensor cores read both layouts, so the backward products need
// no transposed copies. With A transposed, its column sums over K (the bias
// gradient of a weight-gradient product) come from CTAs of the same launch.
//
// One CTA per 128 x 128 or 128 x 32 output tile, 128 threads:
//   warp 0 lane 0  TMA producer: 64-deep bf16 tiles of A and B into a ring of
//                  stages (128-byte swizzle), completion on the stage's "full"
//                  mbarrier (transaction bytes);
//   warp 1         MMA issuer: four tcgen05.mma.kind::f16 (M 128, N the tile's
//                  width, K 16) per K block into an FP32 accumulator in tensor
//                  memory; tcgen05.commit on the stage's "empty" mbarrier frees
//                  the slot, a final commit signals the epilogue;
//   all 4 warps    epilogue: tcgen05.ld of their 32 accumulator lanes (rows),
//                  transposed through the (then idle) stage ring so that a lane
//                  holds 8 columns of a row; bias / GELU / GELU' / conversion on
//                  the way out.
// Wide tiles run three CTAs per SM (64 KiB of shared memory and 128 tensor-memory
// columns each), so that one CTA's epilogue overlaps the others' main loops.
// Every mbarrier wait is bounded; a wait that runs out sets the error word,
// the CTA skips its stores, frees its tensor memory and returns. No TMA load
// uses cluster multicast.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "../../include/bhcb.h"

namespace bhcb {
namespace {

constexpr int BM = 128, BK = 64;
constexpr int GROUP_M = 16;  // tile rows per L2 group of the launch order (8192^3: 1094 -> 1143 TFLOP/s)
constexpr int TILE_A = BM * BK * 2;   // 16 KiB
// Two tile widths. 128 columns, 3 CTAs per SM, for outputs of many tiles; 32
// columns, one CTA per SM with a ring of 160 KiB, for outputs of few: four times
// the CTAs, each bound by its SM's port from L2 (160 rows of 128 bytes per 64 of
// K; 512 x 512 x 32768: 82 us, 128 GB/s per SM). Splitting K would fill the chip
// further, but the accumulator truncates, so at K = 32768 its sum depends on the
// order by 1e-4.
template<int BN> struct Tile {
    static constexpr int KS = BN == 128 ? 1 : 2;       // 64-deep K blocks per stage
    static constexpr int STAGES = BN == 128 ? 2 : 4;
    static constexpr int CTAS = BN == 128 ? 3 : 1;
    static constexpr int TILE_B = BN * BK * 2;
    static constexpr int SMEM_BYTES = STAGES * KS * (TILE_A + TILE_B) + 1024 + 256;
    static constexpr int SUM_STAGES = BN == 128 ? 4 : 8;   // of 128 rows x 64 columns (column_sums)
    // instruction descriptor: FP32 accumulate (bit 4), A and B BF16 (bits 7, 10),
    // transposed A and B (bits 15, 16, set at run time), N >> 3 at bit 17, M >> 4
    // at bit 24
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17)
        | ((uint32_t)(BM >> 4) << 24);
};
constexpr unsigned WAIT_LIMIT = 1u << 24;

__device__ int g_nn_error;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.b32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// false when the wait ran out
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity)
{
    for(unsigned i = 0; i < WAIT_LIMIT; ++i)
        if(mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
                 : "memory");
}
// shared-memory matrix descriptor. K-major: 128-byte rows (64 K) in the 128-byte
// swizzle, groups of 8 rows `sbo` bytes apart. MN-major: rows of 128 (or, for a
// 32-wide tile, 64) bytes of M or N, one per K, groups of 8 K `sbo` bytes apart,
// the next 64 of M or N `lbo` bytes on.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, bool sw64)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)(lbo >> 4) << 16;
    d |= (uint64_t)(sbo >> 4) << 32;
    d |= (uint64_t)1 << 46;                  // descriptor version
    d |= (uint64_t)(sw64 ? 4 : 2) << 61;     // 64- or 128-byte swizzle
    return d;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                 "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}
// 1 in one lane of the (converged) warp
__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "elect.sync _|p, 0xffffffff;\n\t"
                 "selp.b32 %0, 1, 0, p;\n\t}"
                 : "=r"(e));
    return e;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *v)
{
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                   "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
                   "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                   "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for(int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// GELU, tanh form, and its derivative
__device__ __forceinline__ float gelu_f(float x)
{
    const float k = 0.7978845608028654f, c = 0.044715f;
    return 0.5f * x * (1.0f + tanhf(k * (x + c * x * x * x)));
}
__device__ __forceinline__ float dgelu_f(float x)
{
    const float k = 0.7978845608028654f, c = 0.044715f;
    const float u = k * (x + c * x * x * x);
    const float t = tanhf(u);
    return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * k * (1.0f + 3.0f * c * x * x);
}

__device__ __forceinline__ uint4 pack_bf16(const float *x)
{
    __nv_bfloat162 h[4];
#pragma unroll
    for(int i = 0; i < 4; ++i) h[i] = __nv_bfloat162(__float2bfloat16_rn(x[2 * i]), __float2bfloat16_rn(x[2 * i + 1]));
    return *reinterpret_cast<const uint4 *>(h);
}

// db[c] = sum over the K rows of columns [c0, c0 + 64) of A, stored [K][M]: the
// rows one after another in FP32, as one thread per column would add them (the
// weights' later roundings hang on the last bits of these sums). TMA fills the
// ring; two warps add 32 columns each, sixteen rows read ahead of the additions,
// 7 cycles a row in all: 32768 rows in 120 us beside a product of 82
// (a column per thread from global memory took 1915).
template<int BN>
__device__ __forceinline__ void column_sums(uint8_t *ring, uint64_t *full, uint64_t *empty, const CUtensorMap *tmA,
                                            int c0, int M, int K, float *db, int *s_fail)
{
    constexpr int NS = Tile<BN>::SUM_STAGES, BYTES = 128 * 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nk = (K + 127) / 128;
    if(warp == 0 && lane == 0) {
        for(int kb = 0; kb < nk; ++kb) {
            const int s = kb % NS;
            if(kb >= NS && !mbar_wait(&empty[s], (kb / NS - 1) & 1)) {
                *s_fail = 1;
                break;
            }
            mbar_expect_tx(&full[s], BYTES);
            tma_load_2d(ring + s * BYTES, tmA, &full[s], c0, kb * 128);
            tma_load_2d(ring + s * BYTES + BYTES / 2, tmA, &full[s], c0, kb * 128 + 64);
        }
    } else if(warp >= 2) {
        const int col = (warp - 2) * 32 + lane;
        uint32_t at[8];   // of this column in row r: 16-byte chunk c of the row lies at c ^ (r & 7)
#pragma unroll
        for(int r = 0; r < 8; ++r) at[r] = (uint32_t)(r * 128 + (((col >> 3) ^ r) << 4) + (col & 7) * 2);
        float sum = 0.0f;
        uint32_t v[2][16];
        auto read = [&](int stage, int g, uint32_t *o) {
            const uint8_t *t = ring + stage * BYTES + g * 2048;
#pragma unroll
            for(int r = 0; r < 16; ++r)
                o[r] = *reinterpret_cast<const unsigned short *>(t + (r >> 3) * 1024 + at[r & 7]);
        };
        int s = 0;
        uint32_t parity = 0;
        bool ok = mbar_wait(&full[0], 0);
        if(ok) read(0, 0, v[0]);
        for(int kb = 0; ok && kb < nk; ++kb) {
            const int next = s + 1 == NS ? 0 : s + 1;
            if(next == 0) parity ^= 1;
#pragma unroll
            for(int g = 0; g < 8; ++g) {
                if(g < 7) {
                    read(s, g + 1, v[(g + 1) & 1]);
                } else if(kb + 1 < nk) {
                    ok = mbar_wait(&full[next], parity);
                    if(ok) read(next, 0, v[0]);
                }
#pragma unroll
                for(int r = 0; r < 16; ++r) sum += __uint_as_float(v[g & 1][r] << 16);   // rows past K are +0
            }
            __syncwarp();
            if(lane == 0) mbar_arrive(&empty[s]);
            s = next;
        }
        if(!ok) {
            *s_fail = 1;
            return;
        }
        if(c0 + col < M) db[c0 + col] = sum;
    }
}

// vec: rows of C, aux_in and aux_out, and bias, may be accessed 16 bytes at a time.
// a_mn, b_mn: A, B stored [K][M], [K][N]. colsum (a_mn only): blocks of
// blockIdx.z 0 are its CTAs, the product's are the next layer.
template<int EPI, int BN>
__global__ void __launch_bounds__(128, Tile<BN>::CTAS)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N,
                   int K, void *C, const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ aux_in,
                   __nv_bfloat16 *aux_out, int vec, int a_mn, int b_mn, float *colsum)
{
    constexpr int STAGES = Tile<BN>::STAGES, KS = Tile<BN>::KS, TILE_B = Tile<BN>::TILE_B;
    extern __shared__ uint8_t smem_raw[];
    // (an offset, so that accesses stay shared-memory ones)
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *sA = smem;
    uint8_t *sB = smem + STAGES * KS * TILE_A;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * KS * (TILE_A + TILE_B));
    constexpr int BARS = Tile<BN>::SUM_STAGES > STAGES ? Tile<BN>::SUM_STAGES : STAGES;
    uint64_t *empty = full + BARS;
    uint64_t *done = empty + BARS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int s_fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if(colsum && blockIdx.z == 0) {
        const int c0 = 64 * ((int)blockIdx.y * (int)gridDim.x + (int)blockIdx.x);
        if(c0 >= M) return;
        if(threadIdx.x == 0) {
            s_fail = 0;
            for(int s = 0; s < Tile<BN>::SUM_STAGES; ++s) {
                mbar_init(&full[s], 1);
                mbar_init(&empty[s], 2);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        column_sums<BN>(smem, full, empty, &tmA, c0, M, K, colsum, &s_fail);
        __syncthreads();
        if(threadIdx.x == 0 && s_fail) atomicExch(&g_nn_error, 1);
        return;
    }
    // Tile order: the launch order walks groups of GROUP_M tile rows, a column
    // of GROUP_M tiles at a time, so the CTAs resident together share GROUP_M
    // panels of A and a band of B panels that fit in L2 (instead of every B
    // panel against a few A rows).
    int m_t, n_t;
    {
        const int num_m = (int)gridDim.y, num_n = (N + BN - 1) / BN;
        const int t = (int)blockIdx.y * (int)gridDim.x + (int)blockIdx.x;
        if(t >= num_m * num_n) return;   // a layer widened for the column sums
        const int per_group = GROUP_M * num_n;
        const int first_m = (t / per_group) * GROUP_M;
        const int gsz = min(num_m - first_m, GROUP_M);
        const int r = t - (t / per_group) * per_group;
        m_t = first_m + r % gsz;
        n_t = r / gsz;
    }
    const int m0 = m_t * BM, n0 = n_t * BN;
    const int nk = (K + KS * BK - 1) / (KS * BK);
    if(threadIdx.x == 0) {
        s_fail = 0;
        for(int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if(warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if(warp == 0 && lane == 0) {
        // ---- producer (a block past K reads as zero)
        for(int kb = 0; kb < nk; ++kb) {
            const int s = kb % STAGES, round = kb / STAGES;
            if(kb >= STAGES && !mbar_wait(&empty[s], (round - 1) & 1)) {
                s_fail = 1;
                break;
            }
            mbar_expect_tx(&full[s], KS * (TILE_A + TILE_B));
#pragma unroll
            for(int j = 0; j < KS; ++j) {
                const int k0 = (kb * KS + j) * BK;
                uint8_t *a = sA + (s * KS + j) * TILE_A, *b = sB + (s * KS + j) * TILE_B;
                if(a_mn) {
                    tma_load_2d(a, &tmA, &full[s], m0, k0);
                    tma_load_2d(a + TILE_A / 2, &tmA, &full[s], m0 + 64, k0);
                } else {
                    tma_load_2d(a, &tmA, &full[s], k0, m0);
                }
                if(b_mn) {
                    tma_load_2d(b, &tmB, &full[s], n0, k0);
                    if(BN == 128) tma_load_2d(b + TILE_B / 2, &tmB, &full[s], n0 + 64, k0);
                } else {
                    tma_load_2d(b, &tmB, &full[s], k0, n0);
                }
            }
        }
    } else if(warp == 1) {
        // ---- MMA issuer: the whole warp walks the loop, so that descriptors are
        // warp-uniform, and one elected lane issues. In a lane's own branch each
        // descriptor crossed to the uniform registers on its own: 600 cycles per
        // K block of 64 whatever the tile, now 250
        bool ok = true;
        const uint32_t issue = elect_one();
        const uint64_t dA = make_desc(smem_u32(sA), a_mn ? TILE_A / 2 : 16, 1024, false);
        const uint64_t dB = b_mn && BN == 32 ? make_desc(smem_u32(sB), 16, 512, true)
                                             : make_desc(smem_u32(sB), b_mn ? TILE_B / 2 : 16, 1024, false);
        // a K step of 16, in the descriptors' units of 16 bytes: 32 bytes along a
        // K-major row, or 16 rows
        const int ka = a_mn ? 128 : 2, kbs = b_mn ? (BN == 32 ? 64 : 128) : 2;
        const uint32_t idesc = Tile<BN>::IDESC | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16);
        int s = 0;
        uint32_t parity = 0;
        for(int kb = 0; kb < nk; ++kb) {
            if(!mbar_wait(&full[s], parity)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t a0 = dA + (uint64_t)(s * KS * (TILE_A >> 4)), b0 = dB + (uint64_t)(s * KS * (TILE_B >> 4));
            if(issue) {
#pragma unroll
                for(int k = 0; k < KS * 4; ++k)
                    umma_bf16(tmem, a0 + (k & 3) * ka + (k >> 2) * (TILE_A >> 4),
                              b0 + (k & 3) * kbs + (k >> 2) * (TILE_B >> 4), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(&empty[s]);
            }
            __syncwarp();
            if(++s == STAGES) {
                s = 0;
                parity ^= 1;
            }
        }
        if(!ok) s_fail = 1;
        if(issue) umma_commit(done);   // arrives once every MMA issued so far has completed
    }
    // ---- epilogue: lane l of a warp handles columns 8 (l & 3) ... + 7 of rows
    // (l >> 2) + 8 it of each 32 x 32 chunk, as one 16-byte access per operand
    // (two for FP32): the rows' loads are in flight before their first use. One
    // 2-byte access per element and four rows in flight cost the trunk's dGELU
    // products (32768 x 512 x 512) 175 us, with this 50.
    const int q = (lane & 3) * 8, r8 = lane >> 2;
    uint4 aux[4];
    auto load_aux = [&](int c) {
#pragma unroll
        for(int it = 0; it < 4; ++it) {
            const int row = m0 + warp * 32 + it * 8 + r8, col = n0 + c * 32 + q;
            aux[it] = make_uint4(0u, 0u, 0u, 0u);
            if(row < M && col < N) aux[it] = *reinterpret_cast<const uint4 *>(aux_in + (size_t)row * N + col);
        }
    };
    __syncwarp();
    if(EPI == BHCB_NN_EPI_BF16_DGELU && vec) load_aux(0);
    const bool ready = mbar_wait(done, 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    const bool good = ready && s_fail == 0;
    if(!good && threadIdx.x == 0) atomicExch(&g_nn_error, 1);
    if(good) {
        // every MMA has completed, so the stage ring is free: each warp stages
        // its 32 rows x 32 columns through shared memory
        float *stage = reinterpret_cast<float *>(smem) + warp * (32 * 33);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // after the ring's async-proxy use
#pragma unroll 1
        for(int c = 0; c < BN / 32; ++c) {
            float v[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 32), v);
#pragma unroll
            for(int j = 0; j < 32; ++j) stage[lane * 33 + j] = v[j];
            __syncwarp();
            const int col = n0 + c * 32 + q;
            const int ncol = N - col;   // columns of this lane's eight that exist
            float b[8];
#pragma unroll
            for(int k = 0; k < 8; ++k) b[k] = bias && k < ncol ? bias[col + k] : 0.0f;
            uint4 cur[4];
#pragma unroll
            for(int it = 0; it < 4; ++it) cur[it] = aux[it];
            if(EPI == BHCB_NN_EPI_BF16_DGELU && vec && c + 1 < BN / 32) load_aux(c + 1);
#pragma unroll
            for(int it = 0; it < 4; ++it) {
                const int row = m0 + warp * 32 + it * 8 + r8;
                if(row >= M || ncol <= 0) continue;
                const size_t idx = (size_t)row * N + col;
                float x[8], y[8];
#pragma unroll
                for(int k = 0; k < 8; ++k) x[k] = stage[(it * 8 + r8) * 33 + q + k] + b[k];
                if(EPI == BHCB_NN_EPI_BF16_DGELU) {
                    const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&cur[it]);
#pragma unroll
                    for(int k = 0; k < 8; ++k) {
                        const float acc = stage[(it * 8 + r8) * 33 + q + k];
                        float pre = 0.0f;
                        if(vec) pre = __bfloat162float(h[k]);
                        else if(k < ncol) pre = __bfloat162float(aux_in[idx + k]);
                        y[k] = acc * dgelu_f(pre);
                    }
                } else {
#pragma unroll
                    for(int k = 0; k < 8; ++k) y[k] = EPI == BHCB_NN_EPI_BF16_GELU ? gelu_f(x[k]) : x[k];
                }
                if(EPI == BHCB_NN_EPI_F32) {
                    float *o = reinterpret_cast<float *>(C) + idx;
                    if(vec) {
                        reinterpret_cast<float4 *>(o)[0] = make_float4(y[0], y[1], y[2], y[3]);
                        reinterpret_cast<float4 *>(o)[1] = make_float4(y[4], y[5], y[6], y[7]);
                    } else {
#pragma unroll
                        for(int k = 0; k < 8; ++k)
                            if(k < ncol) o[k] = y[k];
                    }
                    continue;
                }
                __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(C) + idx;
                const bool keep = EPI == BHCB_NN_EPI_BF16_GELU && aux_out != nullptr;
                if(vec) {
                    if(keep) *reinterpret_cast<uint4 *>(aux_out + idx) = pack_bf16(x);
                    *reinterpret_cast<uint4 *>(o) = pack_bf16(y);
                } else {
#pragma unroll
                    for(int k = 0; k < 8; ++k)
                        if(k < ncol) {
                            if(keep) aux_out[idx + k] = __float2bfloat16_rn(x[k]);
                            o[k] = __float2bfloat16_rn(y[k]);
                        }
                }
            }
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if(warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN));
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if(!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess
           && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// rows x cols row-major bf16, boxes of box_rows x box_cols, swizzled by their
// width, out-of-range elements read as zero
bool make_map(CUtensorMap *map, const void *ptr, int rows, int cols, int box_rows, int box_cols)
{
    EncodeTiledFn enc = encode_fn();
    if(!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct GemmArgs {
    CUtensorMap ma, mb;
    int M, N, K;
    void *C;
    const float *bias;
    const __nv_bfloat16 *aux_in;
    __nv_bfloat16 *aux_out;
    int vec, a_mn, b_mn;
    float *colsum;
};

template<int EPI, int BN> void launch_gemm(const GemmArgs &g, cudaStream_t st)
{
    static bool done = false;
    if(!done) {
        cudaFuncSetAttribute(gemm_tc_kernel<EPI, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Tile<BN>::SMEM_BYTES);
        done = true;
    }
    // with column sums, a layer of blocks before the product's: two or more for each
    // 128 columns of A, of which ceil(M / 64) have work
    dim3 grid((g.N + BN - 1) / BN, (g.M + BM - 1) / BM);
    if(g.colsum) {
        grid.x = grid.x < 2 ? 2 : grid.x;
        grid.z = 2;
    }
    gemm_tc_kernel<EPI, BN><<<grid, 128, Tile<BN>::SMEM_BYTES, st>>>(g.ma, g.mb, g.M, g.N, g.K, g.C, g.bias, g.aux_in,
                                                                    g.aux_out, g.vec, g.a_mn, g.b_mn, g.colsum);
}

template<int BN> bool launch_epi(int epi, const GemmArgs &g, cudaStream_t st)
{
    switch(epi) {
    case BHCB_NN_EPI_F32: launch_gemm<BHCB_NN_EPI_F32, BN>(g, st); return true;
    case BHCB_NN_EPI_BF16: launch_gemm<BHCB_NN_EPI_BF16, BN>(g, st); return true;
    case BHCB_NN_EPI_BF16_GELU: launch_gemm<BHCB_NN_EPI_BF16_GELU, BN>(g, st); return true;
    case BHCB_NN_EPI_BF16_DGELU: launch_gemm<BHCB_NN_EPI_BF16_DGELU, BN>(g, st); return true;
    default: return false;
    }
}

} // namespace
} // namespace bhcb

using namespace bhcb;

extern "C" int bhcb_nn_gemm_t(const void *A, const void *B, void *C, int32_t M, int32_t N, int32_t K, int32_t a_t,
                              int32_t b_t, int32_t epi, const float *bias, const void *aux_in, void *aux_out,
                              float *colsum, void *stream)
{
    if(!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return BHCB_ERR_ARG;
    // TMA: 16-byte aligned bases and row strides (a multiple of 8 bf16)
    if((K % 8) != 0 || (a_t && M % 8) || (b_t && N % 8) || (reinterpret_cast<uintptr_t>(A) & 15)
       || (reinterpret_cast<uintptr_t>(B) & 15))
        return BHCB_ERR_ARG;
    if(epi == BHCB_NN_EPI_BF16_DGELU && !aux_in) return BHCB_ERR_ARG;
    if(colsum && !a_t) return BHCB_ERR_ARG;
    // narrow tiles while one wave of them covers the output (148 SMs). At K = 1024,
    // wide and narrow: 128 tiles of 32 columns 19 and 13 us, 256 tiles 19 and 21 us
    const int bn = (long long)((M + BM - 1) / BM) * ((N + 31) / 32) <= 148 ? 32 : 128;
    GemmArgs g{};
    if(!(a_t ? make_map(&g.ma, A, K, M, BK, 64) : make_map(&g.ma, A, M, K, BM, BK))
       || !(b_t ? make_map(&g.mb, B, K, N, BK, bn == 32 ? 32 : 64) : make_map(&g.mb, B, N, K, bn, BK)))
        return BHCB_ERR_CUDA;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(bias)
        | reinterpret_cast<uintptr_t>(aux_in) | reinterpret_cast<uintptr_t>(aux_out);
    g.M = M;
    g.N = N;
    g.K = K;
    g.C = C;
    g.bias = bias;
    g.aux_in = reinterpret_cast<const __nv_bfloat16 *>(aux_in);
    g.aux_out = reinterpret_cast<__nv_bfloat16 *>(aux_out);
    g.vec = N % 8 == 0 && (bases & 15) == 0;
    g.a_mn = a_t != 0;
    g.b_mn = b_t != 0;
    g.colsum = colsum;
    const cudaStream_t st = (cudaStream_t)stream;
    if(!(bn == 32 ? launch_epi<32>(epi, g, st) : launch_epi<128>(epi, g, st))) return BHCB_ERR_ARG;
    return cudaGetLastError() == cudaSuccess ? BHCB_OK : BHCB_ERR_CUDA;
}

extern "C" int bhcb_nn_gemm(const void *A, const void *B, void *C, int32_t M, int32_t N, int32_t K, int32_t epi,
                            const float *bias, const void *aux_in, void *aux_out, void *stream)
{
    return bhcb_nn_gemm_t(A, B, C, M, N, K, 0, 0, epi, bias, aux_in, aux_out, nullptr, stream);
}

extern "C" int bhcb_nn_status(int32_t *error, int32_t clear)
{
    int v = 0;
    if(cudaMemcpyFromSymbol(&v, g_nn_error, sizeof v) != cudaSuccess) return BHCB_ERR_CUDA;
    if(error) *error = v;
    if(clear) {
        int z = 0;
        if(cudaMemcpyToSymbol(g_nn_error, &z, sizeof z) != cudaSuccess) return BHCB_ERR_CUDA;
    }
    return BHCB_OK;
}
