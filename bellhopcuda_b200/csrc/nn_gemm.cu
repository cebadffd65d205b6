// BF16 GEMM on the 5th-generation tensor cores (sm_100a) for the TL surrogate.
//
//   C[M, N] = epilogue(A[M, K] * B[N, K]^T)      A, B row-major bf16 (K-major)
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
// K; 512 x 512 x 32768: 72 us, 145 GB/s per SM). Splitting K would fill the chip
// further, but the accumulator truncates, so at K = 32768 its sum depends on the
// order by 1e-4.
template<int BN> struct Tile {
    static constexpr int KS = BN == 128 ? 1 : 2;       // 64-deep K blocks per stage
    static constexpr int STAGES = BN == 128 ? 2 : 4;
    static constexpr int CTAS = BN == 128 ? 3 : 1;
    static constexpr int TILE_B = BN * BK * 2;
    static constexpr int SMEM_BYTES = STAGES * KS * (TILE_A + TILE_B) + 1024 + 256;
    // instruction descriptor: FP32 accumulate (bit 4), A and B BF16 (bits 7, 10),
    // both K-major, N >> 3 at bit 17, M >> 4 at bit 24
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
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
                 : "memory");
}
// shared-memory matrix descriptor of a K-major tile with 128-byte rows in the
// 128-byte swizzle (8-row groups 1024 bytes apart)
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;             // leading byte offset (unused when swizzled)
    d |= (uint64_t)(1024 >> 4) << 32;   // stride byte offset
    d |= (uint64_t)1 << 46;             // descriptor version
    d |= (uint64_t)2 << 61;             // 128-byte swizzle
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

// vec: rows of C, aux_in and aux_out, and bias, may be accessed 16 bytes at a time
template<int EPI, int BN>
__global__ void __launch_bounds__(128, Tile<BN>::CTAS)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N,
                   int K, void *C, const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ aux_in,
                   __nv_bfloat16 *aux_out, int vec)
{
    constexpr int STAGES = Tile<BN>::STAGES, KS = Tile<BN>::KS, TILE_B = Tile<BN>::TILE_B;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem;
    uint8_t *sB = smem + STAGES * KS * TILE_A;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * KS * (TILE_A + TILE_B));
    uint64_t *empty = full + STAGES;
    uint64_t *done = empty + STAGES;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int s_fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Tile order: the launch order walks groups of GROUP_M tile rows, a column
    // of GROUP_M tiles at a time, so the CTAs resident together share GROUP_M
    // panels of A and a band of B panels that fit in L2 (instead of every B
    // panel against a few A rows).
    int m_t, n_t;
    {
        const int num_m = (int)gridDim.y, num_n = (int)gridDim.x;
        const int t = (int)blockIdx.y * num_n + (int)blockIdx.x;
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
                tma_load_2d(sA + (s * KS + j) * TILE_A, &tmA, &full[s], (kb * KS + j) * BK, m0);
                tma_load_2d(sB + (s * KS + j) * TILE_B, &tmB, &full[s], (kb * KS + j) * BK, n0);
            }
        }
    } else if(warp == 1) {
        // ---- MMA issuer: the whole warp walks the loop, so that descriptors are
        // warp-uniform, and one elected lane issues. In a lane's own branch each
        // descriptor crossed to the uniform registers on its own: 600 cycles per
        // K block of 64 whatever the tile, now 250
        bool ok = true;
        const uint32_t issue = elect_one();
        const uint64_t dA = sw128_desc(smem_u32(sA)), dB = sw128_desc(smem_u32(sB));
        int s = 0;
        uint32_t parity = 0;
        for(int kb = 0; kb < nk; ++kb) {
            if(!mbar_wait(&full[s], parity)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // descriptors count in 16 bytes: 32 along a swizzled row per K step of 16
            const uint64_t a0 = dA + (uint64_t)(s * KS * (TILE_A >> 4)), b0 = dB + (uint64_t)(s * KS * (TILE_B >> 4));
            if(issue) {
#pragma unroll
                for(int k = 0; k < KS * 4; ++k)
                    umma_bf16(tmem, a0 + (k & 3) * 2 + (k >> 2) * (TILE_A >> 4),
                              b0 + (k & 3) * 2 + (k >> 2) * (TILE_B >> 4), Tile<BN>::IDESC,
                              (kb > 0 || k > 0) ? 1u : 0u);
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

// rows x K row-major bf16, boxes of 64 columns x box_rows rows, 128-byte swizzle,
// out-of-range elements read as zero
bool make_map(CUtensorMap *map, const void *ptr, int rows, int K, int box_rows)
{
    EncodeTiledFn enc = encode_fn();
    if(!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template<int EPI, int BN>
void launch_gemm(const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int K, void *C, const float *bias,
                 const __nv_bfloat16 *ai, __nv_bfloat16 *ao, int vec, cudaStream_t st)
{
    static bool done = false;
    if(!done) {
        cudaFuncSetAttribute(gemm_tc_kernel<EPI, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Tile<BN>::SMEM_BYTES);
        done = true;
    }
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    gemm_tc_kernel<EPI, BN><<<grid, 128, Tile<BN>::SMEM_BYTES, st>>>(ma, mb, M, N, K, C, bias, ai, ao, vec);
}

template<int BN>
bool launch_epi(int epi, const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int K, void *C, const float *bias,
                const __nv_bfloat16 *ai, __nv_bfloat16 *ao, int vec, cudaStream_t st)
{
    switch(epi) {
    case BHCB_NN_EPI_F32: launch_gemm<BHCB_NN_EPI_F32, BN>(ma, mb, M, N, K, C, bias, ai, ao, vec, st); return true;
    case BHCB_NN_EPI_BF16: launch_gemm<BHCB_NN_EPI_BF16, BN>(ma, mb, M, N, K, C, bias, ai, ao, vec, st); return true;
    case BHCB_NN_EPI_BF16_GELU:
        launch_gemm<BHCB_NN_EPI_BF16_GELU, BN>(ma, mb, M, N, K, C, bias, ai, ao, vec, st);
        return true;
    case BHCB_NN_EPI_BF16_DGELU:
        launch_gemm<BHCB_NN_EPI_BF16_DGELU, BN>(ma, mb, M, N, K, C, bias, ai, ao, vec, st);
        return true;
    default: return false;
    }
}

} // namespace
} // namespace bhcb

using namespace bhcb;

extern "C" int bhcb_nn_gemm(const void *A, const void *B, void *C, int32_t M, int32_t N, int32_t K, int32_t epi,
                            const float *bias, const void *aux_in, void *aux_out, void *stream)
{
    if(!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return BHCB_ERR_ARG;
    // TMA: 16-byte aligned bases and row strides (K a multiple of 8 bf16)
    if((K % 8) != 0 || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15))
        return BHCB_ERR_ARG;
    if(epi == BHCB_NN_EPI_BF16_DGELU && !aux_in) return BHCB_ERR_ARG;
    // narrow tiles while one wave of them covers the output (148 SMs). At K = 1024,
    // wide and narrow: 128 tiles of 32 columns 19 and 13 us, 256 tiles 19 and 21 us
    const int bn = (long long)((M + BM - 1) / BM) * ((N + 31) / 32) <= 148 ? 32 : 128;
    CUtensorMap ma, mb;
    if(!make_map(&ma, A, M, K, BM) || !make_map(&mb, B, N, K, bn)) return BHCB_ERR_CUDA;
    const __nv_bfloat16 *ai = reinterpret_cast<const __nv_bfloat16 *>(aux_in);
    __nv_bfloat16 *ao = reinterpret_cast<__nv_bfloat16 *>(aux_out);
    const uintptr_t bases = reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(bias)
        | reinterpret_cast<uintptr_t>(aux_in) | reinterpret_cast<uintptr_t>(aux_out);
    const int vec = N % 8 == 0 && (bases & 15) == 0;
    const cudaStream_t st = (cudaStream_t)stream;
    if(!(bn == 32 ? launch_epi<32>(epi, ma, mb, M, N, K, C, bias, ai, ao, vec, st)
                  : launch_epi<128>(epi, ma, mb, M, N, K, C, bias, ai, ao, vec, st)))
        return BHCB_ERR_ARG;
    return cudaGetLastError() == cudaSuccess ? BHCB_OK : BHCB_ERR_CUDA;
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
