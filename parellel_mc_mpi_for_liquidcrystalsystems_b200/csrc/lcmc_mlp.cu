// lcmc_mlp.cu - the volume-move surrogate: a 4097 -> 128 -> 128 -> 1 MLP with
// BF16 weights/activations and FP32 accumulation, trained and evaluated on the
// GPU by this file's kernels.  The matrix products run on the 5th-generation
// tensor cores (tcgen05.mma, accumulators in TMEM); bias, activation, loss and
// Adam are small FP32 CUDA-core kernels.  (No reference counterpart: the
// reference has no NPT move at all, MCnptColloid.c:3978.)
#include <cuda.h> // CUtensorMap and its enums (the encoder is taken from the driver at run time)
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <math.h>
#include <stdio.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

#include "../../include/lcmc.h"
#include "lcmc_rng.cuh"
#include "lcmc_tc.cuh"

namespace lcmc {

using bf16 = __nv_bfloat16;

// ---------------------------------------------------------------------------
// C[M x N] (FP32, row-major) (+)= A[M x K] * B[N x K]^T; A, B BF16 row-major
// with K contiguous (lda, ldb in elements, multiples of 8), K a multiple of 64.
// CTA = 128 threads per 128 x BN output tile (BN = 128, or 64 when 128-wide
// tiles would leave most SMs idle).  The K loop runs over 64-wide slices
// through a GT_STAGES-deep ring of shared-memory stages filled by cp.async
// (16-byte copies, zero-filled beyond M and N) in the K-major core-matrix
// layout (8 rows x 16 bytes per core matrix, K halves 128 B apart, 8-row
// groups 1024 B apart).  One elected thread issues the slice's four
// 128 x BN x 16 tcgen05 MMAs and commits them to the stage's mbarrier; a stage
// is refilled once the MMAs that read it have completed, so GT_STAGES - 1
// slices of loads are in flight while the tensor core works.  The accumulator
// lives in BN TMEM columns and is read back with tcgen05.ld (warp w owns TMEM
// lanes 32w..32w+31 = rows).  Waits are bounded: on a timeout the tile sets
// *err, lets its copies and MMAs in flight finish and frees its TMEM.
// ---------------------------------------------------------------------------
constexpr int GT_M = 128, GT_K = 64, GT_STAGES = 4;
// mbarrier tries before a wait gives up (lcmc_set_wait_limit lowers it for tests)
constexpr uint32_t kWaitIters = 1u << 24;
static uint32_t g_wait_iters = kWaitIters;

template <int BN> struct GemmShape {
    static constexpr int A_BYTES = GT_M * GT_K * 2, B_BYTES = BN * GT_K * 2, STAGE = A_BYTES + B_BYTES;
    static constexpr int SMEM = GT_STAGES * STAGE;
};

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int src_bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(smem)), "l"(gmem),
                 "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int NPEND> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(NPEND) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Slice kt of A (128 rows from m0) and B (BN rows from n0) into one stage (sA, sB).
template <int BN>
__device__ __forceinline__ void gemm_load_slice(unsigned char *sA, unsigned char *sB, const bf16 *__restrict__ A,
                                                int lda, const bf16 *__restrict__ B, int ldb, int M, int N, int m0,
                                                int n0, int kt, int t)
{
    const int k0 = kt * GT_K;
#pragma unroll
    for (int i = 0; i < GT_M * 8 / 128; i++) {
        const int v = t + 128 * i;
        const int row = v >> 3, ch = v & 7;
        const int off = ((row >> 3) * 8 + ch) * 128 + (row & 7) * 16;
        const int gm = m0 + row;
        const bool in = gm < M;
        cp_async16(sA + off, in ? (const void *)(A + (size_t)gm * lda + k0 + ch * 8) : (const void *)A, in ? 16 : 0);
    }
#pragma unroll
    for (int i = 0; i < BN * 8 / 128; i++) {
        const int v = t + 128 * i;
        const int row = v >> 3, ch = v & 7;
        const int off = ((row >> 3) * 8 + ch) * 128 + (row & 7) * 16;
        const int gn = n0 + row;
        const bool in = gn < N;
        cp_async16(sB + off, in ? (const void *)(B + (size_t)gn * ldb + k0 + ch * 8) : (const void *)B, in ? 16 : 0);
    }
}

template <int BN>
__global__ void __launch_bounds__(128) k_gemm_tc(const bf16 *__restrict__ A, int lda, const bf16 *__restrict__ B,
                                                 int ldb, float *__restrict__ C, int ldc, int M, int N, int K,
                                                 int accumulate, int *err, uint32_t wait_iters)
{
    using G = GemmShape<BN>;
    constexpr int S = GT_STAGES;
    extern __shared__ __align__(1024) unsigned char gsm[];
    __shared__ __align__(8) uint64_t bar[S];
    __shared__ uint32_t tmem_base;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int m0 = blockIdx.x * GT_M, n0 = blockIdx.y * BN;
    const int nk = K / GT_K;
    if (w == 0) {
        tc::tmem_alloc(&tmem_base, BN);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        for (int i = 0; i < S; i++) tc::mbar_init(&bar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // prologue: slices 0 .. S-2 in flight (one commit group per slice; empty groups past the end)
#pragma unroll
    for (int st = 0; st < S - 1; st++) {
        if (st < nk)
            gemm_load_slice<BN>(gsm + st * G::STAGE, gsm + st * G::STAGE + G::A_BYTES, A, lda, B, ldb, M, N, m0, n0,
                                st, t);
        cp_async_commit();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = tmem_base;
    const uint32_t idesc = tc::idesc_bf16_f32(GT_M, BN);
    bool ok = true;
    int issued = -1; // last slice whose MMAs were committed
    for (int i = 0; i < nk; i++) {
        cp_async_wait<S - 2>();            // this thread's copies of slice i have landed
        tc::fence_proxy_async_smem();      // ... and are visible to the tensor core
        if (__syncthreads_or(!ok)) break;  // every thread's copies of slice i, unless a wait gave up
        const int st = i % S;
        if (t == 0) {
            tc::fence_after_sync();
            const uint32_t a0 = tc::smem_u32(gsm + st * G::STAGE), b0 = a0 + G::A_BYTES;
#pragma unroll
            for (int s = 0; s < GT_K / 16; s++) {
                const uint64_t ad = tc::smem_desc_kmajor(a0 + 256u * s, 128u, 1024u);
                const uint64_t bd = tc::smem_desc_kmajor(b0 + 256u * s, 128u, 1024u);
                tc::mma_bf16(tbase, ad, bd, idesc, (i > 0 || s > 0) ? 1u : 0u);
            }
            tc::mma_commit(&bar[st]);
        }
        issued = i;
        // slice i + S - 1 goes into the stage that slice i - 1 used: wait for those MMAs first
        const int nxt = i + S - 1;
        if (nxt < nk) {
            if (i >= 1 && !tc::mbar_wait_bounded(&bar[(i - 1) % S], (uint32_t)((i - 1) / S) & 1u, wait_iters))
                ok = false;
            if (ok)
                gemm_load_slice<BN>(gsm + (nxt % S) * G::STAGE, gsm + (nxt % S) * G::STAGE + G::A_BYTES, A, lda, B,
                                    ldb, M, N, m0, n0, nxt, t);
        }
        cp_async_commit();
    }
    // the last commit covers every MMA issued before it
    if (ok && issued == nk - 1 && nk > 0 &&
        !tc::mbar_wait_bounded(&bar[issued % S], (uint32_t)(issued / S) & 1u, wait_iters))
        ok = false;
    const bool failed = __syncthreads_or(!ok) != 0;
    cp_async_wait_all();
    tc::fence_after_sync();
    if (!failed) {
        const int row = m0 + 32 * w + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            float v[16];
            tc::tmem_ld16(tbase + ((uint32_t)(32 * w) << 16) + (uint32_t)c0, v);
            if (row < M) {
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int col = n0 + c0 + j;
                    if (col < N) {
                        float *p = C + (size_t)row * ldc + col;
                        *p = accumulate ? *p + v[j] : v[j];
                    }
                }
            }
        }
    } else {
        if (t == 0) atomicOr(err, 1);
        // the MMAs in flight finish before their TMEM is freed (full bound)
        if (issued >= 0) tc::mbar_wait_bounded(&bar[issued % S], (uint32_t)(issued / S) & 1u, kWaitIters);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (w == 0) tc::tmem_dealloc(tbase, BN);
}

// ---------------------------------------------------------------------------
// The same product with TMA tile loads (used when A and B are 16-byte aligned
// with 16-byte row strides): one thread streams 64-wide K slices of A
// (128 rows) and B (BN rows) through GT_TMA_STAGES shared-memory stages with
// cp.async.bulk.tensor (128-byte swizzle, rows beyond M or N filled with
// zeros), each stage's loads completing on its "full" mbarrier; the same
// thread issues the slice's four MMAs once the stage is full and commits them
// to the stage's "empty" mbarrier, and refills the stage the previous slice
// used as soon as that slice's MMAs have completed, so the loads of the next
// GT_TMA_STAGES - 1 slices are in flight while the tensor core works.  The
// other threads wait at a block barrier for the epilogue.  Every wait is
// bounded; on a timeout the tile sets *err, waits (with the full bound) for its
// loads and MMAs in flight and frees its TMEM.
// ---------------------------------------------------------------------------
constexpr int GT_TMA_STAGES = 4;
template <int BN> struct TmaShape {
    static constexpr int A_BYTES = GT_M * GT_K * 2, B_BYTES = BN * GT_K * 2, STAGE = A_BYTES + B_BYTES;
    static constexpr int SMEM = GT_TMA_STAGES * STAGE + 1024; // + slack to align the stages to 1024 bytes
};

// K slice j of A (128 rows from m0) and B (rows from n0) into one stage, on its full barrier.
__device__ __forceinline__ void tma_stage_load(unsigned char *dst, int a_bytes, uint32_t stage_bytes,
                                               const CUtensorMap *ta, const CUtensorMap *tb, int j, int m0, int n0,
                                               uint64_t *full)
{
    tc::mbar_arrive_expect_tx(full, stage_bytes);
    tc::tma_load_2d(dst, ta, j * GT_K, m0, full);
    tc::tma_load_2d(dst + a_bytes, tb, j * GT_K, n0, full);
}

template <int BN>
__global__ void __launch_bounds__(128) k_gemm_tma(const __grid_constant__ CUtensorMap ta,
                                                  const __grid_constant__ CUtensorMap tb, float *__restrict__ C,
                                                  int ldc, int M, int N, int K, int accumulate, int *err,
                                                  uint32_t wait_iters)
{
    using G = TmaShape<BN>;
    constexpr int S = GT_TMA_STAGES;
    extern __shared__ unsigned char gsm_raw[];
    __shared__ __align__(8) uint64_t full[S], empty[S];
    __shared__ uint32_t tmem_base;
    __shared__ int bad;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int m0 = blockIdx.x * GT_M, n0 = blockIdx.y * BN;
    const int nk = K / GT_K;
    const uint32_t raw = tc::smem_u32(gsm_raw);
    unsigned char *gsm = gsm_raw + (((raw + 1023u) & ~1023u) - raw);
    if (w == 0) {
        tc::tmem_alloc(&tmem_base, BN);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        for (int i = 0; i < S; i++) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], 1);
        }
        bad = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = tmem_base;
    if (t == 0) {
        const uint32_t idesc = tc::idesc_bf16_f32(GT_M, BN);
        int last_load[S]; // last slice loaded into each stage (-1: none)
#pragma unroll
        for (int i = 0; i < S; i++) last_load[i] = -1;
        for (int j = 0; j < S && j < nk; j++) {
            tma_stage_load(gsm + j * G::STAGE, G::A_BYTES, (uint32_t)G::STAGE, &ta, &tb, j, m0, n0, &full[j]);
            last_load[j] = j;
        }
        bool ok = true;
        int issued = -1; // last slice whose MMAs were committed
        for (int i = 0; i < nk; i++) {
            const int st = i % S;
            if (!tc::mbar_wait_bounded(&full[st], (uint32_t)(i / S) & 1u, wait_iters)) {
                ok = false;
                break;
            }
            tc::fence_after_sync();
            const uint32_t a0 = tc::smem_u32(gsm + st * G::STAGE), b0 = a0 + G::A_BYTES;
#pragma unroll
            for (int s = 0; s < GT_K / 16; s++)
                tc::mma_bf16(tbase, tc::smem_desc_sw128(a0 + 32u * s), tc::smem_desc_sw128(b0 + 32u * s), idesc,
                             (i > 0 || s > 0) ? 1u : 0u);
            tc::mma_commit(&empty[st]);
            issued = i;
            // refill the stage that slice i - 1 used once its MMAs have completed
            const int j = i - 1 + S;
            if (i >= 1 && j < nk) {
                const int ps = (i - 1) % S;
                if (!tc::mbar_wait_bounded(&empty[ps], (uint32_t)((i - 1) / S) & 1u, wait_iters)) {
                    ok = false;
                    break;
                }
                tma_stage_load(gsm + ps * G::STAGE, G::A_BYTES, (uint32_t)G::STAGE, &ta, &tb, j, m0, n0,
                               &full[ps]);
                last_load[ps] = j;
            }
        }
        // the last commit covers every MMA issued before it
        if (ok && issued >= 0 &&
            !tc::mbar_wait_bounded(&empty[issued % S], (uint32_t)(issued / S) & 1u, wait_iters))
            ok = false;
        if (!ok || issued != nk - 1) {
            bad = 1;
            atomicOr(err, 1);
            // loads and MMAs in flight finish before the block leaves (full bound)
            for (int st = 0; st < S; st++)
                if (last_load[st] >= 0)
                    tc::mbar_wait_bounded(&full[st], (uint32_t)(last_load[st] / S) & 1u, kWaitIters);
            if (issued >= 0) tc::mbar_wait_bounded(&empty[issued % S], (uint32_t)(issued / S) & 1u, kWaitIters);
        }
    }
    __syncthreads();
    tc::fence_after_sync();
    if (!bad) {
        const int row = m0 + 32 * w + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            float v[16];
            tc::tmem_ld16(tbase + ((uint32_t)(32 * w) << 16) + (uint32_t)c0, v);
            if (row < M) {
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int col = n0 + c0 + j;
                    if (col < N) {
                        float *p = C + (size_t)row * ldc + col;
                        *p = accumulate ? *p + v[j] : v[j];
                    }
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (w == 0) tc::tmem_dealloc(tbase, BN);
}

// cuTensorMapEncodeTiled from the driver (no link-time dependency on libcuda)
static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
static int g_encode_state = 0; // 0 unknown, 1 available, -1 not available

static bool tma_available()
{
    if (g_encode_state == 0) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess && fn) {
            g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
            g_encode_state = 1;
        } else {
            cudaGetLastError();
            g_encode_state = -1;
        }
    }
    return g_encode_state == 1;
}

// rows x K BF16 matrix with row stride ld elements, tiles of box_rows x 64
static bool make_tile_map(CUtensorMap *m, const bf16 *p, int rows, int K, int ld, int box_rows)
{
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2u};
    const cuuint32_t box[2] = {(cuuint32_t)GT_K, (cuuint32_t)box_rows};
    const cuuint32_t es[2] = {1u, 1u};
    return g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16 *>(p), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static bool g_gemm_attr = false;

void gemm_tc(const bf16 *A, int lda, const bf16 *B, int ldb, float *C, int ldc, int M, int N, int K, int accumulate,
             int *err, cudaStream_t s)
{
    if (!g_gemm_attr) {
        cudaFuncSetAttribute(k_gemm_tc<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmShape<128>::SMEM);
        cudaFuncSetAttribute(k_gemm_tc<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmShape<64>::SMEM);
        cudaFuncSetAttribute(k_gemm_tma<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, TmaShape<128>::SMEM);
        cudaFuncSetAttribute(k_gemm_tma<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, TmaShape<64>::SMEM);
        g_gemm_attr = true;
    }
    const int mt = (M + GT_M - 1) / GT_M;
    // 128-wide tiles when they give at least two tiles per SM, else 64-wide (twice the CTAs)
    const bool wide = (long long)mt * ((N + 127) / 128) >= 2 * 148;
    if (K >= GT_K && tma_available() && ((uintptr_t)A & 15u) == 0 && ((uintptr_t)B & 15u) == 0 && lda % 8 == 0 &&
        ldb % 8 == 0) {
        CUtensorMap ta, tb;
        if (make_tile_map(&ta, A, M, K, lda, GT_M) && make_tile_map(&tb, B, N, K, ldb, wide ? 128 : 64)) {
            if (wide) {
                dim3 g(mt, (N + 127) / 128);
                k_gemm_tma<128><<<g, 128, TmaShape<128>::SMEM, s>>>(ta, tb, C, ldc, M, N, K, accumulate, err,
                                                                    g_wait_iters);
            } else {
                dim3 g(mt, (N + 63) / 64);
                k_gemm_tma<64><<<g, 128, TmaShape<64>::SMEM, s>>>(ta, tb, C, ldc, M, N, K, accumulate, err,
                                                                  g_wait_iters);
            }
            return;
        }
    }
    if (wide) {
        dim3 g(mt, (N + 127) / 128);
        k_gemm_tc<128><<<g, 128, GemmShape<128>::SMEM, s>>>(A, lda, B, ldb, C, ldc, M, N, K, accumulate, err,
                                                            g_wait_iters);
    } else {
        dim3 g(mt, (N + 63) / 64);
        k_gemm_tc<64><<<g, 128, GemmShape<64>::SMEM, s>>>(A, lda, B, ldb, C, ldc, M, N, K, accumulate, err,
                                                          g_wait_iters);
    }
}

} // namespace lcmc

// Limit of the kernels' bounded mbarrier waits (the GEMMs' here, the sweep's
// phase kernels'), in tries, for launches made and graphs captured from now on
// (0 restores the default).  A wait that runs out sets the kernel's error flag,
// waits for what is in flight with the full bound, frees its TMEM and returns;
// the call reports LCMC_ETIMEOUT.  For tests of that path: a limit of 1 makes
// the first wait give up.
extern "C" int lcmc_set_wait_limit(unsigned int tries)
{
    lcmc::g_wait_iters = tries ? (uint32_t)tries : lcmc::kWaitIters;
    return LCMC_OK;
}

namespace lcmc {

unsigned wait_limit() { return g_wait_iters; }

// ---------------------------------------------------------------------------
// MLP kernels (FP32 CUDA cores)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z)
{
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// Z += bias; H = silu(Z) (BF16, row-major B x H) and its transpose (H x B)
__global__ void k_bias_act(float *Z, const float *bias, bf16 *Hb, bf16 *HbT, int Bn, int Hn)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < Bn * Hn; i += gridDim.x * blockDim.x) {
        const int b = i / Hn, h = i % Hn;
        const float z = Z[i] + bias[h];
        Z[i] = z;
        const float a = silu(z);
        const bf16 ab = __float2bfloat16(a);
        Hb[i] = ab;
        if (HbT) HbT[(size_t)h * Bn + b] = ab;
    }
}

// Second hidden layer and output, warp per row: Z2 += b2, A2 = silu(Z2),
// y = A2 . w3 + b3; with a target also dy = 2 (y - t) / n_valid for rows <
// n_valid and the row's share of the loss.
__global__ void k_act_out(float *Z2, const float *b2, const float *w3, const float *b3, float *A2, float *y,
                          const float *target, float *dy, float *row_loss, int Bn, int Hn, int n_valid)
{
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < Bn; r += (gridDim.x * blockDim.x) >> 5) {
        float s = 0.0f;
        for (int h = lane; h < Hn; h += 32) {
            const size_t i = (size_t)r * Hn + h;
            const float z = Z2[i] + b2[h], a = silu(z);
            Z2[i] = z;
            A2[i] = a;
            s += a * w3[h];
        }
        for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
            const float v = s + b3[0];
            y[r] = v;
            if (target) {
                const float e = r < n_valid ? v - target[r] : 0.0f;
                dy[r] = 2.0f * e / (float)n_valid;
                row_loss[r] = e * e / (float)n_valid;
            }
        }
    }
}

// A layer's backward pass by columns: a block takes BK_COLS of the Hn columns and
// every row.  The sums over the batch are the block's own (no atomics, nothing to
// clear) and run in the rows' order, from shared memory, a thread per sum: 256
// dependent additions take 0.6 us, less than one more launch (a call of 2048 rows
// 2.33 ms, with sums by atomics 2.37).
// A training call so gives the same bits every time.  By atomics two of its runs
// differ: a last bit of a sum turns, through BF16 rounding of dZ, into 2^-9 of an
// element, and Adam divides a gradient by its size, so the step of a weight whose
// gradient is nearly zero may turn.  Relative difference of the weights, 160 seeds,
// eight steps / sixteen steps of 256 rows: two runs by atomics 1e-7 / 6e-6 in the
// median and above 2e-5 in 1 % / 27 % of the seeds; the rows' order against either
// 2e-7 / 6e-6, 1 % / 24 %.
constexpr int BK_COLS = 4, BK_THREADS = 256, BK_ROWS = BK_THREADS / BK_COLS;

// dZ2 = (dy w3) * silu'(Z2) in BF16 (B x H and its transpose); gradients of w3
// and b2, and (block 0) of b3 and the batch loss.
__global__ void __launch_bounds__(BK_THREADS) k_back_out(const float *dy, const float *row_loss, const float *w3,
                                                         const float *Z2, const float *A2, float *gw3, float *gb2,
                                                         float *gb3, float *loss, bf16 *dZ2b, bf16 *dZ2bT, int Bn, int Hn)
{
    __shared__ float term[2 * BK_COLS + 2][BK_THREADS]; // per column: w3, b2; then b3 and the loss
    const int c = threadIdx.x % BK_COLS, h = blockIdx.x * BK_COLS + c;
    float sum = 0.0f;
    for (int b0 = 0; b0 < Bn; b0 += BK_THREADS) {
        const int rows = min(BK_THREADS, Bn - b0);
        __syncthreads();
        for (int r = threadIdx.x / BK_COLS; r < rows; r += BK_ROWS) {
            const int b = b0 + r;
            const size_t i = (size_t)b * Hn + h;
            const float d = dy[b], g = d * w3[h] * dsilu(Z2[i]);
            const bf16 gb = __float2bfloat16(g);
            dZ2b[i] = gb;
            dZ2bT[(size_t)h * Bn + b] = gb;
            term[c][r] = __fmul_rn(d, A2[i]);
            term[BK_COLS + c][r] = g;
            if (c == 0) {
                term[2 * BK_COLS][r] = d;
                term[2 * BK_COLS + 1][r] = row_loss[b];
            }
        }
        __syncthreads();
        if (threadIdx.x < 2 * BK_COLS + 2) {
#pragma unroll 16
            for (int r = 0; r < rows; r++) sum += term[threadIdx.x][r];
        }
    }
    const int t = threadIdx.x;
    if (t < BK_COLS) gw3[h] = sum;
    else if (t < 2 * BK_COLS) gb2[h] = sum;
    else if (t < 2 * BK_COLS + 2 && blockIdx.x == 0) (t == 2 * BK_COLS ? gb3 : loss)[0] = sum;
}

// dZ1 = dH1 * silu'(Z1) -> dZ1^T (H x B) in BF16, and the gradient of b1
__global__ void __launch_bounds__(BK_THREADS) k_back_hidden(const float *dH, const float *Z, bf16 *dZbT, float *gbias,
                                                            int Bn, int Hn)
{
    __shared__ float term[BK_COLS][BK_THREADS];
    const int c = threadIdx.x % BK_COLS, h = blockIdx.x * BK_COLS + c;
    float sum = 0.0f;
    for (int b0 = 0; b0 < Bn; b0 += BK_THREADS) {
        const int rows = min(BK_THREADS, Bn - b0);
        __syncthreads();
        for (int r = threadIdx.x / BK_COLS; r < rows; r += BK_ROWS) {
            const size_t i = (size_t)(b0 + r) * Hn + h;
            const float g = dH[i] * dsilu(Z[i]);
            dZbT[(size_t)h * Bn + b0 + r] = __float2bfloat16(g);
            term[c][r] = g;
        }
        __syncthreads();
        if (threadIdx.x < BK_COLS) {
#pragma unroll 16
            for (int r = 0; r < rows; r++) sum += term[threadIdx.x][r];
        }
    }
    if (threadIdx.x < BK_COLS) gbias[h] = sum;
}

// rows pos[r] of the data set -> row r of X (16 bytes per thread and step)
__global__ void k_gather_rows(const bf16 *D, const int *pos, bf16 *X, int rows, int K1)
{
    const int per = K1 / 8;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows * per; i += gridDim.x * blockDim.x) {
        const int r = i / per, c = i - r * per;
        reinterpret_cast<uint4 *>(X)[i] = reinterpret_cast<const uint4 *>(D)[(size_t)pos[r] * per + c];
    }
}

// B x K (row-major BF16) -> K x B
__global__ void k_transpose_bf16(const bf16 *X, bf16 *XT, int Bn, int Kn)
{
    __shared__ bf16 tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = by + j, c = bx + threadIdx.x;
        if (r < Bn && c < Kn) tile[j][threadIdx.x] = X[(size_t)r * Kn + c];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = bx + j, c = by + threadIdx.x; // r: K index, c: B index
        if (r < Kn && c < Bn) XT[(size_t)r * Bn + c] = tile[threadIdx.x][j];
    }
}

__global__ void k_f32_to_bf16(const float *x, bf16 *y, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = __float2bfloat16(x[i]);
}

// W (rows x cols FP32) -> BF16 copy and BF16 transpose
__global__ void k_weights_bf16(const float *W, bf16 *Wb, bf16 *WbT, int rows, int cols)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows * cols; i += gridDim.x * blockDim.x) {
        const int r = i / cols, c = i % cols;
        const bf16 v = __float2bfloat16(W[i]);
        Wb[i] = v;
        if (WbT) WbT[(size_t)c * rows + r] = v;
    }
}

// Adam (Kingma & Ba 2015), FP32 master weights; the BF16 copies of W1 (the first
// n1 parameters) and W2 (H x H from o2, with its transpose) are written along.
__global__ void k_adam(float *w, const float *g, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2, bf16 *W1b, int n1, bf16 *W2b, bf16 *W2bT, int o2, int H)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        if (i < n1) {
            W1b[i] = __float2bfloat16(wi);
        } else if (i >= o2 && i < o2 + H * H) {
            const int j = i - o2;
            const bf16 x = __float2bfloat16(wi);
            W2b[j] = x;
            W2bT[(j % H) * H + j / H] = x;
        }
    }
}

} // namespace lcmc

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
using namespace lcmc;

// Host rows on their way to the device: rounding and its threads (send_rows has the rest).

// float -> BF16, round to nearest even, NaN to 0x7fff as __float2bfloat16 does
static inline uint16_t bf16_bits(float f)
{
    uint32_t u;
    memcpy(&u, &f, 4);
    if ((u & 0x7fffffffu) > 0x7f800000u) return 0x7fff;
    return (uint16_t)((u + 0x7fffu + ((u >> 16) & 1u)) >> 16);
}

static void convert_row(const float *x, int n_in, int k1, uint16_t *dst)
{
    int i = 0;
#ifdef __SSE2__
    const __m128i one = _mm_set1_epi32(1), bias = _mm_set1_epi32(0x7fff);
    for (; i + 8 <= n_in; i += 8) {
        const __m128 f0 = _mm_loadu_ps(x + i), f1 = _mm_loadu_ps(x + i + 4);
        const __m128i u0 = _mm_castps_si128(f0), u1 = _mm_castps_si128(f1);
        const __m128i v0 = _mm_add_epi32(_mm_add_epi32(u0, bias), _mm_and_si128(_mm_srli_epi32(u0, 16), one));
        const __m128i v1 = _mm_add_epi32(_mm_add_epi32(u1, bias), _mm_and_si128(_mm_srli_epi32(u1, 16), one));
        _mm_storeu_si128((__m128i *)(dst + i), _mm_packs_epi32(_mm_srai_epi32(v0, 16), _mm_srai_epi32(v1, 16)));
        if (_mm_movemask_ps(_mm_cmpunord_ps(f0, f1))) // a NaN among them
            for (int k = 0; k < 8; k++) dst[i + k] = bf16_bits(x[i + k]);
    }
#endif
    for (; i < n_in; i++) dst[i] = bf16_bits(x[i]);
    for (; i < k1; i++) dst[i] = 0;
}

// Host threads that round rows for a network: they come with its first large call,
// sleep between calls and end with it.  A part is done when its rows are: the
// caller takes rows like every thread, and a thread that is not scheduled in time
// (other threads of the process may hold the cores) finds nothing left to do.
// When every thread had to report, and to end with the call, the first prediction
// of 600 rows after other host work took 4.5 ms, now 1.0 (a quiet host 1.1, now 0.9);
// predictions of 4096 rows 2.15 -> 1.85 ms, 2048 rows of training 2.2-2.9 -> 2.13.
class RowConverter {
public:
    ~RowConverter()
    {
        if (threads_.empty()) return;
        if (getpid() != pid_) { // a child process: the threads are the parent's
            for (auto &t : threads_) t.detach();
            return;
        }
        {
            std::lock_guard<std::mutex> l(mu_);
            stop_.store(true);
        }
        cv_.notify_all();
        for (auto &t : threads_) t.join();
    }
    // Before the parts of a call of that many values: threads in proportion (waking one takes as long as rounding a
    // few hundred KB), so that small calls are the caller's alone.
    void begin(size_t values)
    {
        want_ = (int)std::min<size_t>(values >> 19, 12);
        if (want_ <= 1) return;
        const int hw = (int)std::thread::hardware_concurrency();
        want_ = std::min(want_, hw > 0 ? hw : 1);
        if (threads_.empty()) pid_ = getpid();
        else if (getpid() != pid_) want_ = 1;
        try {
            threads_.reserve(16);
            while ((int)threads_.size() < want_ - 1) threads_.emplace_back([this] { work(); });
        } catch (...) { // fewer threads then
        }
        active_.store(true);
    }
    // After a call's last part: the threads may sleep.
    void end() { active_.store(false); }
    bool alone() const { return want_ <= 1; }
    // rows idx[r] (idx null: r) of x -> rows r of dst
    void run(const float *x, const int *idx, int n, int n_in, int k1, uint16_t *dst)
    {
        const uint64_t gen = ++part_;
        next_.store(gen << 32 | 0xffffffffu); // closed: no thread takes a row by the last part's count
        x_ = x, idx_ = idx, n_in_ = n_in, k1_ = k1, dst_ = dst;
        n_.store(n);
        done_.store(0);
        next_.store(gen << 32);
        if (!alone()) {
            {
                std::lock_guard<std::mutex> l(mu_);
                gen_.store(gen);
            }
            if (want_ > (int)threads_.size()) cv_.notify_all(); // (one call of the system for all of them)
            else
                for (int i = 1; i < want_; i++) cv_.notify_one();
        }
        rows(gen);
        while (done_.load() < n) std::this_thread::yield(); // (rows that a thread has taken)
    }

private:
    // rows of part `gen` until none is left
    void rows(uint64_t gen)
    {
        constexpr int STEP = 8;
        for (uint64_t v = next_.load(); v >> 32 == (gen & 0xffffffffu);) {
            const uint32_t r0 = (uint32_t)v;
            const int n = n_.load();
            if (r0 >= (uint32_t)n) return;
            if (!next_.compare_exchange_weak(v, v + STEP)) continue; // (taken: the part's description holds until it is done)
            const int r1 = std::min(n, (int)r0 + STEP);
            for (int r = (int)r0; r < r1; r++)
                convert_row(x_ + (size_t)(idx_ ? idx_[r] : r) * n_in_, n_in_, k1_, dst_ + (size_t)r * k1_);
            done_.fetch_add(r1 - (int)r0);
            v = next_.load();
        }
    }
    void work()
    {
        uint64_t seen = 0;
        for (;;) {
            // the next part of a call follows within 10 to 100 us (a training step's launches lie between two
            // batches): look for it a while before sleeping
            for (int i = 0; i < 2048 && active_.load() && gen_.load() == seen && !stop_.load(); i++)
                std::this_thread::yield();
            if (gen_.load() == seen) {
                std::unique_lock<std::mutex> l(mu_);
                cv_.wait(l, [&] { return stop_.load() || gen_.load() != seen; });
            }
            if (stop_.load()) return;
            seen = gen_.load();
            rows(seen);
        }
    }
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable cv_;
    std::atomic<uint64_t> next_{0}; // part (32 bits), its next row
    std::atomic<uint64_t> gen_{0};  // the part the threads are told of
    std::atomic<int> n_{0}, done_{0};
    std::atomic<bool> stop_{false}, active_{false};
    uint64_t part_ = 0;
    int want_ = 1;
    pid_t pid_ = 0;
    const float *x_ = nullptr;
    const int *idx_ = nullptr;
    int n_in_ = 0, k1_ = 0;
    uint16_t *dst_ = nullptr;
};

struct lcmc_mlp {
    int n_in = 0, k1 = 0, hid = 0, bmax = 0;
    cudaStream_t s = nullptr;
    // FP32 masters, Adam moments and gradients, in one block each
    float *W1 = nullptr, *b1 = nullptr, *W2 = nullptr, *b2 = nullptr, *w3 = nullptr, *b3 = nullptr;
    float *P = nullptr, *G = nullptr, *Mm = nullptr, *Vv = nullptr; // parameter / grad / moment blocks
    size_t np = 0;
    bf16 *W1b = nullptr, *W2b = nullptr, *W2bT = nullptr;
    char *base = nullptr; // of the weights above and the activations (bmax rows)
    bf16 *X = nullptr, *XT = nullptr, *H1 = nullptr, *H1T = nullptr, *dZ2 = nullptr, *dZ2T = nullptr, *dZ1T = nullptr;
    float *Z1 = nullptr, *Z2 = nullptr, *A2 = nullptr, *y = nullptr, *t = nullptr, *dy = nullptr, *row_loss = nullptr,
          *dH1 = nullptr, *loss = nullptr;
    int *err = nullptr;
    // host rows on their way to the device
    static constexpr int SLOTS = 2, STAGE_ROWS = 128;
    uint16_t *stage = nullptr; // pinned, SLOTS x STAGE_ROWS rows of k1 BF16 values each
    cudaEvent_t sent[SLOTS] = {nullptr, nullptr};
    int slot = 0;
    RowConverter rc;
    // training: the rows (BF16), an epoch's targets and places of its rows, its losses (grown as needed)
    bf16 *rows = nullptr;
    float *et = nullptr, *losses = nullptr;
    int *pos = nullptr;
    size_t rows_n = 0, et_n = 0, losses_n = 0, pos_n = 0;
    float *yall = nullptr; // a predict call's outputs (grown as needed)
    size_t yall_n = 0;
    long long step = 0;
    std::string msg;
};

static int mlp_fail(lcmc_mlp *m, const char *what, cudaError_t e)
{
    if (m) m->msg = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? LCMC_ENOMEM : LCMC_ECUDA;
}

extern "C" int lcmc_mlp_destroy(lcmc_mlp *m)
{
    if (!m) return LCMC_EINVAL;
    if (m->s) cudaStreamSynchronize(m->s);
    void *ptrs[] = {m->base, m->yall, m->rows, m->et, m->losses, m->pos};
    if (m->stage) cudaFreeHost(m->stage);
    for (cudaEvent_t ev : m->sent)
        if (ev) cudaEventDestroy(ev);
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (m->s) cudaStreamDestroy(m->s);
    delete m;
    return LCMC_OK;
}

template <typename T>
static cudaError_t grow(T **p, size_t *have, size_t want)
{
    if (want <= *have) return cudaSuccess;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *have = 0;
    cudaError_t e = cudaMalloc((void **)p, want * sizeof(T));
    if (e == cudaSuccess) *have = want;
    return e;
}

// Weights: uniform(-a, a) with a = sqrt(6 / (fan_in + fan_out)) (Glorot & Bengio
// 2010), from Philox so that a seed fixes the network.
extern "C" int lcmc_mlp_create(int n_in, int hidden, int max_batch, uint64_t seed, lcmc_mlp **out)
{
    if (!out || n_in <= 0 || hidden != 128 || max_batch <= 0) return LCMC_EINVAL;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return LCMC_ENODEV;
    }
    lcmc_mlp *m = new lcmc_mlp();
    m->n_in = n_in;
    m->k1 = (n_in + 127) / 128 * 128;
    m->hid = hidden;
    m->bmax = (max_batch + 127) / 128 * 128;
    const int H = hidden, K1 = m->k1, B = m->bmax;
    m->np = (size_t)H * K1 + H + (size_t)H * H + H + H + 1;
    cudaError_t e = cudaStreamCreateWithFlags(&m->s, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        lcmc_mlp_destroy(m);
        return LCMC_ECUDA;
    }
    // one allocation: a dozen MB, where each of its own would take as long as all of it
    const std::pair<void **, size_t> bufs[] = {
        {(void **)&m->P, m->np * 4}, {(void **)&m->G, m->np * 4}, {(void **)&m->Mm, m->np * 4},
        {(void **)&m->Vv, m->np * 4}, {(void **)&m->W1b, (size_t)H * K1 * 2}, {(void **)&m->W2b, (size_t)H * H * 2},
        {(void **)&m->W2bT, (size_t)H * H * 2}, {(void **)&m->X, (size_t)B * K1 * 2},
        {(void **)&m->XT, (size_t)B * K1 * 2}, {(void **)&m->H1, (size_t)B * H * 2},
        {(void **)&m->H1T, (size_t)B * H * 2}, {(void **)&m->dZ2, (size_t)B * H * 2},
        {(void **)&m->dZ2T, (size_t)B * H * 2}, {(void **)&m->dZ1T, (size_t)B * H * 2},
        {(void **)&m->Z1, (size_t)B * H * 4}, {(void **)&m->Z2, (size_t)B * H * 4},
        {(void **)&m->A2, (size_t)B * H * 4}, {(void **)&m->y, (size_t)B * 4}, {(void **)&m->t, (size_t)B * 4},
        {(void **)&m->dy, (size_t)B * 4}, {(void **)&m->row_loss, (size_t)B * 4},
        {(void **)&m->dH1, (size_t)B * H * 4}, {(void **)&m->loss, 4}, {(void **)&m->err, 4}};
    size_t total = 0;
    for (const auto &b : bufs) total += (b.second + 255) / 256 * 256;
    if (cudaMalloc((void **)&m->base, total) != cudaSuccess) {
        cudaGetLastError();
        lcmc_mlp_destroy(m);
        return LCMC_ENOMEM;
    }
    size_t at = 0;
    for (const auto &b : bufs) {
        *b.first = m->base + at;
        at += (b.second + 255) / 256 * 256;
    }
    e = cudaMallocHost((void **)&m->stage, (size_t)lcmc_mlp::SLOTS * lcmc_mlp::STAGE_ROWS * K1 * 2);
    for (cudaEvent_t &ev : m->sent)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = grow(&m->yall, &m->yall_n, (size_t)1 << 16);
    if (e == cudaSuccess) e = grow(&m->et, &m->et_n, (size_t)1 << 16);
    if (e == cudaSuccess) e = grow(&m->losses, &m->losses_n, (size_t)1 << 10);
    if (e != cudaSuccess) {
        lcmc_mlp_destroy(m);
        return LCMC_ENOMEM;
    }
    m->W1 = m->P;
    m->b1 = m->W1 + (size_t)H * K1;
    m->W2 = m->b1 + H;
    m->b2 = m->W2 + (size_t)H * H;
    m->w3 = m->b2 + H;
    m->b3 = m->w3 + H;
    std::vector<float> host(m->np, 0.0f);
    uint32_t key[2];
    seed_key(seed, key);
    auto uni = [&](size_t i, float a) {
        U4 o = draw(key, (uint32_t)(i & 0xFFFFFFFFu), 0xABCD0000ull + (i >> 32), 0x300u);
        return (float)((2.0 * u01(o.x) - 1.0) * a);
    };
    const float a1 = sqrtf(6.0f / (n_in + H)), a2 = sqrtf(6.0f / (2 * H)), a3 = sqrtf(6.0f / (H + 1));
    for (int h = 0; h < H; h++)
        for (int k = 0; k < n_in; k++) host[(size_t)h * K1 + k] = uni((size_t)h * K1 + k, a1); // padding stays 0
    const size_t o2 = (size_t)H * K1 + H;
    for (size_t i = 0; i < (size_t)H * H; i++) host[o2 + i] = uni(o2 + i, a2);
    const size_t o3 = o2 + (size_t)H * H + H;
    for (int h = 0; h < H; h++) host[o3 + h] = uni(o3 + h, a3);
    // on the network's own stream: the conversions below follow the copy
    cudaMemcpyAsync(m->P, host.data(), m->np * 4, cudaMemcpyHostToDevice, m->s);
    cudaMemsetAsync(m->Mm, 0, m->np * 4, m->s);
    cudaMemsetAsync(m->Vv, 0, m->np * 4, m->s);
    cudaMemsetAsync(m->X, 0, (size_t)B * K1 * 2, m->s);
    cudaMemsetAsync(m->err, 0, 4, m->s);
    k_weights_bf16<<<256, 256, 0, m->s>>>(m->W1, m->W1b, nullptr, H, K1);
    k_weights_bf16<<<64, 256, 0, m->s>>>(m->W2, m->W2b, m->W2bT, H, H);
    e = cudaStreamSynchronize(m->s);
    if (e != cudaSuccess) {
        lcmc_mlp_destroy(m);
        return LCMC_ECUDA;
    }
    *out = m;
    return LCMC_OK;
}

// forward on B (a multiple of 128) rows of X -> activations A2, outputs y; with
// targets t also dy and the rows' losses
static void mlp_forward_s(lcmc_mlp *m, const bf16 *X, int B, const float *t, int n_valid, cudaStream_t s)
{
    const int H = m->hid, K1 = m->k1;
    gemm_tc(X, K1, m->W1b, K1, m->Z1, H, B, H, K1, 0, m->err, s);
    k_bias_act<<<(B * H + 255) / 256, 256, 0, s>>>(m->Z1, m->b1, m->H1, m->H1T, B, H);
    gemm_tc(m->H1, H, m->W2b, H, m->Z2, H, B, H, H, 0, m->err, s);
    k_act_out<<<(B * 32 + 255) / 256, 256, 0, s>>>(m->Z2, m->b2, m->w3, m->b3, m->A2, m->y, t, m->dy, m->row_loss, B, H,
                                                   n_valid);
}

namespace lcmc {
// In-sweep inference: the sweep's kernels write the BF16 input rows into
// mlp_input() (leading dimension mlp_ld()), then the forward pass and the
// output layer run on the sweep's stream; returns the device output vector.
void *mlp_input(lcmc_mlp *m) { return m->X; }
int mlp_ld(lcmc_mlp *m) { return m->k1; }
int mlp_bmax(lcmc_mlp *m) { return m->bmax; }
int mlp_n_in(lcmc_mlp *m) { return m->n_in; }
const float *mlp_forward_device(lcmc_mlp *m, int B, cudaStream_t s)
{
    mlp_forward_s(m, m->X, B, nullptr, B, s);
    return m->y;
}
int *mlp_err(lcmc_mlp *m) { return m->err; }
} // namespace lcmc

// ---------------------------------------------------------------------------
// Host rows to the device.  Feature rows come as FP32 in pageable memory, 16 KB
// each; copied as they are, the driver moves them at 8-10 GB/s through its own
// staging, and that was nearly all of a call.  Here host threads round them to
// BF16, which the network takes, into pinned buffers whose copies run while the
// next rows are converted: half the bytes on the link.  Predictions of 4096 rows
// 8.2 -> 1.85 ms, an epoch of 2048 rows in batches of 256 10.6 -> 2.1 ms; bound by
// the threads' reads of the FP32 rows (67 MB in 4096 of them).  That is for rows
// used again and again; the first call of a new network on new rows 8.8 -> 2.6 ms
// (4096 rows) on a quiet host, 9.2 -> 3.6 where other threads still hold the cores.
// ---------------------------------------------------------------------------

// Below 256 rows a single thread converts: its parts are small, so that only the
// last one's copy is left when it is done (96 rows: 245 us a call with one part, 209
// now, 227 with the FP32 rows copied as they are; parts of 48 rows 2 % slower).
constexpr int SMALL_PART = 32;

// Rows idx[0 .. n) (idx null: the first n) of the caller's features to rows [0, B)
// of dst on the network's stream, zeros beyond n.
static cudaError_t send_rows(lcmc_mlp *m, const float *x, const int *idx, int n, int B, bf16 *dst)
{
    cudaError_t e;
    const size_t row = (size_t)m->k1 * 2;
    const int step = m->rc.alone() ? SMALL_PART : lcmc_mlp::STAGE_ROWS;
    for (int off = 0; off < n; off += step) {
        const int i = m->slot, c = std::min(step, n - off);
        m->slot = (i + 1) % lcmc_mlp::SLOTS;
        if ((e = cudaEventSynchronize(m->sent[i])) != cudaSuccess) return e; // its last copy has left
        uint16_t *stage = m->stage + (size_t)i * lcmc_mlp::STAGE_ROWS * m->k1;
        m->rc.run(idx ? x : x + (size_t)off * m->n_in, idx ? idx + off : nullptr, c, m->n_in, m->k1, stage);
        e = cudaMemcpyAsync(dst + (size_t)off * m->k1, stage, (size_t)c * row, cudaMemcpyHostToDevice, m->s);
        if (e != cudaSuccess) return e;
        if ((e = cudaEventRecord(m->sent[i], m->s)) != cudaSuccess) return e;
    }
    if (B > n) return cudaMemsetAsync((char *)dst + (size_t)n * row, 0, (size_t)(B - n) * row, m->s);
    return cudaSuccess;
}

extern "C" int lcmc_mlp_predict(lcmc_mlp *m, const float *x, int n, float *y)
{
    if (!m || !x || !y || n < 0) return LCMC_EINVAL;
    cudaError_t e = cudaSuccess;
    if (n > 0) {
        // outputs of several batches gather on the device: one copy back, after the last rows
        const bool gather = n > m->bmax;
        if (gather && (e = grow(&m->yall, &m->yall_n, (size_t)(n + 127) / 128 * 128)) != cudaSuccess) return mlp_fail(m, "predict", e);
        m->rc.begin((size_t)n * m->n_in);
        for (int off = 0; off < n && e == cudaSuccess; off += m->bmax) {
            const int nb = n - off < m->bmax ? n - off : m->bmax;
            const int B = (nb + 127) / 128 * 128;
            e = send_rows(m, x + (size_t)off * m->n_in, nullptr, nb, B, m->X);
            if (e != cudaSuccess) break;
            mlp_forward_s(m, m->X, B, nullptr, nb, m->s);
            if (gather) e = cudaMemcpyAsync(m->yall + off, m->y, (size_t)nb * 4, cudaMemcpyDeviceToDevice, m->s);
        }
        m->rc.end();
        if (e == cudaSuccess) e = cudaMemcpyAsync(y, gather ? m->yall : m->y, (size_t)n * 4, cudaMemcpyDeviceToHost, m->s);
    }
    const cudaError_t es = cudaStreamSynchronize(m->s);
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) return mlp_fail(m, "predict", e);
    int err = 0;
    cudaMemcpy(&err, m->err, 4, cudaMemcpyDeviceToHost);
    return err ? LCMC_ETIMEOUT : LCMC_OK;
}

// Forward + backward on n rows of X (zeros beyond, up to a multiple of 128; so
// the targets t): gradients in m->G, MSE in *loss.
static void mlp_backward(lcmc_mlp *m, const bf16 *X, const float *t, int n, float *loss)
{
    const int H = m->hid, K1 = m->k1;
    const int B = (n + 127) / 128 * 128;
    mlp_forward_s(m, X, B, t, n, m->s);
    float *gW1 = m->G, *gb1 = gW1 + (size_t)H * K1, *gW2 = gb1 + H, *gb2 = gW2 + (size_t)H * H, *gw3 = gb2 + H,
          *gb3 = gw3 + H;
    k_back_out<<<H / BK_COLS, BK_THREADS, 0, m->s>>>(m->dy, m->row_loss, m->w3, m->Z2, m->A2, gw3, gb2, gb3, loss, m->dZ2,
                                                     m->dZ2T, B, H);
    // dW2 = dZ2^T H1: (H x B) . (H x B)^T
    gemm_tc(m->dZ2T, B, m->H1T, B, gW2, H, H, H, B, 0, m->err, m->s);
    // dH1 = dZ2 W2: (B x H) . (W2^T)^T
    gemm_tc(m->dZ2, H, m->W2bT, H, m->dH1, H, B, H, H, 0, m->err, m->s);
    k_back_hidden<<<H / BK_COLS, BK_THREADS, 0, m->s>>>(m->dH1, m->Z1, m->dZ1T, gb1, B, H);
    // dW1 = dZ1^T X: (H x B) . (X^T)^T with X^T = K1 x B
    dim3 tg((K1 + 31) / 32, (B + 31) / 32), tb(32, 8);
    k_transpose_bf16<<<tg, tb, 0, m->s>>>(X, m->XT, B, K1);
    gemm_tc(m->dZ1T, B, m->XT, B, gW1, K1, H, K1, B, 0, m->err, m->s);
}

// One Adam step on the gradients in m->G.
static void mlp_update(lcmc_mlp *m, float lr)
{
    const int H = m->hid, K1 = m->k1;
    m->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)m->step), c2 = 1.0f - powf(b2, (float)m->step);
    // padding columns of W1 stay exactly zero: their gradient is zero (zero inputs)
    k_adam<<<512, 256, 0, m->s>>>(m->P, m->G, m->Mm, m->Vv, (int)m->np, lr, b1, b2, 1e-8f, c1, c2, m->W1b, H * K1, m->W2b,
                                  m->W2bT, (int)(m->W2 - m->P), H);
}

extern "C" int lcmc_mlp_num_params(const lcmc_mlp *m) { return m ? (int)m->np : 0; }

extern "C" int lcmc_mlp_gradients(lcmc_mlp *m, const float *x, const float *t, int n, float *grad, float *loss)
{
    if (!m || !x || !t || !grad || n <= 0 || n > m->bmax) return LCMC_EINVAL;
    const int B = (n + 127) / 128 * 128;
    cudaError_t e;
    m->rc.begin((size_t)n * m->n_in);
    e = send_rows(m, x, nullptr, n, B, m->X);
    m->rc.end();
    if (e != cudaSuccess) return mlp_fail(m, "gradients", e);
    cudaMemsetAsync(m->t, 0, (size_t)B * 4, m->s);
    cudaMemcpyAsync(m->t, t, (size_t)n * 4, cudaMemcpyHostToDevice, m->s);
    mlp_backward(m, m->X, m->t, n, m->loss);
    cudaMemcpyAsync(grad, m->G, m->np * 4, cudaMemcpyDeviceToHost, m->s);
    if (loss) cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, m->s);
    e = cudaStreamSynchronize(m->s);
    if (e != cudaSuccess) return mlp_fail(m, "gradients", e);
    int err = 0;
    cudaMemcpy(&err, m->err, 4, cudaMemcpyDeviceToHost);
    return err ? LCMC_ETIMEOUT : LCMC_OK;
}

extern "C" int lcmc_mlp_get_params(lcmc_mlp *m, float *params)
{
    if (!m || !params) return LCMC_EINVAL;
    cudaError_t e = cudaMemcpy(params, m->P, m->np * 4, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? LCMC_OK : mlp_fail(m, "get_params", e);
}

extern "C" int lcmc_mlp_set_params(lcmc_mlp *m, const float *params)
{
    if (!m || !params) return LCMC_EINVAL;
    cudaError_t e = cudaMemcpyAsync(m->P, params, m->np * 4, cudaMemcpyHostToDevice, m->s);
    if (e != cudaSuccess) return mlp_fail(m, "set_params", e);
    k_weights_bf16<<<256, 256, 0, m->s>>>(m->W1, m->W1b, nullptr, m->hid, m->k1);
    k_weights_bf16<<<64, 256, 0, m->s>>>(m->W2, m->W2b, m->W2bT, m->hid, m->hid);
    e = cudaStreamSynchronize(m->s);
    return e == cudaSuccess ? LCMC_OK : mlp_fail(m, "set_params", e);
}

// The rows cross the link once: the first epoch sends each batch's and, if there
// are more epochs, keeps them on the device in the order in which it took them;
// the later epochs gather from there.  Rows that would take more than
// TRAIN_KEEP_BYTES, or for which there is no room, are sent in every epoch.
// Nothing waits for a step: the losses stay on the device until the last one.
constexpr size_t TRAIN_KEEP_BYTES = (size_t)1 << 30;

extern "C" int lcmc_mlp_train(lcmc_mlp *m, const float *x, const float *t, int n, int epochs, int batch, float lr,
                              uint64_t seed, float *final_loss)
{
    if (!m || !x || !t || n <= 0 || epochs <= 0 || batch <= 0 || batch > m->bmax) return LCMC_EINVAL;
    std::vector<int> idx(n), at(n); // a batch's rows; their places on the device
    for (int i = 0; i < n; i++) idx[i] = i;
    uint32_t key[2];
    seed_key(seed, key);
    const int nb = n / batch, used = nb * batch, B = (batch + 127) / 128 * 128, K1 = m->k1;
    std::vector<float> et(n), losses(std::max(nb, 1));
    std::vector<int> place(n);
    cudaError_t e = grow(&m->et, &m->et_n, (size_t)n);
    if (e == cudaSuccess) e = grow(&m->losses, &m->losses_n, losses.size());
    if (e != cudaSuccess) return mlp_fail(m, "train", e);
    bool keep = epochs > 1 && nb > 0 && (size_t)n * K1 * 2 <= TRAIN_KEEP_BYTES;
    if (keep && (grow(&m->pos, &m->pos_n, (size_t)n) != cudaSuccess ||
                 grow(&m->rows, &m->rows_n, (size_t)n * K1) != cudaSuccess)) {
        cudaGetLastError();
        keep = false;
    }
    m->rc.begin((size_t)n * m->n_in);
    for (int ep = 0; ep < epochs && e == cudaSuccess && nb > 0; ep++) {
        for (int i = n - 1; i > 0; i--) { // shuffle
            U4 o = draw(key, (uint32_t)i, (uint64_t)ep, 0x301u);
            int j = (int)(o.x % (uint32_t)(i + 1));
            int tmp = idx[i];
            idx[i] = idx[j];
            idx[j] = tmp;
        }
        const bool gather = ep > 0 && keep;
        for (int i = 0; i < n; i++) {
            et[i] = t[idx[i]];
            if (ep == 0) place[idx[i]] = i;
            at[i] = place[idx[i]];
        }
        // (pageable memory: the copies have left it when the calls return)
        e = cudaMemcpyAsync(m->et, et.data(), (size_t)n * 4, cudaMemcpyHostToDevice, m->s);
        if (e == cudaSuccess && gather) e = cudaMemcpyAsync(m->pos, at.data(), (size_t)n * 4, cudaMemcpyHostToDevice, m->s);
        for (int k = 0; k < nb && e == cudaSuccess; k++) {
            const int off = k * batch;
            if (gather) {
                k_gather_rows<<<512, 256, 0, m->s>>>(m->rows, m->pos + off, m->X, batch, K1);
                if (B > batch)
                    e = cudaMemsetAsync(m->X + (size_t)batch * K1, 0, (size_t)(B - batch) * K1 * 2, m->s);
            } else {
                e = send_rows(m, x, idx.data() + off, batch, B, m->X);
                if (e == cudaSuccess && keep)
                    e = cudaMemcpyAsync(m->rows + (size_t)off * K1, m->X, (size_t)batch * K1 * 2,
                                        cudaMemcpyDeviceToDevice, m->s);
            }
            if (e != cudaSuccess) break;
            mlp_backward(m, m->X, m->et + off, batch, m->losses + k);
            mlp_update(m, lr);
        }
        if (ep == 0 && keep && e == cudaSuccess && used < n) // rows that no batch of the first epoch took
            e = send_rows(m, x, idx.data() + used, n - used, n - used, m->rows + (size_t)used * K1);
        if (keep) m->rc.end(); // (later epochs send none)
    }
    m->rc.end();
    if (e == cudaSuccess && nb > 0)
        e = cudaMemcpyAsync(losses.data(), m->losses, (size_t)nb * 4, cudaMemcpyDeviceToHost, m->s);
    const cudaError_t es = cudaStreamSynchronize(m->s);
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) return mlp_fail(m, "train", e);
    double acc = 0.0; // the last epoch's
    for (int k = 0; k < nb; k++) acc += losses[k];
    int err = 0;
    cudaMemcpy(&err, m->err, 4, cudaMemcpyDeviceToHost);
    if (final_loss) *final_loss = nb ? (float)(acc / nb) : 0.0f;
    return err ? LCMC_ETIMEOUT : LCMC_OK;
}

// C[M x N] = A[M x K] B[N x K]^T on the tensor cores, host arrays (test hook).
extern "C" int lcmc_gemm_bf16(const float *A, const float *B, float *C, int M, int N, int K)
{
    if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0 || K % 64) return LCMC_EINVAL;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return LCMC_ENODEV;
    }
    float *fa, *fb, *fc;
    bf16 *ba, *bb;
    int *err;
    if (cudaMalloc(&fa, (size_t)M * K * 4) || cudaMalloc(&fb, (size_t)N * K * 4) ||
        cudaMalloc(&fc, (size_t)M * N * 4) || cudaMalloc(&ba, (size_t)M * K * 2) ||
        cudaMalloc(&bb, (size_t)N * K * 2) || cudaMalloc(&err, 4))
        return LCMC_ENOMEM;
    cudaMemcpy(fa, A, (size_t)M * K * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(fb, B, (size_t)N * K * 4, cudaMemcpyHostToDevice);
    cudaMemset(err, 0, 4);
    k_f32_to_bf16<<<256, 256>>>(fa, ba, M * K);
    k_f32_to_bf16<<<256, 256>>>(fb, bb, N * K);
    gemm_tc(ba, K, bb, K, fc, N, M, N, K, 0, err, 0);
    cudaError_t e = cudaMemcpy(C, fc, (size_t)M * N * 4, cudaMemcpyDeviceToHost);
    int herr = 0;
    cudaMemcpy(&herr, err, 4, cudaMemcpyDeviceToHost);
    cudaFree(fa);
    cudaFree(fb);
    cudaFree(fc);
    cudaFree(ba);
    cudaFree(bb);
    cudaFree(err);
    if (e != cudaSuccess) return LCMC_ECUDA;
    return herr ? LCMC_ETIMEOUT : LCMC_OK;
}
