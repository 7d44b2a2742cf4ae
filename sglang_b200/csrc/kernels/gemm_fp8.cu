// Block-scaled fp8 (e4m3) GEMM on tcgen05 for sm_100a + the activation quantiser that feeds it.
//
//   C[M,N] (bf16) = sum_kb  xs[m,kb] * ws[n/128,kb] * ( A[m, kb*128:(kb+1)*128] . W[n, kb*128:(kb+1)*128] )
//
//   A  [M,K]  e4m3, xs [M, K/128] fp32  (per-token, per-128-channel group scales — produced by per_token_group_quant_fp8)
//   W  [N,K]  e4m3, ws [N/128, K/128] fp32 (128x128 weight blocks — the DeepSeek-V3 / "fp8 block" checkpoint format)
//
// Scales change every 128-wide K block, so partial products cannot simply accumulate in TMEM.  Each K block is
// therefore ONE 128-byte-swizzled smem stage (128 fp8 = 128 B per row) = 4 tcgen05.mma kind::f8f6f4 (K=32 each) into a
// fresh TMEM accumulator stage; the epilogue warps drain that stage with tcgen05.ld, apply xs*ws and accumulate in fp32
// registers ("promotion") while the tensor core already fills the next TMEM stage.  Two kernels:
//
//   prompt shapes (gemm_fp8_block_kernel): rows of A are the UMMA M dimension, 256 / 128 / 64 weight rows the N dimension, persistent CTAs.
//     warp 0 : TMA producer      warp 1 : MMA issuer      warp 2 : TMEM alloc      warps 4.. : promotion + epilogue, 64 columns each at most
//   decode shapes (gemm_fp8_swap_kernel, up to 64 tokens): 128 weight rows are the M dimension, the tokens the N dimension, so no tensor or TMA
//     work goes into padding rows; a cluster shares a tile's K blocks and adds its partial sums through distributed shared memory.
//
// Reference counterparts: python/sglang/srt/layers/quantization/fp8_kernel.py (per_token_group_quant_fp8,
// w8a8_block_fp8_matmul), fp8_utils.py:552-808 (DeepGEMM / cutlass / triton dispatch), sgl-kernel fp8_blockwise_gemm.
#include "common.cuh"
#include "tma_host.h"

#include <algorithm>

namespace sglb {

constexpr int F8_BM = 128;
constexpr int F8_BK = 128;          // fp8 elements = bytes per swizzled row = one scale group
// sum pair += s * (a, b): one packed instruction for two fp32 fused multiply-adds, each rounded as fmaf rounds it
__device__ __forceinline__ void fma_pair(float2& sum, float s, uint32_t a, uint32_t b) {
  uint64_t acc = *reinterpret_cast<uint64_t*>(&sum), v, m;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b));
  asm("mov.b64 %0, {%1, %1};" : "=l"(m) : "r"(__float_as_uint(s)));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(m), "l"(v));
  sum = *reinterpret_cast<float2*>(&acc);
}

// Bound by the hand-off of an accumulator to the promotion (TMEM loads, 32 packed multiply-adds a warp, and the waits on both sides take about three times
// the 256 cycles that 128 columns cost the tensor core), so a 256-wide tile has two halves with two accumulators each: one half is drained while the other is
// formed.  The promotion warps take the registers of the other warpgroup, so that sixteen columns are on their way while sixteen are multiplied.
// Measured, us a block (quantiser, [2I x H], SiLU, quantiser, [H x I]), blocks one behind the other on the same inputs, before (whole 256-wide accumulators, one
// thread each for copies and products) and now: 3001 tokens of 4096 / 14336: 723 / 696 (inputs that change: 823 / 793), 188: 126 / 109; 624 tokens of 8192 / 3584:
// 112 / 104, 147: 66 / 55, 65: 59 / 49.
template <int BN>
struct F8Cfg {
  static constexpr int A_BYTES = F8_BM * F8_BK;
  static constexpr int B_BYTES = BN * F8_BK;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 256 ? 4 : BN == 128 ? 6 : 8;
  static constexpr int HALVES = BN == 256 ? 2 : 1;              // a wide tile's halves have accumulators of their own: one is drained while the other is formed
  static constexpr int BH = BN / HALVES;
  static constexpr int NACC = BN == 256 ? 2 : 4;                // TMEM accumulator stages of a half
  static constexpr int TMEM_COLS = NACC * BN;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
  static constexpr int COLS = BN == 64 ? 32 : 64;               // columns of one epilogue warp
  static constexpr int EPI_WARPS = 4 * (BN / COLS);
  static constexpr int HALF_WARPS = EPI_WARPS / HALVES;
  static constexpr int THREADS = 128 + 32 * EPI_WARPS;
};

template <int BN>
__global__ void __launch_bounds__(F8Cfg<BN>::THREADS, 1)
gemm_fp8_block_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const float* __restrict__ xs, const float* __restrict__ ws, __nv_bfloat16* __restrict__ C, int M, int N, int K,
                      int ldc, int xs_stride, int ws_stride) {
  using Cfg = F8Cfg<BN>;
  constexpr int STAGES = Cfg::STAGES, NACC = Cfg::NACC, COLS = Cfg::COLS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * Cfg::A_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = tfull + NACC * Cfg::HALVES;                // (both [half][stage])
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tempty + NACC * Cfg::HALVES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = (M + F8_BM - 1) / F8_BM, n_tiles = (N + BN - 1) / BN;
  const int num_tiles = m_tiles * n_tiles;
  const int num_kb = (K + F8_BK - 1) / F8_BK;

  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < NACC * Cfg::HALVES; ++i) { mbar_init(&tfull[i], 1); mbar_init(&tempty[i], Cfg::HALF_WARPS); }
    fence_barrier_init();
  }
  if (warp == 2) { tmem_alloc(tmem_ptr, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  // (producer and issuer keep their warp together and elect a lane: addresses and descriptors stay in uniform registers)
  if (warp < 4) {
    if constexpr (BN == 256) regs_down<32>();
    if (warp == 0) {
      const bool one = elect_one();
      int stage = 0; uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
        const int m_blk = tile % m_tiles, n_blk = tile / m_tiles;
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait_brief(&empty[stage], phase ^ 1);
          if (one) {
            mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
            tma_load_2d(sA + stage * Cfg::A_BYTES, &tmA, &full[stage], kb * F8_BK, m_blk * F8_BM);
            tma_load_2d(sB + stage * Cfg::B_BYTES, &tmB, &full[stage], kb * F8_BK, n_blk * BN);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    } else if (warp == 1) {
      constexpr uint32_t idesc = make_idesc(UMMA_E4M3, UMMA_E4M3, F8_BM, Cfg::BH, 0, 0);
      const uint64_t da = make_smem_desc_sw128(smem_u32(sA), 0, 1024), db = make_smem_desc_sw128(smem_u32(sB), 0, 1024);
      const bool one = elect_one();
      int stage = 0; uint32_t phase = 0;
      int acc = 0; uint32_t acc_phase = 0;
      for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait_brief(&full[stage], phase);
#pragma unroll
          for (int h = 0; h < Cfg::HALVES; ++h) {
            mbar_wait_brief(&tempty[h * NACC + acc], acc_phase ^ 1);
            tc_fence_after();
            const uint64_t adesc = da + stage * (Cfg::A_BYTES / 16), bdesc = db + stage * (Cfg::B_BYTES / 16) + h * (Cfg::BH * F8_BK / 16);
            if (one) {
#pragma unroll
              for (int k = 0; k < F8_BK / 32; ++k) umma_f8_ss(tmem_base + (h * NACC + acc) * Cfg::BH, adesc + 2 * k, bdesc + 2 * k, idesc, k != 0);
              umma_commit(&tfull[h * NACC + acc]);
            }
          }
          if (one) umma_commit(&empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
          if (++acc == NACC) { acc = 0; acc_phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else {
    if constexpr (BN == 256) regs_up<112>();
    const int q = warp & 3, c0 = ((warp - 4) >> 2) * COLS;          // a warp reads the TMEM lanes of its index modulo 4
    const int half = c0 / Cfg::BH;
    uint64_t *my_full = tfull + half * NACC, *my_empty = tempty + half * NACC;
    const uint32_t t_half = tmem_base + ((uint32_t)(q * 32) << 16) + half * NACC * Cfg::BH + c0 % Cfg::BH;
    const bool wide = (ldc & 15) == 0 && (reinterpret_cast<uintptr_t>(C) & 31) == 0;      // 32-byte stores: whole sectors of a row by one lane
    const float *xs_row, *ws_row;
    auto scales_of = [&](int tile) {                          // the warp's columns (64 from a multiple of 64) lie in one 128-wide weight block
      xs_row = xs + (size_t)min((tile % m_tiles) * F8_BM + q * 32 + lane, M - 1) * xs_stride;
      ws_row = ws + (size_t)(min(tile / m_tiles * BN + c0, N - 1) >> 7) * ws_stride;
    };
    int acc = 0; uint32_t acc_phase = 0;
    scales_of(min((int)blockIdx.x, num_tiles - 1));
    float a_scale = __ldg(xs_row), w_scale = __ldg(ws_row);
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const int row = (tile % m_tiles) * F8_BM + q * 32 + lane, col0 = tile / m_tiles * BN + c0;
      float2 sum[COLS / 2];
#pragma unroll
      for (int i = 0; i < COLS / 2; ++i) sum[i] = make_float2(0.f, 0.f);
      for (int kb = 0; kb < num_kb; ++kb) {
        const float s = a_scale * w_scale;
        // the next block's scales; those of the next tile's first block while this tile ends
        if (kb + 1 == num_kb) scales_of(min(tile + (int)gridDim.x, num_tiles - 1));
        const int next = kb + 1 == num_kb ? 0 : kb + 1;
        a_scale = __ldg(xs_row + next);
        w_scale = __ldg(ws_row + next);
        mbar_wait_brief(&my_full[acc], acc_phase);
        tc_fence_after();
        const uint32_t t_row = t_half + acc * Cfg::BH;
        // sixteen columns are multiplied while the next are on their way; the accumulator is free once all of them are in registers
        uint32_t r[2][16];
        tmem_ld_32x32b_x16(t_row, r[0]);
#pragma unroll
        for (int c = 0; c < COLS; c += 16) {
          uint32_t (&v)[16] = r[(c >> 4) & 1];
          tmem_ld_wait();
          if (c + 16 < COLS) {
            tmem_ld_32x32b_x16(t_row + c + 16, r[((c >> 4) & 1) ^ 1]);
          } else {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&my_empty[acc]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) fma_pair(sum[c / 2 + i], s, v[2 * i], v[2 * i + 1]);
        }
        if (++acc == NACC) { acc = 0; acc_phase ^= 1; }
      }
      if (row < M) {
        __nv_bfloat16* dst = C + (size_t)row * ldc + col0;
#pragma unroll
        for (int v = 0; v < COLS / 16; ++v) {
          uint32_t o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = pack_bf16(sum[v * 8 + i].x, sum[v * 8 + i].y);
          if (wide && col0 + v * 16 + 8 < N) {
            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + v * 16), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]),
                         "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
          } else {
            if (col0 + v * 16 < N) st128(dst + v * 16, U4{o[0], o[1], o[2], o[3]});
            if (col0 + v * 16 + 8 < N) st128(dst + v * 16 + 8, U4{o[4], o[5], o[6], o[7]});
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
}

template <int BN>
static void launch_fp8(const void* A, const float* xs, const void* W, const float* ws, void* C, int M, int N, int K, int lda, int ldw,
                       int ldc, int xs_stride, int ws_stride, int num_sms, cudaStream_t stream) {
  using Cfg = F8Cfg<BN>;
  uint64_t dA[2] = {(uint64_t)K, (uint64_t)M}, sAs[1] = {(uint64_t)lda};
  uint64_t dB[2] = {(uint64_t)K, (uint64_t)N}, sBs[1] = {(uint64_t)ldw};
  uint32_t bA[2] = {F8_BK, F8_BM}, bB[2] = {F8_BK, (uint32_t)BN};
  CUtensorMap tmA = make_tmap(A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, dA, sAs, bA, CU_TENSOR_MAP_SWIZZLE_128B);
  CUtensorMap tmB = make_tmap(W, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, dB, sBs, bB, CU_TENSOR_MAP_SWIZZLE_128B);
  auto kern = gemm_fp8_block_kernel<BN>;
  static bool configured = false;
  if (!configured) {
    SGLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    configured = true;
  }
  const int m_tiles = (M + F8_BM - 1) / F8_BM, n_tiles = (N + BN - 1) / BN;
  const int grid = (int)std::min<long long>((long long)m_tiles * n_tiles, num_sms);
  kern<<<grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream>>>(tmA, tmB, xs, ws, (__nv_bfloat16*)C, M, N, K, ldc, xs_stride, ws_stride);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------- decode shapes: weights as the UMMA M dimension
// Bound by streaming the weights.  Every CTA owns (128 weight rows) x (a share of the K blocks); the CTAs of a cluster share one tile, park their
// fp32 partial sums in their own shared memory and each adds up (in rank order) and writes an equal part of the tokens.  Small CTAs (three 16 KB
// weight stages): an SM holds four, three or two of them at 16, 32 and 64 tokens, which keep 192, 144 or 96 KB of weights in flight and hide one
// another's start and end.
// Measured, 9 tokens, [7168 x 8192] and [8192 x 3584]: 43.6 -> 15.1 us a product on average (the version before ran 32-wide tiles of 128 padded rows).
constexpr int F8S_THREADS = 192;
template <int NT>
struct F8SwapCfg {
  static constexpr int W_BYTES = 128 * F8_BK;
  static constexpr int STAGE_BYTES = W_BYTES + NT * F8_BK;
  static constexpr int STAGES = 3;
  // accumulator stages: the CTAs that shared memory lets onto an SM never want more than its 512 TMEM columns (a cluster must not wait for them)
  static constexpr int NACC = NT <= 32 ? 4 : 2;
  static constexpr int TMEM_COLS = NACC * NT;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 8 * NT * 4 + 256 + 1024;
  static_assert((228 * 1024 / (SMEM_BYTES + 1024)) * TMEM_COLS <= 512, "TMEM columns of the co-resident CTAs");
  static_assert(NT * 128 * 4 <= STAGES * STAGE_BYTES, "the partial sums reuse the stages");
};

template <int NT>
__global__ void __launch_bounds__(F8S_THREADS)
gemm_fp8_swap_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const float* __restrict__ xs,
                     const float* __restrict__ ws, __nv_bfloat16* __restrict__ C, int M, int N, int K, int ldc, int xs_stride, int ws_stride, int splits) {
  using Cfg = F8SwapCfg<NT>;
  constexpr int STAGES = Cfg::STAGES, NACC = Cfg::NACC;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = smem + STAGES * Cfg::W_BYTES;
  float* s_scale = reinterpret_cast<float*>(smem + STAGES * Cfg::STAGE_BYTES);     // [warp][2][NT] token scales of a K block, a copy per warp
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_scale + 8 * NT);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = bars + 2 * STAGES + NACC;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2 * NACC);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / splits, rank = blockIdx.x % splits;
  const int num_kb = (K + F8_BK - 1) / F8_BK;
  const int kb0 = num_kb * rank / splits, kb1 = num_kb * (rank + 1) / splits;

  if (warp == 5 && lane == 0) { tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX); }
  if (warp == 4 && lane == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < NACC; ++i) { mbar_init(&tfull[i], 1); mbar_init(&tempty[i], 4); }
    fence_barrier_init();
  }
  if (warp == 0) { tmem_alloc(tmem_ptr, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  if (warp == 5) {
    const bool one = elect_one();
    int stage = 0; uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(&empty[stage], phase ^ 1);
      if (one) {
        mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
        tma_load_2d(sW + stage * Cfg::W_BYTES, &tmW, &full[stage], kb * F8_BK, tile * 128);
        tma_load_2d(sX + stage * NT * F8_BK, &tmX, &full[stage], kb * F8_BK, 0);
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    __syncwarp();
  } else if (warp == 4) {
    constexpr uint32_t idesc = make_idesc(UMMA_E4M3, UMMA_E4M3, 128, NT, 0, 0);
    const uint64_t dw = make_smem_desc_sw128(smem_u32(sW), 0, 1024), dx = make_smem_desc_sw128(smem_u32(sX), 0, 1024);
    const bool one = elect_one();
    int stage = 0; uint32_t phase = 0;
    int acc = 0; uint32_t acc_phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(&tempty[acc], acc_phase ^ 1);
      mbar_wait(&full[stage], phase);
      tc_fence_after();
      const uint64_t wdesc = dw + stage * (Cfg::W_BYTES / 16), xdesc = dx + stage * (NT * F8_BK / 16);
      if (one) {
#pragma unroll
        for (int k = 0; k < F8_BK / 32; ++k) umma_f8_ss(tmem_base + acc * NT, wdesc + 2 * k, xdesc + 2 * k, idesc, k != 0);
        umma_commit(&empty[stage]);
        umma_commit(&tfull[acc]);
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
      if (++acc == NACC) { acc = 0; acc_phase ^= 1; }
    }
    __syncwarp();
  } else {
    float sum[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) sum[i] = 0.f;
    const float* ws_row = ws + (size_t)tile * ws_stride;                // 128 rows from a multiple of 128: one scale per K block
    float* mine = s_scale + warp * 2 * NT;
    constexpr int PL = (NT + 31) / 32;
    float nx[PL];
    auto fetch = [&](int kb) {
      const float w = __ldg(ws_row + kb);
#pragma unroll
      for (int i = 0; i < PL; ++i) nx[i] = i * 32 + lane < M ? __ldg(xs + (size_t)(i * 32 + lane) * xs_stride + kb) * w : 0.f;
    };
    if (kb0 < kb1) fetch(kb0);
    int acc = 0; uint32_t acc_phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      float* sc = mine + (kb & 1) * NT;
#pragma unroll
      for (int i = 0; i < PL; ++i)
        if (i * 32 + lane < NT) sc[i * 32 + lane] = nx[i];
      if (kb + 1 < kb1) fetch(kb + 1);
      __syncwarp();                     // (the other half is rewritten only after every lane has passed the next one)
      mbar_wait(&tfull[acc], acc_phase);
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16) + acc * NT;
#pragma unroll
      for (int c = 0; c < NT; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_row + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 f = *reinterpret_cast<const float4*>(sc + c + i);
          sum[c + i] = fmaf(f.x, __uint_as_float(r[i]), sum[c + i]);
          sum[c + i + 1] = fmaf(f.y, __uint_as_float(r[i + 1]), sum[c + i + 1]);
          sum[c + i + 2] = fmaf(f.z, __uint_as_float(r[i + 2]), sum[c + i + 2]);
          sum[c + i + 3] = fmaf(f.w, __uint_as_float(r[i + 3]), sum[c + i + 3]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
      if (++acc == NACC) { acc = 0; acc_phase ^= 1; }
    }
    const int n = tile * 128 + threadIdx.x;
    if (splits == 1) {
      if (n < N) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
          if (j < M) C[(size_t)j * ldc + n] = __float2bfloat16(sum[j]);
      }
    } else {
      // the last block's accumulator is drained, so its multiplications have read the stages: their memory takes the partial sums
      float* part = reinterpret_cast<float*>(smem);
#pragma unroll
      for (int j = 0; j < NT; ++j) part[j * 128 + threadIdx.x] = sum[j];
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  if (splits > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int n = tile * 128 + threadIdx.x;
    if (threadIdx.x < 128 && n < N) {
      const int j1 = min(M, NT * (rank + 1) / splits);
      const uint32_t base = smem_u32(smem) + threadIdx.x * 4;
      for (int j = NT * rank / splits; j < j1; ++j) {
        float v[8], t = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          uint32_t a;
          v[r] = 0.f;
          if (r < splits) {
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(base + j * 512), "r"(r));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[r]) : "r"(a) : "memory");
          }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) t += v[r];
        C[(size_t)j * ldc + n] = __float2bfloat16(t);
      }
    }
    // nobody leaves while a peer still reads its partial sums
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

template <int NT>
static void launch_fp8_swap(const void* A, const float* xs, const void* W, const float* ws, void* C, int M, int N, int K, int lda, int ldw,
                            int ldc, int xs_stride, int ws_stride, int num_sms, cudaStream_t stream) {
  using Cfg = F8SwapCfg<NT>;
  uint64_t dW[2] = {(uint64_t)K, (uint64_t)N}, sWs[1] = {(uint64_t)ldw};
  uint64_t dX[2] = {(uint64_t)K, (uint64_t)M}, sXs[1] = {(uint64_t)lda};
  uint32_t bW[2] = {F8_BK, 128}, bX[2] = {F8_BK, (uint32_t)NT};
  CUtensorMap tmW = make_tmap(W, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, dW, sWs, bW, CU_TENSOR_MAP_SWIZZLE_128B);
  CUtensorMap tmX = make_tmap(A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, dX, sXs, bX, CU_TENSOR_MAP_SWIZZLE_128B);
  auto kern = gemm_fp8_swap_kernel<NT>;
  SGLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
  const int tiles = (N + 127) / 128, num_kb = (K + F8_BK - 1) / F8_BK;
  // share a tile's K blocks while the CTAs fit the chip at once and each still has two blocks to stream
  const int slots = num_sms * (228 * 1024 / (Cfg::SMEM_BYTES + 1024));
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= slots && num_kb >= splits * 4) splits *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * splits); cfg.blockDim = dim3(F8S_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM_BYTES; cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  SGLB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, xs, ws, (__nv_bfloat16*)C, M, N, K, ldc, xs_stride, ws_stride, splits));
}

void gemm_fp8_block(const void* A, const float* xs, const void* W, const float* ws, void* C, int M, int N, int K, int lda, int ldw,
                    int ldc, int xs_stride, int ws_stride, bool fixed_order, int num_sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return;
  if (K % 16 || N % 8 || lda % 16 || ldw % 16) throw std::runtime_error("sglb fp8 gemm: K, lda, ldw must be multiples of 16 and N of 8");
#define SGLB_F8(F) F(A, xs, W, ws, C, M, N, K, lda, ldw, ldc, xs_stride, ws_stride, num_sms, stream)
  // Up to 64 tokens: a promotion thread holds its weight row's 64 sums and an SM two CTAs.  128 sums leave one CTA an SM behind one serial chain, so
  // from 65 tokens on the rows of A are the M dimension.  us at [7168 x 8192] / [8192 x 3584] / [28672 x 4096] / [4096 x 14336], weights from memory:
  // 64 tokens 21 / 13 / 30 / 18 here, 27 / 14 / 26 / 44 there; 65 tokens 44 / 30 / 60 / 54 here (128 tokens wide), 27 / 15 / 26 / 44 there
  // fixed_order: the swapped kernel's shares of K follow the token bucket, the other kernel adds K block by block at any M and width
  if (!fixed_order) {
    if (M <= 16) { SGLB_F8(launch_fp8_swap<16>); return; }
    if (M <= 32) { SGLB_F8(launch_fp8_swap<32>); return; }
    if (M <= 64) { SGLB_F8(launch_fp8_swap<64>); return; }
  }
  // the width whose waves take the least time: a tile costs its columns plus a start and an end worth about 32 of them
  const int m_tiles = (M + F8_BM - 1) / F8_BM;
  int bn = 0;
  long long best = 0;
  for (int w : {256, 128, 64}) {
    const long long tiles = (long long)m_tiles * ((N + w - 1) / w), cost = (tiles + num_sms - 1) / num_sms * (w + 32);
    if (!bn || cost < best) { bn = w; best = cost; }
  }
  switch (bn) {
    case 256: SGLB_F8(launch_fp8<256>); break;
    case 128: SGLB_F8(launch_fp8<128>); break;
    default: SGLB_F8(launch_fp8<64>); break;
  }
#undef SGLB_F8
}

// ---------------------------------------------------------------- activation quantiser: one warp per (row, 128-group)
__global__ void __launch_bounds__(256) per_token_group_quant_fp8_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q,
                                                                        float* __restrict__ scales, int M, int K, int x_stride,
                                                                        int groups, int ue8m0) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= M * groups) return;
  const int row = gw / groups, g = gw % groups;
  const int col = g * 128 + lane * 4;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (col + 3 < K && ((x_stride & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 7) == 0)) {      // (rows of another stride are read value by value)
    const uint2 raw = *reinterpret_cast<const uint2*>(x + (size_t)row * x_stride + col);
    v[0] = bf16_lo(raw.x); v[1] = bf16_hi(raw.x); v[2] = bf16_lo(raw.y); v[3] = bf16_hi(raw.y);
  } else {
    for (int i = 0; i < 4; ++i)
      if (col + i < K) v[i] = __bfloat162float(x[(size_t)row * x_stride + col + i]);
  }
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  amax = warp_max(amax);
  float scale = fmaxf(amax, 1e-10f) / 448.f;
  if (ue8m0) scale = exp2f(ceilf(log2f(scale)));
  const float inv = 1.f / scale;
  if (lane == 0) scales[(size_t)row * groups + g] = scale;
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_fp8_storage_t b = __nv_cvt_float_to_fp8(v[i] * inv, __NV_SATFINITE, __NV_E4M3);
    packed |= (uint32_t)b << (8 * i);
  }
  if (col + 3 < K) {
    *reinterpret_cast<uint32_t*>(q + (size_t)row * K + col) = packed;
  } else {
    for (int i = 0; i < 4; ++i)
      if (col + i < K) q[(size_t)row * K + col + i] = (uint8_t)(packed >> (8 * i));
  }
}

// 16-byte rows: a thread takes eight values, half a warp a group, and a warp four groups whose loads are all in flight together.
// [3001, 4096] and [3001, 14336], on average: 36 -> 20 us (it was one 8-byte load a lane and a warp per group).
__global__ void __launch_bounds__(256) per_token_group_quant_fp8_vec_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q,
                                                                            float* __restrict__ scales, long long total, int K, int x_stride,
                                                                            int groups, int ue8m0) {
  const int lane = threadIdx.x & 31, half = lane >> 4, l = lane & 15;
  const long long g0 = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * 4 + half;
  U4 raw[2];
  int row[2], col[2], grp[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const long long g = g0 + 2 * i;
    row[i] = g < total ? (int)((unsigned)g / (unsigned)groups) : -1;
    grp[i] = row[i] < 0 ? 0 : (int)((unsigned)g - (unsigned)row[i] * (unsigned)groups);
    col[i] = grp[i] * 128 + l * 8;
    raw[i] = row[i] >= 0 && col[i] < K ? ldg128(x + (size_t)row[i] * x_stride + col[i]) : U4{0, 0, 0, 0};
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float v[8] = {bf16_lo(raw[i].x), bf16_hi(raw[i].x), bf16_lo(raw[i].y), bf16_hi(raw[i].y),
                        bf16_lo(raw[i].z), bf16_hi(raw[i].z), bf16_lo(raw[i].w), bf16_hi(raw[i].w)};
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    float scale = fmaxf(amax, 1e-10f) / 448.f;
    if (ue8m0) scale = exp2f(ceilf(log2f(scale)));
    const float inv = 1.f / scale;
    if (row[i] < 0) continue;
    if (l == 0) scales[(size_t)row[i] * groups + grp[i]] = scale;
    if (col[i] >= K) continue;
    uint32_t w[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j] * inv, v[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j + 2] * inv, v[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
      w[j] = lo | hi << 16;
    }
    *reinterpret_cast<uint2*>(q + (size_t)row[i] * K + col[i]) = make_uint2(w[0], w[1]);
  }
}

void per_token_group_quant_fp8(const void* x, void* q, float* scales, int M, int K, int x_stride, bool ue8m0, cudaStream_t stream) {
  if (M <= 0) return;
  if (K % 4) throw std::runtime_error("sglb fp8 quant: K must be a multiple of 4");
  const int groups = (K + 127) / 128;
  const long long warps = (long long)M * groups;
  if (K % 8 == 0 && x_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0 && warps < (1ll << 31)) {
    per_token_group_quant_fp8_vec_kernel<<<(int)((warps + 31) / 32), 256, 0, stream>>>((const __nv_bfloat16*)x, (uint8_t*)q, scales, warps, K, x_stride,
                                                                                       groups, ue8m0);
    SGLB_CUDA_CHECK(cudaGetLastError());
    return;
  }
  const int grid = (int)((warps * 32 + 255) / 256);
  per_token_group_quant_fp8_kernel<<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, (uint8_t*)q, scales, M, K, x_stride, groups, ue8m0);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

}  // namespace sglb
