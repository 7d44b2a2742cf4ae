// Expert-grouped GEMM for decode batches (few rows per expert) on tcgen05:  C[row, n] = epilogue( X[row, :] . W[expert(row)][n, :] )
//
// Bound by streaming the experts' weights, so the weights are the UMMA M dimension (128 rows of W fill every tensor lane and every TMA byte is
// useful) and the expert's rows - a tile of 16 / 32 / 64 / 128 from moe_align - the N dimension.  One CTA per (128 weight rows, row tile, share of K);
// the CTAs of a cluster share one tile's K and add their fp32 partial sums through distributed shared memory in rank order.  Small CTAs: three of
// them per SM (two at 128 rows) keep about 200 KB of weights in flight and hide one another's start and end.  From 3 to 36 rows an expert on
// gemm_grouped_pair.cu is faster, but for narrow experts and for few of them, whose tiles do not fill the pairs of SMs (the line: moe_plan in binding.cpp).
//
//   warps 0..3 : epilogue      warp 4 : MMA issuer      warp 5 : TMA producer
//
// The kernel it replaced for these shapes (gemm_tc.cu, grouped) gave 128 TMEM lanes and two thirds of its shared memory to padding rows.
// Measured, bf16, both products of a block: 20 tokens, 8 experts of 4096 x 14336, 2 each: 617 -> 425 us (2.8 GB of weights, 6.6 TB/s); 128 experts of
// 2048 x 192 at 16 rows each: 138 -> 101 us.
#include "common.cuh"
#include "tma_host.h"

#include <algorithm>

namespace sglb {

enum GroupedEpilogue { GD_NONE = 0, GD_SILU = 1, GD_ROWSCALE = 2, GD_RELU2 = 3 };
constexpr int GD_THREADS = 192;
constexpr int GD_BK = 64;

template <int NT>
struct GdCfg {
  static constexpr int W_BYTES = 128 * GD_BK * 2;
  static constexpr int X_BYTES = NT * GD_BK * 2;
  static constexpr int STAGES = NT == 16 ? 4 : 3;
  static constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
  static constexpr int TMEM_COLS = NT < 32 ? 32 : NT;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + NT * 4 + 128 + 1024;
  static_assert((228 * 1024 / (SMEM_BYTES + 1024)) * TMEM_COLS <= 512, "a cluster must never wait for TMEM columns");
  static_assert(NT * 128 * 4 <= STAGES * STAGE_BYTES, "the partial sums reuse the stages");
};

__device__ __forceinline__ float gd_peer(uint32_t addr, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

template <int NT, int EPI>
__global__ void __launch_bounds__(GD_THREADS)
gemm_grouped_decode_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, __nv_bfloat16* __restrict__ C,
                           const float* __restrict__ row_scale, const int* __restrict__ sorted_row, const int* __restrict__ tile_expert,
                           const int* __restrict__ num_tiles, int max_tiles, int n_out, int K, int ldc, int splits) {
  using Cfg = GdCfg<NT>;
  constexpr int STAGES = Cfg::STAGES;
  constexpr bool SILU = EPI == GD_SILU;
  constexpr int BN = SILU ? 64 : 128;                     // output columns: gate rows and their up rows share the 128 lanes
  const int rank = blockIdx.x % splits, tile = (blockIdx.x / splits) % max_tiles, n0 = blockIdx.x / splits / max_tiles * BN;
  if (tile >= min(__ldg(num_tiles), max_tiles)) return;   // (the whole cluster)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = smem + STAGES * Cfg::W_BYTES;
  int* s_row = reinterpret_cast<int*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(s_row + NT);
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (K + GD_BK - 1) / GD_BK;
  const int kb0 = num_kb * rank / splits, kb1 = num_kb * (rank + 1) / splits;

  if (warp == 5 && lane == 0) { tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX); }
  if (warp == 4 && lane == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 0) { tmem_alloc(tmem_ptr, Cfg::TMEM_COLS); tmem_relinquish(); }
  int row = -1;
  if (threadIdx.x < NT) s_row[threadIdx.x] = row = __ldg(sorted_row + tile * NT + threadIdx.x);
  tc_fence_before();
  // live rows come first in a tile: only they are loaded and multiplied, in steps of 16 (what the SM takes in is what bounds the kernel)
  const int live = __syncthreads_count(row >= 0), blocks = NT == 16 ? 1 : (live + 15) / 16;
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;

  // (both roles keep their warp together and elect a lane: addresses and descriptors stay in uniform registers)
  if (warp == 5) {
    const int expert = __ldg(tile_expert + tile);
    const bool one = elect_one();
    int stage = 0; uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(&empty[stage], phase ^ 1);
      if (one) {
        mbar_expect_tx(&full[stage], Cfg::W_BYTES + blocks * 16 * GD_BK * 2);
        uint8_t* w = sW + stage * Cfg::W_BYTES;
        tma_load_3d(w, &tmW, &full[stage], kb * GD_BK, n0, expert);
        if (SILU) tma_load_3d(w + Cfg::W_BYTES / 2, &tmW, &full[stage], kb * GD_BK, n_out + n0, expert);
        for (int b = 0; b < blocks; ++b) tma_load_2d(sX + stage * Cfg::X_BYTES + b * 16 * GD_BK * 2, &tmX, &full[stage], kb * GD_BK, tile * NT + b * 16);
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    __syncwarp();
  } else if (warp == 4) {
    const uint32_t idesc = make_idesc(UMMA_BF16, UMMA_BF16, 128, blocks * 16, 0, 0);
    const uint64_t dw = make_smem_desc_sw128(smem_u32(sW), 0, 1024), dx = make_smem_desc_sw128(smem_u32(sX), 0, 1024);
    const bool one = elect_one();
    int stage = 0; uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(&full[stage], phase);
      tc_fence_after();
      const uint64_t wdesc = dw + stage * (Cfg::W_BYTES / 16), xdesc = dx + stage * (Cfg::X_BYTES / 16);
      if (one) {
#pragma unroll
        for (int k = 0; k < GD_BK / 16; ++k) umma_f16_ss(tmem, wdesc + 2 * k, xdesc + 2 * k, idesc, kb != kb0 || k != 0);
        umma_commit(&empty[stage]);
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (one) umma_commit(done);
    __syncwarp();
  } else {
    // every multiplication is done, so nothing reads the stages any more: they take the partial sums, [row of the tile][weight row]
    mbar_wait(done, 0);
    tc_fence_after();
    float* part = reinterpret_cast<float*>(smem);
#pragma unroll 1
    for (int c = 0; c < blocks * 16; c += 16) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(tmem + ((uint32_t)(warp * 32) << 16) + c, r);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) part[(c + i) * 128 + threadIdx.x] = __uint_as_float(r[i]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, Cfg::TMEM_COLS);
  if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x < 128) {
    const int t = threadIdx.x, n = SILU ? t & 63 : t;
    const int j0 = blocks * 16 * rank / splits, j1 = blocks * 16 * (rank + 1) / splits;
    const float* part = reinterpret_cast<const float*>(smem);
    const uint32_t base = smem_u32(smem);
    auto total = [&](int at) {
      if (splits == 1) return part[at];
      float v[8], s = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = r < splits ? gd_peer(base + at * 4, r) : 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) s += v[r];
      return s;
    };
    if (n0 + n < n_out)
      for (int j = j0 + (SILU ? t >> 6 : 0); j < j1; j += SILU ? 2 : 1) {
        if (s_row[j] < 0) continue;
        float v = total(j * 128 + n);
        if (SILU) {
          const float u = total(j * 128 + 64 + n);
          v = v / (1.f + __expf(-v)) * u;
        }
        if (EPI == GD_RELU2) { v = fmaxf(v, 0.f); v *= v; }
        if (EPI == GD_ROWSCALE) v *= __ldg(row_scale + tile * NT + j);
        C[(size_t)(tile * NT + j) * ldc + n0 + n] = __float2bfloat16(v);
      }
  }
  // nobody leaves while a peer still reads its partial sums
  if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int NT, int EPI>
static void launch_grouped_decode(const void* X, const void* W, void* C, const float* row_scale, const int* sorted_row, int n_out, int K, int lda, int ldc,
                                  int E, const int* tile_expert, const int* num_tiles, int max_tiles, int live_tiles, int num_sms, cudaStream_t stream) {
  using Cfg = GdCfg<NT>;
  constexpr int BN = EPI == GD_SILU ? 64 : 128;
  const int w_rows = EPI == GD_SILU ? 2 * n_out : n_out;
  uint64_t dW[3] = {(uint64_t)K, (uint64_t)w_rows, (uint64_t)E}, sWs[2] = {(uint64_t)K * 2, (uint64_t)w_rows * K * 2};
  uint32_t bW[3] = {GD_BK, (uint32_t)BN, 1};
  uint64_t dX[2] = {(uint64_t)K, (uint64_t)max_tiles * NT}, sXs[1] = {(uint64_t)lda * 2};
  uint32_t bX[2] = {GD_BK, 16};
  CUtensorMap tmW = make_tmap(W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dW, sWs, bW, CU_TENSOR_MAP_SWIZZLE_128B);
  CUtensorMap tmX = make_tmap(X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dX, sXs, bX, CU_TENSOR_MAP_SWIZZLE_128B);
  auto kern = gemm_grouped_decode_kernel<NT, EPI>;
  SGLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
  const int n_tiles = (n_out + BN - 1) / BN, num_kb = (K + GD_BK - 1) / GD_BK;
  // share K until the live CTAs fill the chip four times over (an even last wave), while each still streams 16 blocks (256 KB)
  const long long slots = (long long)num_sms * (228 * 1024 / (Cfg::SMEM_BYTES + 1024));
  int splits = 1;
  while (splits < 8 && (long long)n_tiles * live_tiles * splits < 4 * slots && num_kb >= splits * 32) splits *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)n_tiles * max_tiles * splits); cfg.blockDim = dim3(GD_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM_BYTES; cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  SGLB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, (__nv_bfloat16*)C, row_scale, sorted_row, tile_expert, num_tiles, max_tiles, n_out, K, ldc, splits));
}

// X rows are expert-sorted with every expert's rows padded to tiles of ``tile`` (16, 32, 64 or 128; sorted_row < 0 marks padding, whose output is not
// written); W is [E][n_out or 2 n_out][K].  live_tiles: how many of max_tiles the caller expects to be live
void gemm_grouped_decode(const void* X, const void* W, void* C, const float* row_scale, const int* sorted_row, int tile, int n_out, int K, int lda, int ldc,
                         int E, const int* tile_expert, const int* num_tiles, int max_tiles, int live_tiles, int epi, int num_sms, cudaStream_t stream) {
  if (max_tiles <= 0 || n_out <= 0) return;
  if (K % 8 || lda % 8) throw std::runtime_error("sglb grouped decode gemm: K % 8, lda % 8 required");
#define GD_RUN(NT, EPI) \
  launch_grouped_decode<NT, EPI>(X, W, C, row_scale, sorted_row, n_out, K, lda, ldc, E, tile_expert, num_tiles, max_tiles, live_tiles, num_sms, stream)
#define GD_EPI(NT)                                       \
  switch (epi) {                                         \
    case GD_SILU: GD_RUN(NT, GD_SILU); break;            \
    case GD_ROWSCALE: GD_RUN(NT, GD_ROWSCALE); break;    \
    case GD_RELU2: GD_RUN(NT, GD_RELU2); break;          \
    default: GD_RUN(NT, GD_NONE); break;                 \
  }
  switch (tile) {
    case 16: GD_EPI(16); break;
    case 32: GD_EPI(32); break;
    case 64: GD_EPI(64); break;
    case 128: GD_EPI(128); break;
    default: throw std::runtime_error("sglb grouped decode gemm: row tile must be 16, 32, 64 or 128");
  }
#undef GD_EPI
#undef GD_RUN
}

}  // namespace sglb
