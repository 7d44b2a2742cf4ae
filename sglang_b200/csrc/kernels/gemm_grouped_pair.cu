// Expert-grouped GEMM of prompts (many rows per expert) on pairs of SMs:  C[row, n] = epilogue( X[row, :] . W[expert(row)][n, :] )
//
// Bound by the tensor cores, and before them by what L2 hands to the SMs: a 128 x 256 tile of one CTA takes 96 bytes a cycle and SM.  Here two CTAs work on
// one tile (tcgen05 cta_group::2): 256 weight rows are the UMMA M dimension, 128 from each CTA, and up to 256 tokens of an expert the N dimension, half of
// them from each, so that every operand byte is loaded by one SM only (64 bytes a cycle).  Weights as M leave the number of tokens free in steps of 16: an
// expert's rows are cut into tiles of one size, none of which is padded to 128.
//
//   warps 0, 3 : TMA producers of W and X (each CTA loads its own rows; the even CTA's barrier counts both)
//   warp 1 : MMA issuer (even CTA)      warp 2 : TMEM allocation, two accumulators of 256 columns      warps 4..7 : epilogue
//
// In the accumulator lanes are output features and columns tokens: two lanes exchange a value, so that a store takes two features of a token.  For
// silu(gate) * up a CTA's lanes are 64 gate rows and their 64 up rows, which swap halves of their tokens through shared memory.
#include "common.cuh"
#include "tma_host.h"

#include <algorithm>

namespace sglb {

enum GroupedPairEpilogue { GP_NONE = 0, GP_SILU = 1, GP_ROWSCALE = 2, GP_RELU2 = 3 };
constexpr int GP_THREADS = 256, GP_BK = 64, GP_STAGES = 6;
constexpr int GP_A_BYTES = 128 * GP_BK * 2, GP_B_BYTES = 128 * GP_BK * 2, GP_STAGE_BYTES = GP_A_BYTES + GP_B_BYTES;
constexpr int GP_XBOX = 32;                                   // rows of a TMA copy of X: a map each for one to four times as many
struct GpMaps { CUtensorMap x[4]; };
constexpr int GP_MAX_E = 512, GP_LIST = 2048;                 // experts, row tiles
constexpr int GP_SWAP = 2 * 4 * 16 * 32 * 4;                  // [buffer][warp][token][lane]: what gate and up warps hand each other
constexpr int GP_SMEM = GP_STAGES * GP_STAGE_BYTES + GP_SWAP + GP_LIST * 8 + 256 + 1024;

__device__ __forceinline__ uint32_t gp_leader(const void* p) {            // the same address in the even CTA of the pair
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(0));
  return a;
}
__device__ __forceinline__ void gp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void gp_load_2d(void* dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void gp_load_4d(void* dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void gp_commit(uint64_t* bar) {                // arrives at this offset in both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// The tiles of one SM pair: expert by expert, so that an expert's rows stay in L2 while its weights pass, and those who share weights follow one another
struct GpWork {
  const uint2* tiles;
  int item, step, items, f_blocks, first = 0, base = 0;
  int row0, n, expert, f_block;
  __device__ __forceinline__ GpWork(const uint2* t, int start, int step_, int num_tiles, int fb)
      : tiles(t), item(start - step_), step(step_), items(num_tiles * fb), f_blocks(fb) {}
  __device__ __forceinline__ bool next() {
    item += step;
    if (item >= items) return false;
    int parts = tiles[first].y >> 16;
    while (item - base >= parts * f_blocks) {
      base += parts * f_blocks;
      first += parts;
      parts = tiles[first].y >> 16;
    }
    const int r = item - base;
    const uint2 t = tiles[first + r % parts];
    f_block = r / parts;
    row0 = t.x;
    n = (t.y & 31) * 16;
    expert = t.y >> 5 & 0x3ff;
    return true;
  }
};

template <int EPI>
__global__ void __launch_bounds__(GP_THREADS, 1)
gemm_grouped_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ GpMaps tmX, __nv_bfloat16* __restrict__ C,
                         const float* __restrict__ row_scale, const int* __restrict__ expert_start, int E, int n_out, int K, int ldc) {
  constexpr bool SILU = EPI == GP_SILU;
  constexpr int BF = SILU ? 128 : 256;                        // output features of a tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + GP_STAGES * GP_A_BYTES;
  float* s_swap = reinterpret_cast<float*>(smem + GP_STAGES * GP_STAGE_BYTES);
  uint2* s_tile = reinterpret_cast<uint2*>(smem + GP_STAGES * GP_STAGE_BYTES + GP_SWAP);      // first row; tokens / 16 (5 bits), expert (10; one unused), row tiles of the expert
  uint64_t* full = reinterpret_cast<uint64_t*>(s_tile + GP_LIST);
  uint64_t* empty = full + GP_STAGES;
  uint64_t* tfull = empty + GP_STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tempty + 2);
  int* s_count = reinterpret_cast<int*>(tmem_ptr + 1);        // [5]: tiles by size, then [1]: this launch's

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = blockIdx.x & 1;
  const int f_blocks = (n_out + BF - 1) / BF, num_kb = (K + GP_BK - 1) / GP_BK, pairs = gridDim.x >> 1;

  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX.x[3]); }
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < GP_STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tfull[i], 1); mbar_init(&tempty[i], 8); }
    fence_barrier_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_ptr)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }

  // Row tiles: every expert's rows in equal parts of at most `most` steps of 16.  Of five sizes the one whose rounds over the SM pairs cost least (a tile
  // costs its tokens and a start and end worth about 24 of them): 7.1 rounds of 256 tokens take 8, of 192 tokens 10.4 take 11.
  if (tid < 5) s_count[tid] = 0;
  __syncthreads();
  int steps[GP_MAX_E / GP_THREADS], row0[GP_MAX_E / GP_THREADS];
#pragma unroll
  for (int i = 0; i < GP_MAX_E / GP_THREADS; ++i) {
    const int e = tid * (GP_MAX_E / GP_THREADS) + i;
    row0[i] = e < E ? __ldg(expert_start + e) : 0;
    steps[i] = e < E ? __ldg(expert_start + e + 1) - row0[i] : 0;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int most = 16 - 2 * k;
    int n = 0;
#pragma unroll
    for (int i = 0; i < GP_MAX_E / GP_THREADS; ++i) n += (steps[i] + most - 1) / most;
    n = warp_sum(n);
    if (lane == 0 && n) atomicAdd(&s_count[k], n);
  }
  __syncthreads();
  int most = 16;
  {
    const long long total = __ldg(expert_start + E);
    float best = 0.f;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int n = s_count[k];
      if (!n) continue;
      const float cost = (float)(((long long)n * f_blocks + pairs - 1) / pairs) * (16.f * (float)total / (float)n + 24.f);
      if (k == 0 || cost < best * 0.97f) { best = cost; most = 16 - 2 * k; }
    }
  }
  int mine = 0;
#pragma unroll
  for (int i = 0; i < GP_MAX_E / GP_THREADS; ++i) mine += (steps[i] + most - 1) / most;
  int at = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += v;
  }
  __syncthreads();
  if (lane == 31) s_count[warp] = at;                         // (eight warps; the counts are done with)
  __syncthreads();
  int num_tiles = 0;
  at -= mine;
#pragma unroll
  for (int w = 0; w < GP_THREADS / 32; ++w) {
    if (w < warp) at += s_count[w];
    num_tiles += s_count[w];
  }
#pragma unroll
  for (int i = 0; i < GP_MAX_E / GP_THREADS; ++i) {
    const int parts = (steps[i] + most - 1) / most;
    for (int j = 0; j < parts; ++j) {
      const int a = steps[i] * j / parts, z = steps[i] * (j + 1) / parts;
      s_tile[at++] = make_uint2((row0[i] + a) * 16, (z - a) | (tid * (GP_MAX_E / GP_THREADS) + i) << 5 | parts << 16);
    }
  }
  tc_fence_before();
  __syncthreads();
  gp_cluster_sync();                                          // the other CTA's barriers are there
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  GpWork work(s_tile, blockIdx.x >> 1, pairs, num_tiles, f_blocks);

  if (warp == 0 || warp == 3) {
    // one copy a K block each, from two warps: one thread that issued five or six of them was what the kernel waited for (925 cycles a block instead of 512)
    const bool one = elect_one();
    int stage = 0; uint32_t phase = 0;
    while (work.next()) {
      const int expert = work.expert, f0 = work.f_block * BF, r0 = work.row0 + rank * (work.n / 2), boxes = (work.n / 2 + GP_XBOX - 1) / GP_XBOX;
      for (int kb = 0; kb < num_kb; ++kb) {
        mbar_wait(&empty[stage], phase ^ 1);
        const uint32_t bar = gp_leader(&full[stage]);
        if (one) {
          if (warp == 0) {
            if (rank == 0) mbar_expect_tx(&full[stage], 2 * (GP_A_BYTES + boxes * GP_XBOX * GP_BK * 2));
            if (SILU) gp_load_4d(sA + stage * GP_A_BYTES, &tmW, bar, kb * GP_BK, f0 + rank * 64, 0, expert);
            else gp_load_4d(sA + stage * GP_A_BYTES, &tmW, bar, kb * GP_BK, f0 + rank * 128, 0, expert);
          } else {
            gp_load_2d(sB + stage * GP_B_BYTES, &tmX.x[boxes - 1], bar, kb * GP_BK, r0);
          }
        }
        if (++stage == GP_STAGES) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      const uint64_t da = make_smem_desc_sw128(smem_u32(sA), 0, 1024), db = make_smem_desc_sw128(smem_u32(sB), 0, 1024);
      const bool one = elect_one();
      int stage = 0; uint32_t phase = 0;
      int acc = 0; uint32_t acc_phase = 0;
      while (work.next()) {
        const uint32_t idesc = make_idesc(UMMA_BF16, UMMA_BF16, 256, work.n, 0, 0);
        mbar_wait(&tempty[acc], acc_phase ^ 1);
        tc_fence_after();
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(&full[stage], phase);
          tc_fence_after();
          const uint64_t a = da + stage * (GP_A_BYTES / 16), b = db + stage * (GP_B_BYTES / 16);
          if (one) {
#pragma unroll
            for (int k = 0; k < GP_BK / 16; ++k) gp_mma(tmem + acc * 256, a + 2 * k, b + 2 * k, idesc, (kb | k) != 0);
            gp_commit(&empty[stage]);
          }
          if (++stage == GP_STAGES) { stage = 0; phase ^= 1; }
        }
        if (one) gp_commit(&tfull[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    const int q = warp - 4, odd = lane & 1;
    const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16);
    int acc = 0; uint32_t acc_phase = 0;
    int buf = 0;                                              // swap buffer of the chunk: it runs on from tile to tile, so that the barrier of one use orders the reads
                                                              // of the last use of the other (a tile of an odd number of chunks would end and begin on the same one)
    while (work.next()) {
      const int n = work.n, f0 = work.f_block * BF;
      const int f = f0 + (SILU ? rank * 64 + (q & 1) * 32 : rank * 128 + q * 32) + lane;
      __nv_bfloat16* out = C + (size_t)(work.row0 + odd) * ldc + (f & ~1);
      const bool live = f < n_out;                            // (an even number of features)
      // values of tokens t, t + 1 of this lane's feature -> two features of one token
      auto store = [&](int t, float a, float b) {
        const float other = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
        if (live && t < n) *reinterpret_cast<uint32_t*>(out + (size_t)t * ldc) = odd ? pack_bf16(other, b) : pack_bf16(a, other);
      };
      mbar_wait(&tfull[acc], acc_phase);
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < n; c += 32, buf ^= 1) {             // (n is a multiple of 16: a last half chunk holds what an earlier tile left, and is not stored)
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_lane + acc * 256 + c, r);
        tmem_ld_wait();
        if constexpr (SILU) {
          // gate warps (q < 2) finish tokens 0..15 of the chunk, up warps 16..31
          const int half = q >> 1;
          float* mine_s = s_swap + ((buf * 4 + q) * 16) * 32 + lane;
          const float* other_s = s_swap + ((buf * 4 + (q ^ 2)) * 16) * 32 + lane;
#pragma unroll
          for (int i = 0; i < 16; ++i) mine_s[i * 32] = __uint_as_float(half ? r[i] : r[16 + i]);
          asm volatile("bar.sync %0, 64;" ::"r"(1 + (q & 1)) : "memory");
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float own = __uint_as_float(half ? r[16 + i] : r[i]), their = other_s[i * 32];
            const float g = half ? their : own, u = half ? own : their;
            v[i] = g / (1.f + __expf(-g)) * u;
          }
#pragma unroll
          for (int i = 0; i < 16; i += 2) store(c + half * 16 + i, v[i], v[i + 1]);
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = __uint_as_float(r[i + k]);
            if (EPI == GP_ROWSCALE) {
              const float4 s = c + i < n ? __ldg(reinterpret_cast<const float4*>(row_scale + work.row0 + c + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
              v[0] *= s.x; v[1] *= s.y; v[2] *= s.z; v[3] *= s.w;
            }
            if (EPI == GP_RELU2) {
#pragma unroll
              for (int k = 0; k < 4; ++k) { const float a = fmaxf(v[k], 0.f); v[k] = a * a; }
            }
            store(c + i, v[0], v[1]);
            store(c + i + 2, v[2], v[3]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(gp_leader(&tempty[acc])) : "memory");
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }
  tc_fence_before();
  __syncthreads();
  gp_cluster_sync();                                          // neither CTA's barriers nor its operands are needed by the other any more
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

template <int EPI>
static void launch_grouped_pair(const void* X, const void* W, void* C, const float* row_scale, int cap_rows, int n_out, int K, int lda, int ldc, int E,
                                const int* expert_start, int num_sms, cudaStream_t stream) {
  // gate and up rows (the other products: one set of rows) are a dimension of their own, so that one copy brings both
  const uint64_t sets = EPI == GP_SILU ? 2 : 1;
  uint64_t dW[4] = {(uint64_t)K, (uint64_t)n_out, sets, (uint64_t)E}, sWs[3] = {(uint64_t)K * 2, (uint64_t)n_out * K * 2, sets * n_out * K * 2};
  uint32_t bW[4] = {GP_BK, EPI == GP_SILU ? 64u : 128u, (uint32_t)sets, 1};
  uint64_t dX[2] = {(uint64_t)K, (uint64_t)cap_rows}, sXs[1] = {(uint64_t)lda * 2};
  CUtensorMap tmW = make_tmap(W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, dW, sWs, bW, CU_TENSOR_MAP_SWIZZLE_128B);
  GpMaps tmX;
  for (int i = 0; i < 4; ++i) {
    uint32_t bX[2] = {GP_BK, (uint32_t)(GP_XBOX * (i + 1))};
    tmX.x[i] = make_tmap(X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dX, sXs, bX, CU_TENSOR_MAP_SWIZZLE_128B);
  }
  auto kern = gemm_grouped_pair_kernel<EPI>;
  SGLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(num_sms & ~1); cfg.blockDim = dim3(GP_THREADS); cfg.dynamicSmemBytes = GP_SMEM; cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  SGLB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, (__nv_bfloat16*)C, row_scale, expert_start, E, n_out, K, ldc));
}

// row tiles a launch may have to list: rows in steps of 16, at least eight of them a tile but for an expert's last
bool gemm_grouped_pair_fits(int cap_rows, int E) { return E <= GP_MAX_E && cap_rows / 128 + E <= GP_LIST; }

// X rows are expert-sorted, every expert's rows padded to 16 (padding rows may hold anything; theirs are written too); expert_start[e] counts the 16-row
// steps before expert e, expert_start[E] all.  W is [E][n_out or 2 n_out][K].  row_scale: one number a row, 16-byte aligned
void gemm_grouped_pair(const void* X, const void* W, void* C, const float* row_scale, int cap_rows, int n_out, int K, int lda, int ldc, int E,
                       const int* expert_start, int epi, int num_sms, cudaStream_t stream) {
  if (cap_rows <= 0 || n_out <= 0) return;
  if (K % 8 || lda % 8 || n_out % 2 || ldc % 2) throw std::runtime_error("sglb grouped pair gemm: K % 8, lda % 8, n_out % 2, ldc % 2 required");
#define GP_RUN(EPI) launch_grouped_pair<EPI>(X, W, C, row_scale, cap_rows, n_out, K, lda, ldc, E, expert_start, num_sms, stream)
  switch (epi) {
    case GP_SILU: GP_RUN(GP_SILU); break;
    case GP_ROWSCALE: GP_RUN(GP_ROWSCALE); break;
    case GP_RELU2: GP_RUN(GP_RELU2); break;
    default: GP_RUN(GP_NONE); break;
  }
#undef GP_RUN
}

}  // namespace sglb
