// Mixture-of-experts kernels for sm_100a (everything around the expert-grouped tcgen05 GEMM in gemm_tc.cu):
//
//   moe_topk_softmax   one warp per token: softmax over E router logits in registers, K rounds of warp arg-max,
//                      optional renormalisation of the selected weights.
//   moe_align          counting sort of the T*K (token, k) pairs by LOCAL expert into segments padded to the GEMM's row tile
//                      (128, or 16..128 for decode batches), producing sorted_row[pos] -> pair, inv_pos[pair] -> pos, the per-row
//                      routing weight, tile_expert[m_tile] and the number of live M tiles — all in device memory, so
//                      the whole MoE block is CUDA-graph capturable with no host round trip.
//   moe_gather         xs[pos,:] = x[sorted_row[pos] / K, :]     (padding rows are left as they are: nothing reads what they give), optionally times the pair's routing weight (routers
//                      whose weight multiplies an expert's input)
//   moe_combine        out[t,:] = sum_k ys[inv_pos[t*K+k],:]     (fixed k order -> deterministic), optionally PUSHED into
//                      slot [rank] of every peer's NVLink arena so the expert-parallel all-reduce needs no further kernel
//                      on the producer side (consumer: nvl_local_reduce_add_rmsnorm in comm/nvl_allreduce.cu).
//
// Reference counterparts: kernels/aot/csrc/moe/moe_topk_softmax_kernels.cu:628-715, moe_align_kernel.cu:350-386,
// python/sglang/srt/layers/moe/fused_moe_triton/fused_moe_triton_kernels.py:324 (grouped GEMM), moe_sum_reduce.
#include "common.cuh"
#include "tma_host.h"

namespace sglb {

// ---------------------------------------------------------------- top-k softmax
template <int VPT, typename T>
__global__ void __launch_bounds__(128) moe_topk_softmax_kernel(const T* __restrict__ logits, float* __restrict__ out_w,
                                                               int* __restrict__ out_ids, int n_tokens, int E, int K, int stride,
                                                               int renorm) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + warp;
  if (t >= n_tokens) return;
  float v[VPT];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int e = i * 32 + lane;
    v[i] = e < E ? (float)logits[(size_t)t * stride + e] : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    v[i] = (i * 32 + lane) < E ? __expf(v[i] - mx) : -1.f;
    sum += fmaxf(v[i], 0.f);
  }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
  float sel_sum = 0.f;
  float my_w = 0.f;
  int my_id = 0;
  for (int k = 0; k < K; ++k) {
    float best = -2.f;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
      if (v[i] > best) { best = v[i]; best_e = i * 32 + lane; }
    // warp arg-max; ties -> lowest expert id (matches torch.topk on distinct values, deterministic otherwise)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
      if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
    }
    if ((best_e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < VPT; ++i)
        if (i == (best_e >> 5)) v[i] = -1.f;
    }
    sel_sum += best;
    if (lane == k) { my_w = best; my_id = best_e; }
  }
  if (lane < K) {
    out_w[(size_t)t * K + lane] = renorm ? my_w / sel_sum : my_w * inv;
    out_ids[(size_t)t * K + lane] = my_id;
  }
}

void moe_topk_softmax(const void* logits, bool bf16, float* out_w, int* out_ids, int T, int E, int K, int stride, bool renorm,
                      cudaStream_t stream) {
  if (T <= 0) return;
  if (E > 512 || K > 32 || K > E) throw std::runtime_error("sglb moe_topk_softmax: need E <= 512, K <= min(32, E)");
  const int grid = (T + 3) / 4;
  const int vpt = (E + 31) / 32;
#define SGLB_TOPK(V)                                                                                                              \
  do {                                                                                                                            \
    if (bf16) moe_topk_softmax_kernel<V, __nv_bfloat16><<<grid, 128, 0, stream>>>((const __nv_bfloat16*)logits, out_w, out_ids, T, \
                                                                                   E, K, stride, renorm);                         \
    else moe_topk_softmax_kernel<V, float><<<grid, 128, 0, stream>>>((const float*)logits, out_w, out_ids, T, E, K, stride, renorm); \
  } while (0)
  if (vpt <= 1) SGLB_TOPK(1); else if (vpt <= 2) SGLB_TOPK(2); else if (vpt <= 4) SGLB_TOPK(4); else if (vpt <= 8) SGLB_TOPK(8);
  else SGLB_TOPK(16);
#undef SGLB_TOPK
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------- align (single CTA counting sort)
// Bound by latency: the ids are loaded once, all in flight together, and stay in registers between counting and placing; segment starts come from a
// block scan.  2664 pairs over 128 experts: 20.1 -> 6.2 us, 8002 pairs over 8: 10.3 -> 7.7 us (it was one thread's walk over the experts between two dependent
// passes over the ids).
constexpr int MOE_MAX_E = 512;
constexpr int ALIGN_THREADS = 1024;

// PER: ids per thread kept in registers (0: more than 16 K pairs, read twice)
template <int PER>
__global__ void __launch_bounds__(ALIGN_THREADS) moe_align_kernel(const int* __restrict__ topk_ids, const float* __restrict__ topk_w,
                                                                  int n_pairs, int E, int expert_offset, int tile, int* __restrict__ sorted_row,
                                                                  int* __restrict__ inv_pos, float* __restrict__ row_w,
                                                                  int* __restrict__ tile_expert, int* __restrict__ num_tiles, int max_tiles,
                                                                  int* __restrict__ expert_start) {
  __shared__ int cnt[MOE_MAX_E], cursor[MOE_MAX_E], start[MOE_MAX_E + 1];
  __shared__ int warp_tiles[MOE_MAX_E / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int STEP = 8;
  int id[PER > 0 ? PER : STEP];
  [[maybe_unused]] float wt[PER > 0 ? PER : 1];
  if (tid < MOE_MAX_E) cnt[tid] = 0;
  auto load = [&](int i) {
    const int e = i < n_pairs ? __ldg(topk_ids + i) - expert_offset : -1;
    return e >= 0 && e < E ? e : -1;
  };
  if (PER > 0) {
#pragma unroll
    for (int k = 0; k < PER; ++k) id[k] = load(tid + k * ALIGN_THREADS);
#pragma unroll
    for (int k = 0; k < PER; ++k) wt[k] = tid + k * ALIGN_THREADS < n_pairs ? __ldg(topk_w + tid + k * ALIGN_THREADS) : 0.f;
  }
  __syncthreads();
  if (PER > 0) {
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (id[k] >= 0) atomicAdd(&cnt[id[k]], 1);
  } else {
    for (int i0 = tid; i0 < n_pairs; i0 += STEP * ALIGN_THREADS) {
#pragma unroll
      for (int k = 0; k < STEP; ++k) id[k] = load(i0 + k * ALIGN_THREADS);
#pragma unroll
      for (int k = 0; k < STEP; ++k)
        if (id[k] >= 0) atomicAdd(&cnt[id[k]], 1);
    }
  }
  __syncthreads();
  int nt = 0, incl = 0;
  if (tid < MOE_MAX_E) {
    nt = tid < E ? (cnt[tid] + tile - 1) / tile : 0;
    incl = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tiles[warp] = incl;
  }
  __syncthreads();
  if (tid < MOE_MAX_E) {
    int before = 0;
    for (int w = 0; w < warp; ++w) before += warp_tiles[w];
    const int t0 = before + incl - nt;
    start[tid] = cursor[tid] = t0 * tile;
    if (expert_start && tid <= E) expert_start[tid] = t0;
    for (int j = 0; j < nt && t0 + j < max_tiles; ++j) tile_expert[t0 + j] = tid;
    if (tid == MOE_MAX_E - 1) { start[MOE_MAX_E] = (before + incl) * tile; *num_tiles = min(before + incl, max_tiles); if (expert_start && E == MOE_MAX_E) expert_start[E] = before + incl; }
  }
  __syncthreads();
  auto place = [&](int i, int e, float w) {
    if (i >= n_pairs) return;
    if (e < 0) { inv_pos[i] = -1; return; }
    const int p = atomicAdd(&cursor[e], 1);
    sorted_row[p] = i;
    row_w[p] = w;
    inv_pos[i] = p;
  };
  if (PER > 0) {
#pragma unroll
    for (int k = 0; k < PER; ++k) place(tid + k * ALIGN_THREADS, id[k], wt[k]);
  } else {
    for (int i0 = tid; i0 < n_pairs; i0 += STEP * ALIGN_THREADS) {
#pragma unroll
      for (int k = 0; k < STEP; ++k) id[k] = load(i0 + k * ALIGN_THREADS);
#pragma unroll
      for (int k = 0; k < STEP; ++k) place(i0 + k * ALIGN_THREADS, id[k], i0 + k * ALIGN_THREADS < n_pairs ? __ldg(topk_w + i0 + k * ALIGN_THREADS) : 0.f);
    }
  }
  for (int e = warp; e < E; e += ALIGN_THREADS / 32)
    for (int p = start[e] + cnt[e] + lane; p < start[e + 1]; p += 32) { sorted_row[p] = -1; row_w[p] = 0.f; }
}

void moe_align(const int* topk_ids, const float* topk_w, int n_pairs, int E, int expert_offset, int tile, int* sorted_row, int* inv_pos,
               float* row_w, int* tile_expert, int* num_tiles, int max_tiles, cudaStream_t stream, int* expert_start) {
  if (E > MOE_MAX_E) throw std::runtime_error("sglb moe_align: more than 512 local experts");
#define ALIGN(PER) \
  moe_align_kernel<PER><<<1, ALIGN_THREADS, 0, stream>>>(topk_ids, topk_w, n_pairs, E, expert_offset, tile, sorted_row, inv_pos, row_w, tile_expert, \
                                                         num_tiles, max_tiles, expert_start)
  if (n_pairs <= 4 * ALIGN_THREADS) ALIGN(4);
  else if (n_pairs <= 16 * ALIGN_THREADS) ALIGN(16);
  else ALIGN(0);
#undef ALIGN
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------- gather into expert-sorted order
// 64 threads a row, so that no row waits for another's index and few rows still spread over the chip; padding rows cost one load.
template <bool SCALE>
__global__ void __launch_bounds__(256) moe_gather_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ sorted_row,
                                                         const int* __restrict__ num_tiles, __nv_bfloat16* __restrict__ xs, int H,
                                                         int x_stride, int K, int cap_rows, int tile, const float* __restrict__ row_w) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 6), lane = threadIdx.x & 63;
  if (row >= min(cap_rows, __ldg(num_tiles) * tile)) return;
  const int pair = __ldg(sorted_row + row), nvec = H >> 3;
  if (pair < 0) return;
  __nv_bfloat16* dst = xs + (size_t)row * H;
  const __nv_bfloat16* src = x + (size_t)(pair / K) * x_stride;
  [[maybe_unused]] const float w = SCALE ? __ldg(row_w + row) : 1.f;
#pragma unroll 8
  for (int v = lane; v < nvec; v += 64) {
    U4 a = ldg128(src + v * 8);
    if (SCALE)
      a = U4{pack_bf16(bf16_lo(a.x) * w, bf16_hi(a.x) * w), pack_bf16(bf16_lo(a.y) * w, bf16_hi(a.y) * w),
             pack_bf16(bf16_lo(a.z) * w, bf16_hi(a.z) * w), pack_bf16(bf16_lo(a.w) * w, bf16_hi(a.w) * w)};
    st128(dst + v * 8, a);
  }
}

void moe_gather(const void* x, const int* sorted_row, const int* num_tiles, void* xs, int H, int x_stride, int K, int cap_rows,
                int tile, cudaStream_t stream, const float* row_w) {
  if (H % 8) throw std::runtime_error("sglb moe_gather: hidden size must be a multiple of 8");
  const int grid = (cap_rows + 3) / 4;
  if (row_w)
    moe_gather_kernel<true><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, sorted_row, num_tiles, (__nv_bfloat16*)xs, H, x_stride, K, cap_rows, tile, row_w);
  else
    moe_gather_kernel<false><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, sorted_row, num_tiles, (__nv_bfloat16*)xs, H, x_stride, K, cap_rows, tile, nullptr);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------- combine (+ optional NVLink push)
struct MoePush {
  __nv_bfloat16* peer_slot[8];
  uint32_t* peer_flags[8];
  const uint32_t* epoch_ptr;
  uint32_t* done_ctr;
  long long slot_stride;
  int rank, world;
};

// 256 vectors of one token per CTA, all K rows' loads in flight together (K is a template argument; 0: any), sums in the order of k
template <int KT>
__global__ void __launch_bounds__(256) moe_combine_kernel(const __nv_bfloat16* __restrict__ ys, const int* __restrict__ inv_pos,
                                                          const float* __restrict__ pair_w, __nv_bfloat16* __restrict__ out, int H, int K) {
  const int t = blockIdx.x, v = blockIdx.y * 256 + threadIdx.x;
  if (v >= (H >> 3)) return;
  constexpr int G = KT > 0 ? KT : 4;
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int k0 = 0; k0 < (KT > 0 ? KT : K); k0 += G) {
    U4 y[G];
    float w[G];
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int p = KT > 0 || k0 + k < K ? __ldg(inv_pos + t * K + k0 + k) : -1;
      w[k] = p < 0 ? 0.f : pair_w ? __ldg(pair_w + t * K + k0 + k) : 1.f;
      y[k] = p < 0 ? U4{0, 0, 0, 0} : ld128(ys + (size_t)p * H + v * 8);
    }
#pragma unroll
    for (int k = 0; k < G; ++k) {
      a[0] += w[k] * bf16_lo(y[k].x); a[1] += w[k] * bf16_hi(y[k].x); a[2] += w[k] * bf16_lo(y[k].y); a[3] += w[k] * bf16_hi(y[k].y);
      a[4] += w[k] * bf16_lo(y[k].z); a[5] += w[k] * bf16_hi(y[k].z); a[6] += w[k] * bf16_lo(y[k].w); a[7] += w[k] * bf16_hi(y[k].w);
    }
  }
  st128(out + (size_t)t * H + v * 8, U4{pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7])});
}

__global__ void __launch_bounds__(256) moe_combine_push_kernel(const __nv_bfloat16* __restrict__ ys, const int* __restrict__ inv_pos,
                                                               const float* __restrict__ pair_w, int T, int H, int K, const MoePush push) {
  const int nvec = H >> 3;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
      float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int k = 0; k < K; ++k) {
        const int p = __ldg(inv_pos + t * K + k);
        if (p < 0) continue;
        const float w = pair_w ? __ldg(pair_w + t * K + k) : 1.f;
        const U4 y = ld128(ys + (size_t)p * H + v * 8);
        a[0] += w * bf16_lo(y.x); a[1] += w * bf16_hi(y.x); a[2] += w * bf16_lo(y.y); a[3] += w * bf16_hi(y.y);
        a[4] += w * bf16_lo(y.z); a[5] += w * bf16_hi(y.z); a[6] += w * bf16_lo(y.w); a[7] += w * bf16_hi(y.w);
      }
      const U4 o = U4{pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7])};
      const size_t off = (size_t)push.rank * push.slot_stride + (size_t)t * H + v * 8;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < push.world) st128(push.peer_slot[r] + off, o);
    }
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const uint32_t n = atomicAdd(push.done_ctr, 1u);
    if (n == gridDim.x - 1) {
      *push.done_ctr = 0;
      __threadfence_system();
      const uint32_t epoch = *((volatile const uint32_t*)push.epoch_ptr) + 1;
      for (int r = 0; r < push.world; ++r)
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(push.peer_flags[r] + push.rank), "r"(epoch) : "memory");
    }
  }
}

void moe_combine(const void* ys, const int* inv_pos, const float* pair_w, void* out, int T, int H, int K, cudaStream_t stream) {
  if (T <= 0) return;
  const dim3 grid(T, (H / 8 + 255) / 256);
#define COMBINE(KT) moe_combine_kernel<KT><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)ys, inv_pos, pair_w, (__nv_bfloat16*)out, H, K)
  if (K == 1) COMBINE(1);
  else if (K == 2) COMBINE(2);
  else if (K == 4) COMBINE(4);
  else if (K == 8) COMBINE(8);
  else COMBINE(0);
#undef COMBINE
  SGLB_CUDA_CHECK(cudaGetLastError());
}

void moe_combine_push(const void* ys, const int* inv_pos, const float* pair_w, int T, int H, int K, const int64_t* peer_slot_ptrs,
                      const int64_t* peer_flag_ptrs, int rank, int world, const uint32_t* epoch_ptr, uint32_t* done_ctr, int num_sms,
                      cudaStream_t stream) {
  if (T <= 0) return;
  if (world > 8) throw std::runtime_error("sglb moe_combine_push: world size > 8");
  MoePush p{};
  for (int r = 0; r < world; ++r) {
    p.peer_slot[r] = reinterpret_cast<__nv_bfloat16*>(peer_slot_ptrs[r]);
    p.peer_flags[r] = reinterpret_cast<uint32_t*>(peer_flag_ptrs[r]);
  }
  p.epoch_ptr = epoch_ptr; p.done_ctr = done_ctr; p.slot_stride = (long long)T * H; p.rank = rank; p.world = world;
  const int grid = max(1, min(T, num_sms * 4));
  moe_combine_push_kernel<<<grid, 256, 0, stream>>>((const __nv_bfloat16*)ys, inv_pos, pair_w, T, H, K, p);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------- soft-max router with a choice-only correction and identity experts
//   s = softmax(logits) over all E columns; the top_k largest (s + correction) are chosen and weighted by their plain s (not renormalised).
//   Columns >= n_real are identity experts (they return their input): their chosen weights are summed into ident[t] and zeroed in w.
// One warp per token; scores and choice values sit in shared memory; every pick is a warp arg-max (equal values: the lower index).
__global__ void __launch_bounds__(128) moe_softmax_bias_route_kernel(const float* __restrict__ logits, int ld, const float* __restrict__ corr, int T, int E,
                                                                     int K, int n_real, float* __restrict__ w, int* __restrict__ ids,
                                                                     float* __restrict__ ident) {
  extern __shared__ float rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + warp;
  if (t >= T) return;
  float* sc = rsm + (size_t)warp * 2 * E;
  float* ch = sc + E;
  const float* row = logits + (size_t)t * ld;
  float mx = -INFINITY;
  for (int e = lane; e < E; e += 32) mx = fmaxf(mx, row[e]);
  mx = warp_max(mx);
  float sum = 0.f;
  for (int e = lane; e < E; e += 32) {
    const float v = expf(row[e] - mx);
    sc[e] = v;
    sum += v;
  }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
  for (int e = lane; e < E; e += 32) {
    const float v = sc[e] * inv;
    sc[e] = v;
    ch[e] = v + (corr ? corr[e] : 0.f);
  }
  __syncwarp();
  float idw = 0.f;
  for (int k = 0; k < K; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32)
      if (ch[e] > best) { best = ch[e]; bi = e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) {
      const float sv = sc[bi];
      const bool idn = bi >= n_real;
      w[(size_t)t * K + k] = idn ? 0.f : sv;
      ids[(size_t)t * K + k] = bi;
      if (idn) idw += sv;
      ch[bi] = -INFINITY;
    }
    __syncwarp();
  }
  if (lane == 0) ident[t] = idw;
}

void moe_softmax_bias_route(const float* logits, int ld, const float* corr, int T, int E, int K, int n_real, float* w, int* ids, float* ident,
                            cudaStream_t stream) {
  if (T <= 0) return;
  if (E > 1024 || K > E) throw std::runtime_error("sglb moe_softmax_bias_route: at most 1024 router columns, top_k <= columns");
  moe_softmax_bias_route_kernel<<<(T + 3) / 4, 128, sizeof(float) * 8 * E, stream>>>(logits, ld, corr, T, E, K, n_real, w, ids, ident);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------- sigmoid router: the K largest logits win and are weighted sigmoid(logit) (times scale;
// renorm: divided by their sum first).  One warp per token; the choice works on the logits, whose order is that of the scores.
__global__ void __launch_bounds__(128) moe_sigmoid_route_kernel(const float* __restrict__ logits, int ld, int T, int E, int K, int renorm, float scale,
                                                                float* __restrict__ w, int* __restrict__ ids) {
  extern __shared__ float rsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + warp;
  if (t >= T) return;
  float* ch = rsm + (size_t)warp * E;
  const float* row = logits + (size_t)t * ld;
  for (int e = lane; e < E; e += 32) ch[e] = row[e];
  __syncwarp();
  float mine = 0.f, sum = 0.f;                          // lane k keeps pick k (K <= 32)
  int my_id = 0;
  for (int k = 0; k < K; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32)
      if (ch[e] > best || bi == 0x7fffffff) { best = ch[e]; bi = e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (oi != 0x7fffffff && (bi == 0x7fffffff || ob > best || (ob == best && oi < bi))) { best = ob; bi = oi; }
    }
    const float sv = 1.f / (1.f + expf(-best));
    sum += sv;
    if (lane == k) { mine = sv; my_id = bi; }
    if (lane == 0) ch[bi] = -INFINITY;
    __syncwarp();
  }
  if (lane < K) {
    w[(size_t)t * K + lane] = (renorm ? mine / sum : mine) * scale;
    ids[(size_t)t * K + lane] = my_id;
  }
}

void moe_sigmoid_route(const float* logits, int ld, int T, int E, int K, bool renorm, float scale, float* w, int* ids, cudaStream_t stream) {
  if (T <= 0) return;
  if (E > 2048 || K > E || K > 32) throw std::runtime_error("sglb moe_sigmoid_route: at most 2048 experts, top_k <= min(32, experts)");
  moe_sigmoid_route_kernel<<<(T + 3) / 4, 128, sizeof(float) * 4 * E, stream>>>(logits, ld, T, E, K, renorm ? 1 : 0, scale, w, ids);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// y[t] += ident[t] * h[t] + sigmoid(gate[t]) * shared[t]   (identity experts and the always-on expert join the routed experts' sum), fp32 sums
template <typename T> __device__ __forceinline__ float mc_ld(const T* p);
template <> __device__ __forceinline__ float mc_ld<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float mc_ld<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void mc_st(T* p, float v);
template <> __device__ __forceinline__ void mc_st<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void mc_st<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }

template <typename T>
__global__ void __launch_bounds__(256) moe_identity_shared_combine_kernel(T* __restrict__ y, const T* __restrict__ h, const float* __restrict__ ident,
                                                                          const T* __restrict__ shared, const float* __restrict__ gate, int W) {
  const size_t base = (size_t)blockIdx.x * W;
  const float iw = ident ? ident[blockIdx.x] : 0.f;
  const float sg = shared ? (gate ? 1.f / (1.f + expf(-gate[blockIdx.x])) : 1.f) : 0.f;          // no gate: the shared output joins as it is
  for (int c = threadIdx.x; c < W; c += 256) {
    float v = mc_ld<T>(y + base + c);
    if (ident) v += iw * mc_ld<T>(h + base + c);
    if (shared) v += sg * mc_ld<T>(shared + base + c);
    mc_st<T>(y + base + c, v);
  }
}

void moe_identity_shared_combine(void* y, const void* h, const float* ident, const void* shared, const float* gate, bool bf16, int T, int W,
                                 cudaStream_t stream) {
  if (T <= 0) return;
  if (bf16)
    moe_identity_shared_combine_kernel<__nv_bfloat16><<<T, 256, 0, stream>>>((__nv_bfloat16*)y, (const __nv_bfloat16*)h, ident, (const __nv_bfloat16*)shared,
                                                                             gate, W);
  else
    moe_identity_shared_combine_kernel<float><<<T, 256, 0, stream>>>((float*)y, (const float*)h, ident, (const float*)shared, gate, W);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

}  // namespace sglb
