// Mamba-2 recurrence of prompts, 64 tokens a step, on the tensor cores in 32-bit precision.
//
// With P_t = decay 0..t of the chunk's tokens and w_s = (decay s+1..63) dt_s the recurrence over a chunk is four products
//   G = C B^T        Y = P_t (C S) + M X,  M[t,s] = G[t,s] (decay s+1..t) dt_s for s <= t, plus D at s = t        S <- P_63 S + (w B)^T X
// (the decays as products of the tokens' own, never quotients or exponentials of differences, so nothing cancels).
//
// 32-bit precision: every operand is the sum of three bf16 (its rounding, that of what is left, and that of what is left then: 24 bits and more) and a
// product is the six pairs down to 2^-18, the smallest first, into one fp32 accumulator; the pairs left out are below 2^-26.  Sums of 128 such products
// are 1.2e-7 off 64 bits, those of an fp32 product 2.0e-7 (2-norms, normal values; 1.4e-7 and 1.8e-7 for SiLU outputs); with the largest pair first
// the accumulator's truncation costs 1.4e-6.  Most of what is left is a bias, see MC_BIAS.
//
// First kernel: a CTA per (chunk, group of heads) splits B and C once for all heads, in the layout the tensor cores read, forms G and the heads' decays.
// Second kernel: a CTA per (request, 128 columns: a head's, or two heads of 64 with the same B and C) walks the request's chunks.  Transposed, so that
// the columns are the UMMA M dimension and a thread owns one of them:
//   S'^T[col, n] = (w X)^T B      Y1^T[col, t] = S^T C^T      Y2^T[col, t] = X^T M^T
// with S^T and (w X)^T as A operands in TMEM.  Its warps:
//   0..7    state: half of a column's rows (fp32 registers) a thread
//   8..15   inputs: splits of x and w x
//   16..23  outputs: half of a column's tokens a thread
//   24..27  M
//   28, 29  issuer of the products, loader of B, C and the steps (30, 31 only fill the warpgroup)
// Inputs are a chunk ahead; what a chunk waits for are its products (4.8 of its 10 thousand cycles), the state's split before them and its update
// between them.  That chain, about 5.5 us a chunk of the longest request, bounds the kernel.  A role holds what its registers can: a spilled value goes to L2
// (shared memory leaves the L1 cache little), and 150 bytes of them a thread cost a quarter of the time.
// Measured, 64 heads of 64 x 128, 3001 tokens in 5 requests: 588 us eight tokens a step, 143 us here; one request of 1000: 333 and 111; 16 heads of
// 128 x 128, one request of 3000: 982 and 300.  Error of y and of the state against 64 bits, 500 tokens in 12 requests: 1.18e-7 and 5.9e-8 eight tokens
// a step, 9.3e-8 and 1.6e-8 here (the decays' products are formed in 64 bits); one of 1000: 8.9e-8 and 6.9e-9, 8.2e-8 and 3.4e-9.
// Other values, 500 + 130 tokens, mean error against the sum of the terms' magnitudes over that of eight tokens a step: normal 0.5, one sign or alternating signs 0.5, over
// six decades 0.6, cancelling pairs 0.3, one term alone 0.6 (constant decay 0.3 to 0.9).  Only where decay and step are exactly 1, and eight tokens a step round nothing
// but sums, it is larger: 1.3 (N = 64: 1.8) for one sign, 1.8 for equal values, 2.5 for a single moving term, at most 1.3e-7.  Without MC_BIAS all but equal values
// are worse (one sign at a decay of 1: 2.5).
// Not finite: an infinite x, or one above 3.38e38, makes its column NaN from that token to the end (an infinite x is one of both signs in S^T C as soon as C changes sign).
#include "common.cuh"
#include "mamba2.h"
#include "tma_host.h"

namespace sglb {
namespace {

constexpr int MC_L = 64, MC_COLS = 128, MC_THREADS = 1024, MC_SPLIT_THREADS = 256;
constexpr int MC_ORDER = 256;                                 // batches up to this size are taken longest request first
constexpr int MC_BLK = 64 * 128;                              // 64 rows of 64 bf16, 128-byte swizzled
// TMEM columns: S^T split (3 x N / 2), (w X)^T split (3 x 32), the accumulator of S' (N) and then those of Y1 (64) and Y2 (64, two heads: 128)
constexpr int MC_TS = 0, MC_TX = 192, MC_TACC = 320, MC_TY2 = 384;
// The accumulator cuts what it cannot hold, so sums of 32, 64 and 128 products come out small by about these shares (measured on normal values and SiLU
// outputs, whose means are 7.5e-8 and 9.8e-8 for 128, 4.6e-8 and 5.2e-8 for 64).  The factors that a product meets anyway carry them back
constexpr float MC_BIAS_32 = 2.5e-8f, MC_BIAS_64 = 5e-8f, MC_BIAS_128 = 9e-8f;
constexpr int MC_GACC = 4;                                    // accumulators of G, a quarter of K each: the error of its sums goes into all of M
// steps and decays of a head's chunk (bytes MC_STEPS): floats dt, P, w, the decay from a block of 16 tokens' start to t, the decay behind s to its block's end
// times dt_s; the whole decay and those of blocks 1, 1 and 2, 2; the tokens' decays
constexpr int MC_DT = 0, MC_P = 64, MC_W = 128, MC_PIN = 192, MC_WS = 256, MC_ALL = 320, MC_DA = 324 /*floats*/, MC_STEPS = 388 * 4;

template <int N>
struct McCfg {
  static constexpr int HALVES = N / 64;
  static constexpr int IMG = 3 * HALVES * MC_BLK;             // B or C of a chunk: [part][64 states][64 tokens]
  static constexpr int SLOT = 2 * IMG + MC_L * MC_L * 4;      // what the first kernel leaves for a (chunk, group): C, B, G (G as [s / 4][t][4]), steps of its heads
  static constexpr int X = 0, B = X + 6 * MC_BLK, C = B + IMG, M = C + IMG, STEPS = M + 6 * MC_BLK;
  static constexpr int BAD = STEPS + 2 * 2 * MC_STEPS, ORDER = BAD + 4 * MC_COLS * 4, BARS = ORDER + 8 + MC_ORDER * 4;
  static constexpr int SMEM = BARS + 128 + 1024;
  static constexpr int SPLIT_SMEM = 2 * IMG + 1024 + 64;
};

__device__ __forceinline__ void mc_sub(float& a, float& b, uint32_t part) {      // (exact: what is left of a rounding fits)
  asm("{\n\t.reg .b64 v, h, n;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 h, {%2, %3};\n\tmov.b64 n, {%4, %4};\n\tfma.rn.f32x2 v, h, n, v;\n\tmov.b64 {%0, %1}, v;\n\t}"
      : "+f"(a), "+f"(b) : "f"(bf16_lo(part)), "f"(bf16_hi(part)), "f"(-1.f));
}
__device__ __forceinline__ void mc_split(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(a, b);
  mc_sub(a, b, hi);
  mid = pack_bf16(a, b);
  mc_sub(a, b, mid);
  lo = pack_bf16(a, b);
}
__device__ __forceinline__ void mc_split8(const float* v, uint4& a, uint4& m, uint4& l) {
  mc_split(v[0], v[1], a.x, m.x, l.x);
  mc_split(v[2], v[3], a.y, m.y, l.y);
  mc_split(v[4], v[5], a.z, m.z, l.z);
  mc_split(v[6], v[7], a.w, m.w, l.w);
}
// pairs of parts, smallest products first: (2,0) (0,2) (1,1) (1,0) (0,1) (0,0)
__device__ __forceinline__ int mc_part_a(int i) { return (0x001102 >> (4 * i)) & 3; }
__device__ __forceinline__ int mc_part_b(int i) { return (0x010120 >> (4 * i)) & 3; }
template <typename T> __device__ __forceinline__ float mc_ld(const T* p);
template <> __device__ __forceinline__ float mc_ld<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float mc_ld<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void mc_arrive(uint64_t* bar, int lane) {      // this warp's shared-memory and TMEM accesses are done and visible to the products
  fence_proxy_async_smem();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
// a stride whose multiples the compiler works out where they are used, instead of keeping all of them in registers over the whole loop
__device__ __forceinline__ size_t mc_stride(size_t v) {
  asm volatile("" : "+l"(v));
  return v;
}
// z / (1 + exp(-z)) without a branch: quotient by the reciprocal's approximation, and one Newton step by what it leaves (Newton-Raphson on d q = z).
// 1 + exp(-z) is at least 1, and where it would overflow z over the largest number is as good as zero.  From 20 on it is 1: z itself, infinity too (the step would
// take it from itself)
__device__ __forceinline__ float mc_silu(float z) {
  const float d = fminf(1.f + expf(-z), 3e38f), r = rcp_approx(d), q = z * r;
  return z > 20.f ? z : fmaf(fmaf(-d, q, z), r, q);
}
// Chunk c of request b has slot cu_q[b] / 64 + b + c: no two share one, and none lies beyond T / 64 + B.
__device__ __forceinline__ int mc_slot(int q0, int b) { return q0 / MC_L + b; }

template <typename TZ, int N>
__global__ void __launch_bounds__(MC_SPLIT_THREADS) mamba2_split_kernel(const Mamba2Params p, int B, uint8_t* __restrict__ ws, int g0) {
  using Cfg = McCfg<N>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_req;
  __shared__ uint64_t done;
  __shared__ uint32_t tmem_ptr;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = g0 + blockIdx.x, slot = blockIdx.y;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) s_req = -1;
  __syncthreads();
  for (int j = tid; j < B; j += MC_SPLIT_THREADS) {
    const int q = p.cu_q[j], c = slot - mc_slot(q, j);
    if (c >= 0 && c * MC_L < p.cu_q[j + 1] - q) s_req = j;
  }
  __syncthreads();
  const int b = s_req;
  if (b < 0) return;
  if (tid == 0) { mbar_init(&done, 1); fence_barrier_init(); }
  if (warp == 0) { tmem_alloc(&tmem_ptr, MC_GACC * 64); tmem_relinquish(); }
  const int q0 = p.cu_q[b], t0 = (slot - mc_slot(q0, b)) * MC_L, left = p.cu_q[b + 1] - q0 - t0;
  // eight values of a row a thread, four rows in flight; rows beyond the request's end are zeros
  const float* src0 = p.u + (size_t)(q0 + t0) * p.ldu + p.H * p.P + g * N;
#pragma unroll
  for (int i0 = 0; i0 < N / 16; i0 += 4) {
    float v[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int id = (i0 + i) * MC_SPLIT_THREADS + tid, r = id / (N / 8), j = id % (N / 8), t = r & 63;
      const float4* src = reinterpret_cast<const float4*>(src0 + (size_t)t * p.ldu + (r < 64 ? p.G * N : 0) + j * 8);
      const bool ok = t < left;
      *reinterpret_cast<float4*>(v[i]) = ok ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(v[i] + 4) = ok ? __ldg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int id = (i0 + i) * MC_SPLIT_THREADS + tid, r = id / (N / 8), j = id % (N / 8), t = r & 63;
      uint4 a, m, l;
      mc_split8(v[i], a, m, l);
      uint8_t* dst = smem + (r < 64 ? 0 : Cfg::IMG) + (j >> 3) * MC_BLK + t * 128 + (((j & 7) ^ (t & 7)) << 4);
      *reinterpret_cast<uint4*>(dst) = a;
      *reinterpret_cast<uint4*>(dst + Cfg::HALVES * MC_BLK) = m;
      *reinterpret_cast<uint4*>(dst + 2 * Cfg::HALVES * MC_BLK) = l;
    }
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_ptr;
  const int heads = p.H / p.G;
  uint8_t* out = ws + ((size_t)slot * gridDim.x + blockIdx.x) * (Cfg::SLOT + heads * MC_STEPS);
  if (tid == 0) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out), "r"(smem_u32(smem)), "n"(2 * Cfg::IMG) : "memory");
    tma_store_commit();
    // G[t, s]: rows 64.. of the A operand are whatever lies behind C's rows (inside the two images) and give rows that nobody reads
    constexpr uint32_t idesc = make_idesc(UMMA_BF16, UMMA_BF16, 128, 64, 0, 0);
    const uint64_t dc = make_smem_desc_sw128(smem_u32(smem), 0, 1024), db = dc + Cfg::IMG / 16;
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {
      const uint64_t a = dc + mc_part_a(i) * (Cfg::HALVES * MC_BLK / 16), w = db + mc_part_b(i) * (Cfg::HALVES * MC_BLK / 16);
#pragma unroll
      for (int k = 0; k < N / 16; ++k) {
        const uint32_t off = ((k >> 2) * MC_BLK + (k & 3) * 32) / 16;
        umma_f16_ss(tmem + k / (N / 16 / MC_GACC) * 64, a + off, w + off, idesc, i != 0 || k % (N / 16 / MC_GACC) != 0);
      }
    }
    umma_commit(&done);
  }
  __syncwarp();
  // steps and decays, a warp a head, tokens lane and lane + 32: in 64 bits (their products over a chunk are what the old 32-bit chain lost most by)
  for (int h = warp; h < heads; h += MC_SPLIT_THREADS / 32) {
    const int head = g * heads + h;
    double dt[2], da[2], pin[2], suf[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {                             // beyond the end: step 0, decay 1
      const int t = lane + 32 * i;
      const size_t row = q0 + t0 + t;
      dt[i] = 0.;
      da[i] = 1.;
      if (t < left) {
        if (p.gates) {
          const float* gt = p.gates + (row * p.H + head) * p.gstride;
          da[i] = gt[0];
          dt[i] = gt[1];
        } else if (p.decay) {
          da[i] = p.decay[head];
          dt[i] = 1.;
        } else {
          const double x = (double)mc_ld<TZ>(reinterpret_cast<const TZ*>(p.dt_raw) + row * p.lddt + head) + p.dt_bias[head];
          dt[i] = x > 20. ? x : log1p(exp(x));
          da[i] = exp(-exp((double)p.A_log[head]) * dt[i]);
        }
      }
      pin[i] = suf[i] = da[i];
    }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double up = __shfl_up_sync(0xffffffffu, pin[i], o, 16), down = __shfl_down_sync(0xffffffffu, suf[i], o, 16);
        if ((lane & 15) >= o) pin[i] *= up;
        if ((lane & 15) + o < 16) suf[i] *= down;
      }
    }
    double blk[4];                                            // whole decays of the blocks of 16
#pragma unroll
    for (int i = 0; i < 4; ++i) blk[i] = __shfl_sync(0xffffffffu, pin[i >> 1], (i & 1) * 16 + 15);
    float* s = reinterpret_cast<float*>(out + Cfg::SLOT + h * MC_STEPS);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = lane + 32 * i, k = t >> 4;
      double after = __shfl_down_sync(0xffffffffu, suf[i], 1, 16);
      if ((lane & 15) == 15) after = 1.;
      const double before = k == 0 ? 1. : k == 1 ? blk[0] : k == 2 ? blk[0] * blk[1] : blk[0] * blk[1] * blk[2];
      const double behind = k == 3 ? 1. : k == 2 ? blk[3] : k == 1 ? blk[2] * blk[3] : blk[1] * blk[2] * blk[3];
      s[MC_DT + t] = (float)(dt[i] * (1. + MC_BIAS_32));
      s[MC_P + t] = (float)(before * pin[i] * (1. + (N == 128 ? MC_BIAS_128 : MC_BIAS_64)));
      s[MC_W + t] = (float)(after * behind * dt[i] * (1. + MC_BIAS_64));
      s[MC_PIN + t] = (float)pin[i];
      s[MC_WS + t] = (float)(after * dt[i] * (1. + MC_BIAS_32));
      s[MC_DA + t] = (float)da[i];
    }
    if (lane == 0) *reinterpret_cast<float4*>(s + MC_ALL) = make_float4((float)(blk[0] * blk[1] * blk[2] * blk[3]), (float)blk[1], (float)(blk[1] * blk[2]), (float)blk[2]);
  }
  mbar_wait_brief(&done, 0);
  tc_fence_after();
  if ((warp & 3) < 2) {
    const int t = (warp & 3) * 32 + lane, s0 = (warp >> 2) * 32;
    const uint32_t tg = tmem + ((uint32_t)((warp & 3) * 32) << 16) + s0;
    uint4* gp = reinterpret_cast<uint4*>(out + 2 * Cfg::IMG) + (s0 / 4) * MC_L + t;
#pragma unroll 1
    for (int j = 0; j < 32; j += 8) {
      uint32_t r[MC_GACC][8];
#pragma unroll
      for (int k = 0; k < MC_GACC; ++k) tmem_ld_32x32b_x8(tg + k * 64 + j, r[k]);
      tmem_ld_wait();
      uint32_t v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = __float_as_uint((__uint_as_float(r[0][i]) + __uint_as_float(r[1][i])) + (__uint_as_float(r[2][i]) + __uint_as_float(r[3][i])));
      gp[j / 4 * MC_L] = make_uint4(v[0], v[1], v[2], v[3]);
      gp[(j / 4 + 1) * MC_L] = make_uint4(v[4], v[5], v[6], v[7]);
    }
  }
  if (tid == 0) tma_store_wait0();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, MC_GACC * 64);
}

template <typename TZ, int N, bool PAIR>
__global__ void __launch_bounds__(MC_THREADS, 1) mamba2_chunk_kernel(const Mamba2Params p, const uint8_t* __restrict__ ws, int g0, int groups) {
  using Cfg = McCfg<N>;
  constexpr int HALVES = Cfg::HALVES, NT = N / 2, HEADS = PAIR ? 2 : 1;   // state rows of a thread; heads of the CTA
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint8_t* steps = smem + Cfg::STEPS;                   // [chunk parity][head][MC_STEPS]
  int* s_bad = reinterpret_cast<int*>(smem + Cfg::BAD);       // [parity][reader][column]: first token with an x that is not finite, 64 without one
  int* s_req = reinterpret_cast<int*>(smem + Cfg::ORDER);
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(s_req + 1);
  int* s_len = s_req + 2;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::BARS);
  uint64_t *b_full = bars, *c_full = bars + 1, *wx_ready = bars + 2, *xm_ready = bars + 3, *s_read = bars + 4, *y_read = bars + 5;
  uint64_t *s_full = bars + 6, *y2_full = bars + 7, *y1_full = bars + 8, *st_full = bars + 9 /*2*/, *st_empty = bars + 11 /*2*/;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 28 && lane == 0) {
    mbar_init(b_full, 1); mbar_init(c_full, 1);
    mbar_init(wx_ready, 8); mbar_init(xm_ready, 12); mbar_init(s_read, 8); mbar_init(y_read, 8);
    mbar_init(s_full, 1); mbar_init(y2_full, 1); mbar_init(y1_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(st_full + i, 1); mbar_init(st_empty + i, 28); }
    fence_barrier_init();
  }
  // CTAs start in order of their index: the longest request first, so that none is left alone at the end
  const int B = gridDim.y;
  const bool ordered = B > 1 && B <= MC_ORDER;
  if (ordered) {
    if (tid < B) s_len[tid] = p.cu_q[tid + 1] - p.cu_q[tid];
    __syncthreads();
    if (tid < B) {
      const int mine = s_len[tid];
      int rank = 0;
      for (int j = 0; j < B; ++j) rank += s_len[j] > mine || (s_len[j] == mine && j < tid);
      if (rank == (int)blockIdx.y) *s_req = tid;
    }
    __syncthreads();
  }
  const int b = ordered ? *s_req : blockIdx.y;
  const int q0 = p.cu_q[b], n = p.cu_q[b + 1] - q0;
  if (n <= 0) return;
  const int chunks = (n + MC_L - 1) / MC_L;
  if (warp == 0) { tmem_alloc(tmem_ptr, 512); tmem_relinquish(); }
  if (tid < 4 * MC_COLS) s_bad[tid] = MC_L;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;

  const int P = p.P, H = p.H, inner = H * P, col0 = (g0 * (H / p.G) * P / MC_COLS + blockIdx.x) * MC_COLS, head0 = col0 / P, g = head0 / (H / p.G);
  const size_t slot_bytes = Cfg::SLOT + (H / p.G) * MC_STEPS, chunk_bytes = groups * slot_bytes;
  const uint8_t* slot0 = ws + mc_slot(q0, b) * chunk_bytes + (g - g0) * slot_bytes;

  if (warp >= 28) {
    // ------------------------------------------------------------ issuer, loader
    regs_down<32>();
    if (warp == 28) {
      // (all lanes stay together and one is elected: descriptors stay in uniform registers, 34 cycles a 64-wide product instead of 60 by a lane alone)
      constexpr uint32_t id_s = make_idesc(UMMA_BF16, UMMA_BF16, 128, N, 0, 1), id_y1 = make_idesc(UMMA_BF16, UMMA_BF16, 128, 64, 0, 0);
      constexpr uint32_t id_y2 = make_idesc(UMMA_BF16, UMMA_BF16, 128, 64 * HEADS, 1, 0);
      // operand descriptors of part 0, k 0; an offset of o bytes adds o / 16
      const uint64_t d_b = make_smem_desc_sw128(smem_u32(smem + Cfg::B), MC_BLK, 1024), d_x = make_smem_desc_sw128(smem_u32(smem + Cfg::X), MC_BLK, 1024);
      const uint64_t d_c = make_smem_desc_sw128(smem_u32(smem + Cfg::C), 0, 1024), d_m = make_smem_desc_sw128(smem_u32(smem + Cfg::M), 0, 1024);
      const bool one = elect_one();
      for (int c = 0; c < chunks; ++c) {
        const uint32_t par = c & 1;
        mbar_wait_brief(b_full, par);
        mbar_wait_brief(wx_ready, par);
        mbar_wait_brief(y_read, par ^ 1);
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t a = tmem + MC_TX + mc_part_a(i) * 32;
          const uint64_t w = d_b + mc_part_b(i) * (HALVES * MC_BLK / 16);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (one) umma_f16_ts(tmem + MC_TACC, a + k * 8, w + k * (2048 / 16), id_s, (i | k) != 0);
        }
        if (one) umma_commit(s_full);
        mbar_wait_brief(xm_ready, par);
        mbar_wait_brief(s_read, par);
        tc_fence_after();
        // two heads: each with the M of both (columns), of which it needs its own
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint64_t a = d_x + mc_part_a(i) * (2 * MC_BLK / 16), w = d_m + mc_part_b(i) * (HEADS * MC_BLK / 16);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (one) umma_f16_ss(tmem + MC_TY2, a + k * (2048 / 16), w + k * 2, id_y2, (i | k) != 0);
        }
        if (one) umma_commit(y2_full);
        mbar_wait_brief(c_full, par);
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t a = tmem + MC_TS + mc_part_a(i) * (N / 2);
          const uint64_t w = d_c + mc_part_b(i) * (HALVES * MC_BLK / 16);
#pragma unroll
          for (int k = 0; k < N / 16; ++k)
            if (one) umma_f16_ts(tmem + MC_TACC, a + k * 8, w + ((k >> 2) * MC_BLK + (k & 3) * 32) / 16, id_y1, (i | k) != 0);
        }
        if (one) umma_commit(y1_full);
      }
    } else if (warp == 29) {
      // x and z of the chunk after next on their way into L2: their readers wait for one row batch after another
      auto prefetch = [&](int c) {
        for (int t = c * MC_L + lane; t < min(n, (c + 1) * MC_L); t += 32) {
          const char* x = reinterpret_cast<const char*>(p.u + (size_t)(q0 + t) * p.ldu + col0);
#pragma unroll
          for (int i = 0; i < MC_COLS * 4; i += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(x + i));
          if (p.z) {
            const char* z = reinterpret_cast<const char*>(reinterpret_cast<const TZ*>(p.z) + (size_t)(q0 + t) * p.ldz + col0);
#pragma unroll
            for (int i = 0; i < MC_COLS * (int)sizeof(TZ); i += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(z + i));
          }
        }
      };
      prefetch(0);
      prefetch(1);
      asm volatile("griddepcontrol.wait;" ::: "memory");
      for (int c = 0; c < chunks; ++c) {
        const uint8_t* src = slot0 + c * chunk_bytes;
        const int ring = c & 1;
        mbar_wait_brief(st_empty + ring, ((c >> 1) & 1) ^ 1);
        if (lane == 0) {
          mbar_expect_tx(st_full + ring, HEADS * MC_STEPS);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       ::"r"(smem_u32(steps + ring * HEADS * MC_STEPS)), "l"(src + Cfg::SLOT + (head0 - g * (H / p.G)) * MC_STEPS), "n"(HEADS * MC_STEPS),
                       "r"(smem_u32(st_full + ring)) : "memory");
        }
        if (c > 0) mbar_wait_brief(s_full, (c - 1) & 1);
        if (lane == 0) {
          mbar_expect_tx(b_full, Cfg::IMG);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       ::"r"(smem_u32(smem + Cfg::B)), "l"(src + Cfg::IMG), "n"(Cfg::IMG), "r"(smem_u32(b_full)) : "memory");
        }
        prefetch(c + 2);
        if (c > 0) mbar_wait_brief(y1_full, (c - 1) & 1);
        if (lane == 0) {
          mbar_expect_tx(c_full, Cfg::IMG);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                       ::"r"(smem_u32(smem + Cfg::C)), "l"(src), "n"(Cfg::IMG), "r"(smem_u32(c_full)) : "memory");
        }
      }
    }
    __syncwarp();
  } else if (warp >= 24) {
    // ------------------------------------------------------------ M: row mt, blocks of 16 tokens s
    regs_up<80>();
    const int w4 = warp - 24, mt = (w4 & 1) * 32 + lane, mh = PAIR ? w4 >> 1 : 0, mb = mt >> 4;
    const float dskip = p.D ? p.D[head0 + mh] : 0.f;
    const int first = PAIR ? 0 : (w4 >> 1) * 2, last = PAIR ? 3 : first + 1, top = (w4 & 1) * 2 + 1;      // blocks of this thread; the last below the diagonal of its warp
    uint8_t* dst = smem + Cfg::M + mh * MC_BLK + mt * 128;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int c = 0; c < chunks; ++c) {
      const int ring = c & 1;
      const float4* gp = reinterpret_cast<const float4*>(slot0 + c * chunk_bytes + 2 * Cfg::IMG) + mt;
      float next[16];                                         // G of the next block; zeros where all is above the diagonal
      auto fetch = [&](int k) {
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          *reinterpret_cast<float4*>(next + i) = k <= last && k <= top ? __ldg(gp + (4 * k + i / 4) * MC_L) : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      fetch(first);
      mbar_wait_brief(st_full + ring, (c >> 1) & 1);
      const float* sp = reinterpret_cast<const float*>(steps + (ring * HEADS + mh) * MC_STEPS);
      const float pin = sp[MC_PIN + mt];
#pragma unroll 1
      for (int k = first; k <= last; ++k) {
        float r[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = next[i];
        fetch(k + 1);
        if (k < mb) {
          // the decay splits at the blocks' borders
          const float f = pin * (k + 1 == mb ? 1.f : sp[MC_ALL + (mb == 2 ? 1 : k == 0 ? 2 : 3)]);
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 w = *reinterpret_cast<const float4*>(sp + MC_WS + 16 * k + i);
            r[i] *= f * w.x; r[i + 1] *= f * w.y; r[i + 2] *= f * w.z; r[i + 3] *= f * w.w;
          }
        } else if (k == mb) {
          float run = 1.f;                                    // the decay from t down
#pragma unroll
          for (int i = 12; i >= 0; i -= 4) {
            const float4 dt = *reinterpret_cast<const float4*>(sp + MC_DT + 16 * k + i), da = *reinterpret_cast<const float4*>(sp + MC_DA + 16 * k + i);
            const float dts[4] = {dt.x, dt.y, dt.z, dt.w}, das[4] = {da.x, da.y, da.z, da.w};
#pragma unroll
            for (int s = 3; s >= 0; --s) {
              const bool in = 16 * k + i + s <= mt;
              r[i + s] = in ? r[i + s] * (run * dts[s]) + (16 * k + i + s == mt ? dskip : 0.f) : 0.f;
              if (in) run *= das[s];
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = 0.f;
        }
        if (c > 0 && k == first) mbar_wait_brief(y2_full, (c - 1) & 1);      // the last chunk's M has been read
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint4 a, m, l;
          mc_split8(r + 8 * j, a, m, l);
          const int off = ((2 * k + j) ^ (mt & 7)) << 4;
          *reinterpret_cast<uint4*>(dst + off) = a;
          *reinterpret_cast<uint4*>(dst + HEADS * MC_BLK + off) = m;
          *reinterpret_cast<uint4*>(dst + 2 * HEADS * MC_BLK + off) = l;
        }
      }
      mc_arrive(xm_ready, lane);
      if (lane == 0) mbar_arrive(st_empty + ring);
    }
  } else if (warp >= 16) {
    // ------------------------------------------------------------ outputs
    regs_up<72>();
    const int q = warp & 3, hf = (warp - 16) >> 2, pl = q * 32 + lane, hs = PAIR ? q >> 1 : 0, col = col0 + pl;
    const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16) + hf * 32;
    const TZ* zp = reinterpret_cast<const TZ*>(p.z);
    if (zp) zp += (size_t)(q0 + hf * 32) * p.ldz + col;
    float* op = p.out + (size_t)(q0 + hf * 32) * inner + col;
    for (int c = 0; c < chunks; ++c) {
      const int ring = c & 1, left = n - c * MC_L - hf * 32;  // tokens left of this thread's
      const uint32_t par = c & 1;
      float gate[32];                                         // (ready before the products are)
      if (zp) {
        const size_t ld = mc_stride(p.ldz);
#pragma unroll
        for (int i = 0; i < 32; ++i, zp += ld) gate[i] = i < left ? mc_ld<TZ>(zp) : 0.f;
        zp += 32 * ld;
#pragma unroll
        for (int i = 0; i < 32; ++i) gate[i] = mc_silu(gate[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) gate[i] = 1.f;
      }
      mbar_wait_brief(st_full + ring, (c >> 1) & 1);
      const float* sp = reinterpret_cast<const float*>(steps + (ring * HEADS + hs) * MC_STEPS) + MC_P + hf * 32;
      mbar_wait_brief(y2_full, par);
      mbar_wait_brief(y1_full, par);
      tc_fence_after();
      int* bad = s_bad + (ring * 2 + hf) * MC_COLS + pl;
      if (*bad < MC_L) {
        const int first_bad = *bad - hf * 32;
        *bad = MC_L;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i >= first_bad) gate[i] = __int_as_float(0x7fffffff);
      }
#pragma unroll
      for (int i0 = 0; i0 < 32; i0 += 8) {
        uint32_t y1[8], y2[8];
        tmem_ld_32x32b_x8(t_lane + MC_TACC + i0, y1);
        tmem_ld_32x32b_x8(t_lane + MC_TY2 + hs * 64 + i0, y2);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float v = __uint_as_float(y2[i]);
          gate[i0 + i] *= v + fmaf(v, MC_BIAS_64, __uint_as_float(y1[i]) * sp[i0 + i]);
        }
      }
      mc_arrive(y_read, lane);
      const size_t ld = mc_stride(inner);
      if (left >= 32) {
#pragma unroll
        for (int i = 0; i < 32; ++i, op += ld) *op = gate[i];
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i, op += ld)
          if (i < left) *op = gate[i];
      }
      op += 32 * ld;
      if (lane == 0) mbar_arrive(st_empty + ring);
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------ inputs
    regs_down<40>();
    const int w8 = warp - 8, q = w8 & 3, hf = w8 >> 2, pl = q * 32 + lane, hs = PAIR ? q >> 1 : 0;
    const float* xp = p.u + (size_t)(q0 + hf * 32) * p.ldu + col0 + pl;
    const uint32_t t_x = tmem + ((uint32_t)(q * 32) << 16) + MC_TX + hf * 16;
    // the split of x itself goes by eight columns of a token a thread: columns xc.., tokens xt, xt + 16, ...
    const int xt = (tid - 256) >> 4, xc = (tid & 15) * 8;
    const float* xr = p.u + (size_t)(q0 + xt) * p.ldu + col0 + xc;
    for (int c = 0; c < chunks; ++c) {
      const int left = n - c * MC_L, ring = c & 1;
      const uint32_t prev = (c - 1) & 1;
      mbar_wait_brief(st_full + ring, (c >> 1) & 1);
      if (c > 0) mbar_wait_brief(s_full, prev);                       // the last chunk's w X has been read
      tc_fence_after();
      const float* w = reinterpret_cast<const float*>(steps + (ring * HEADS + hs) * MC_STEPS) + MC_W + hf * 32;
#pragma unroll 1
      for (int i0 = 0; i0 < 32; i0 += 8) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = hf * 32 + i0 + i < left ? __ldg(xp + (size_t)i * p.ldu) : 0.f;
        xp += (size_t)8 * p.ldu;
        uint32_t a[4], m[4], l[4];
        const float4 f0 = *reinterpret_cast<const float4*>(w + i0), f1 = *reinterpret_cast<const float4*>(w + i0 + 4);
        mc_split(f0.x * x[0], f0.y * x[1], a[0], m[0], l[0]);
        mc_split(f0.z * x[2], f0.w * x[3], a[1], m[1], l[1]);
        mc_split(f1.x * x[4], f1.y * x[5], a[2], m[2], l[2]);
        mc_split(f1.z * x[6], f1.w * x[7], a[3], m[3], l[3]);
        tmem_st_32x32b_x4(t_x + i0 / 2, a);
        tmem_st_32x32b_x4(t_x + 32 + i0 / 2, m);
        tmem_st_32x32b_x4(t_x + 64 + i0 / 2, l);
      }
      xp += (size_t)(MC_L - 32) * p.ldu;
      tmem_st_wait();
      mc_arrive(wx_ready, lane);
      if (c > 0) mbar_wait_brief(y2_full, prev);                      // the last chunk's X has been read
#pragma unroll 2
      for (int s = xt; s < MC_L; s += 16) {
        float v[8];
        const bool ok = s < left;
        *reinterpret_cast<float4*>(v) = ok ? __ldg(reinterpret_cast<const float4*>(xr)) : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(v + 4) = ok ? __ldg(reinterpret_cast<const float4*>(xr) + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        xr += (size_t)16 * p.ldu;
        // A value that is not finite would reach earlier tokens through the zeros of M: it stays out, and its column's outputs from that token on are
        // made NaN  (1.005: what would round up to a bf16 infinity)
        float zero = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) zero = fmaf(1.005f * v[i], 0.f, zero);
        if (zero != 0.f) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (1.005f * v[i] * 0.f != 0.f) {
              for (int k = 0; k < 2; ++k) atomicMin(s_bad + (ring * 2 + k) * MC_COLS + xc + i, s);
              v[i] = 0.f;
            }
        }
        uint4 a, m, l;
        mc_split8(v, a, m, l);
        uint8_t* dst = smem + Cfg::X + (xc >> 6) * MC_BLK + s * 128 + ((((xc >> 3) & 7) ^ (s & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = a;
        *reinterpret_cast<uint4*>(dst + 2 * MC_BLK) = m;
        *reinterpret_cast<uint4*>(dst + 4 * MC_BLK) = l;
      }
      mc_arrive(xm_ready, lane);
      if (lane == 0) mbar_arrive(st_empty + ring);
    }
  } else {
    // ------------------------------------------------------------ state
    regs_up<88>();
    const int q = warp & 3, hf = warp >> 2, pl = q * 32 + lane, hs = PAIR ? q >> 1 : 0, head = head0 + hs;
    const uint32_t t_lane = tmem + ((uint32_t)(q * 32) << 16);
    float* st = p.state + (((size_t)p.req_slots[b] * H + head) * N + hf * NT) * P + (col0 + pl - head * P);
    float S[NT];
    {
      const bool fresh = p.seq_lens[b] - n == 0;
      const size_t ld = mc_stride(P);
      const float* s = st;
#pragma unroll
      for (int j = 0; j < NT; ++j, s += ld) S[j] = fresh ? 0.f : *s;
    }
    for (int c = 0; c < chunks; ++c) {
      const int ring = c & 1;
      const uint32_t par = c & 1;
      // S^T of before the chunk, split
      if (c > 0) {
        mbar_wait_brief(y1_full, par ^ 1);                            // the last chunk's products have read theirs
        tc_fence_after();
      }
#pragma unroll
      for (int j0 = 0; j0 < NT / 2; j0 += 4) {
        uint32_t a[4], m[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) mc_split(S[2 * (j0 + j)], S[2 * (j0 + j) + 1], a[j], m[j], l[j]);
        const uint32_t t = t_lane + MC_TS + hf * (NT / 2) + j0;
        tmem_st_32x32b_x4(t, a);
        tmem_st_32x32b_x4(t + N / 2, m);
        tmem_st_32x32b_x4(t + N, l);
      }
      tmem_st_wait();
      mbar_wait_brief(st_full + ring, (c >> 1) & 1);
      const float all = reinterpret_cast<const float*>(steps + (ring * HEADS + hs) * MC_STEPS)[MC_ALL];
      mbar_wait_brief(s_full, par);
      tc_fence_after();
#pragma unroll
      for (int j0 = 0; j0 < NT; j0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_lane + MC_TACC + hf * NT + j0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) S[j0 + j] = fmaf(S[j0 + j], all, __uint_as_float(r[j]));
      }
      mc_arrive(s_read, lane);
      if (lane == 0) mbar_arrive(st_empty + ring);
    }
    const size_t ld = mc_stride(P);
#pragma unroll
    for (int j = 0; j < NT; ++j, st += ld) *st = S[j];
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// Groups whose chunks are in the workspace at once: all of them up to 256 MB, which long prompts of many groups go beyond
constexpr size_t MC_WORKSPACE = size_t(256) << 20;
int mc_groups(int slots, int G, size_t slot_bytes) {
  const size_t fit = MC_WORKSPACE / (slots * slot_bytes);
  return fit < 1 ? 1 : fit < (size_t)G ? (int)fit : G;
}

template <typename TZ, int N, bool PAIR>
void launch_mc(const Mamba2Params& p, int B, int T, uint8_t* ws, cudaStream_t stream) {
  using Cfg = McCfg<N>;
  auto split = mamba2_split_kernel<TZ, N>;
  auto kern = mamba2_chunk_kernel<TZ, N, PAIR>;
  SGLB_CUDA_CHECK(cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SPLIT_SMEM));
  SGLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM));
  const int slots = T / MC_L + B, most = mc_groups(slots, p.G, Cfg::SLOT + p.H / p.G * MC_STEPS);
  for (int g0 = 0; g0 < p.G; g0 += most) {
    const int groups = p.G - g0 < most ? p.G - g0 : most;
    split<<<dim3(groups, slots), MC_SPLIT_THREADS, Cfg::SPLIT_SMEM, stream>>>(p, B, ws, g0);
    SGLB_CUDA_CHECK(cudaGetLastError());
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(groups * (p.H / p.G) * p.P / MC_COLS, B); cfg.blockDim = dim3(MC_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM; cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;    // (its warps wait for the first kernel themselves)
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    SGLB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, p, (const uint8_t*)ws, g0, groups));
  }
}

}  // namespace

size_t mamba2_chunk_workspace(const float* u, int ldu, int B, int T, int H, int P, int N, int G) {
  const bool columns = P % MC_COLS == 0 || (P == 64 && (H / G) % 2 == 0);
  if (B <= 0 || (N != 64 && N != 128) || !columns || ldu % 4 || reinterpret_cast<uintptr_t>(u) % 16 || T / MC_L + B > 65535) return 0;
  const size_t slot = (N == 64 ? McCfg<64>::SLOT : McCfg<128>::SLOT) + H / G * MC_STEPS;
  const int slots = T / MC_L + B;
  return slots * mc_groups(slots, G, slot) * slot;
}

void mamba2_chunk_scan(const Mamba2Params& p, bool z_bf16, int B, int T, void* ws, cudaStream_t stream) {
#define SGLB_MC(TZ, N) (p.P == 64 ? launch_mc<TZ, N, true>(p, B, T, (uint8_t*)ws, stream) : launch_mc<TZ, N, false>(p, B, T, (uint8_t*)ws, stream))
  if (z_bf16) p.N == 64 ? SGLB_MC(__nv_bfloat16, 64) : SGLB_MC(__nv_bfloat16, 128);
  else p.N == 64 ? SGLB_MC(float, 64) : SGLB_MC(float, 128);
#undef SGLB_MC
}

}  // namespace sglb
