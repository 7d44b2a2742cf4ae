// Sampling kernels: greedy argmax, temperature + top-k / top-p / min-p sampling, grammar bitmask, penalties.
//
// Reference counterparts: python/sglang/srt/layers/sampler.py:98-320 (softmax + FlashInfer
// top_k_top_p_sampling_from_probs / min_p), kernels/aot/csrc/grammar/apply_token_bitmask_inplace_cuda.cu:157,
// sampling/penaltylib.  Design difference: a single fused kernel produces the token (and its logprob) straight
// from logits and scatters it into the per-request-slot `next_token_buf` the next decode step gathers from,
// so sampled ids never round-trip through the host on the critical path.
#include "common.cuh"
#include "tma_host.h"

namespace sglb {

constexpr int SAMP_THREADS = 1024;
constexpr int SAMP_BINS = 2048;

__device__ __forceinline__ float block_reduce_max(float v, float* red) {
  v = warp_max(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : -INFINITY;
  r = warp_max(r);
  r = __shfl_sync(0xffffffffu, r, 0);
  // broadcast from warp 0 to everyone
  __syncthreads();
  if (threadIdx.x == 0) red[0] = r;
  __syncthreads();
  return red[0];
}

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// counter-based RNG (splitmix64 finaliser over (seed, row, step)) -> uniform in [0,1)
__device__ __forceinline__ float rng_uniform(unsigned long long seed, unsigned long long a, unsigned long long b) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (a + 1) + 0xD1B54A32D192ED03ull * (b + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return (float)(z >> 40) * (1.0f / 16777216.0f);
}

struct SampleParams {
  const float* temperature;   // [B]
  const int* top_k;           // [B]  (1 => greedy)
  const float* top_p;         // [B]
  const float* min_p;         // [B]
  const long long* seeds;     // [B, 2] (per-request seed, per-request output position) or null; position < 0 -> this row uses the global stream
  const int* out_slots;       // [B] scatter index into next_token_buf (or null)
  int* next_token_buf;        // [max_reqs+1]
  int* out_tokens;            // [B]
  float* out_logprobs;        // [B] or null
  unsigned long long global_seed;
  const long long* step_ptr;  // device counter (graph-replay safe) or null
  long long step;
  int V, stride;
};

// ---------------------------------------------------------------- the sampler: a cluster of eight CTAs per row
// Eight CTAs take an eighth of a row each (the batch's logits stay in L2 between passes) and exchange block results (maximum, sums, histogram segments)
// through distributed shared memory.  A lane always takes 8 consecutive logits, a warp a contiguous range, so that index order survives everywhere.
//
// top-k / top-p: two-level histogram over d = (max - logit) / T (r = p / p_max = e^-d): 2048 bins of width 1/64 cover r down to e^-32, a second
// 2048 bins refine the one that holds the boundary (7.6e-6 in d).  Shared-memory atomics are native for integers only (a float add is a
// compare-and-swap loop that collapses on the popular bins of a broad tail), so both levels count integers: elements, or r over the bin's largest r
// in fixed point.  The fixed-point mass only nominates a bin; the masses before and inside it are then summed in fp32 and the nomination is moved,
// to its neighbour and then by halves, until they enclose the target.  Elements beyond d = 32 (masked ones, cold temperatures) meet in the last bin and are added up in registers.
//
// What can be kept is usually a handful of candidates: the threads' own maxima (2048 of them) bound the boundary from below, one pass collects
// what lies above that bound, and the first CTA alone finishes the row on that list without further cluster barriers.  A row whose list would not fit
// (a broad nucleus, a large k) goes through the same steps on the whole row with all eight.
//
// Bound by the two passes over the row and a chain of about eight cluster barriers.  Measured (B200, bf16, rows asking in turn for greedy / nucleus /
// top-k / min-p / plain): 121 x 128256 in 38 us, 256 in 62, one greedy row in 11; one CTA per row with scalar loads and float atomics took 2594 for
// the 121, the cluster without candidate lists 69.
constexpr int SAMP_CL = 8;              // CTAs per row: a portable cluster
constexpr int SAMP_SEG = SAMP_BINS / SAMP_CL;
// One width for every batch, so that a row's sums, and with them a seeded request's token, do not follow how many rows there are.  256 threads, several
// CTAs an SM, against 1024, one: 16 and 21 us against 21 and 23 for 8 rows of 32000 and 128256, 23 against 33 for 32 of 128256, 11 either way for one
constexpr int SAMP_NT = 256;

__device__ __forceinline__ uint32_t cl_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// the two halves of a first barrier: a CTA's shared memory may be written by its peers only once it has started, and this is what tells them so
__device__ __forceinline__ void cl_started() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_all_started() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_map(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cl_st(const void* p, uint32_t rank, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_map(p, rank)), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t cl_ld(const void* p, uint32_t rank) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cl_map(p, rank)) : "memory");
  return v;
}

constexpr int SAMP_LIST = 1024;         // candidates the first CTA takes on alone

template <int NW>
struct SampShared {
  uint32_t slot[2][2][SAMP_CL];         // [parity][value][rank]: block results of a reduction
  uint32_t wred[2][NW];
  uint32_t hist[SAMP_BINS];
  float seg_total[SAMP_CL], scan[NW];
  int hit;
  uint32_t cand_bin[SAMP_CL], cand_before[SAMP_CL];
  uint32_t kept[SAMP_CL * NW];          // kept mass of every warp of the row; before that, its candidates
  int pick;
  float pick_run, pick_u;
  float own_d[SAMP_LIST], all_d[SAMP_LIST];      // candidates: of this CTA (an equal part per warp), of the row (first CTA)
  int own_i[SAMP_LIST], all_i[SAMP_LIST];
};

__device__ __forceinline__ void samp_load8(const __nv_bfloat16* p, float (&v)[8]) {
  const U4 a = ld128(p);
  v[0] = bf16_lo(a.x); v[1] = bf16_hi(a.x); v[2] = bf16_lo(a.y); v[3] = bf16_hi(a.y);
  v[4] = bf16_lo(a.z); v[5] = bf16_hi(a.z); v[6] = bf16_lo(a.w); v[7] = bf16_hi(a.w);
}
__device__ __forceinline__ void samp_load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <typename T>
__global__ void __cluster_dims__(SAMP_CL, 1, 1) __launch_bounds__(SAMP_NT, 6)
sample_kernel(const T* __restrict__ logits, SampleParams p, int per_warp) {
  constexpr int NT = SAMP_NT, NW = NT / 32, WCAP = SAMP_LIST / NW;
  __shared__ SampShared<NW> sh;
  cl_started();
  const int rank = (int)cl_rank(), row = blockIdx.x / SAMP_CL;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int V = p.V;
  const T* lr = logits + (size_t)row * p.stride;
  const int w0 = (rank * NW + warp) * per_warp, w1 = min(w0 + per_warp, V);      // this warp's contiguous range
  const bool vec = (reinterpret_cast<uintptr_t>(lr) & 15) == 0;

  auto get8 = [&](int i, float (&v)[8]) {                              // 8 logits from i; those beyond the row are NaN (every comparison fails)
    if (vec && i + 8 <= V) { samp_load8(lr + i, v); return; }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = i + j < V ? to_f<T>(lr[i + j]) : __int_as_float(0x7fffffff);
  };
  int par = 0;
  auto reduce2 = [&](float& a, float& b) {                             // sums over the row, the same bits in every thread
    a = warp_sum(a); b = warp_sum(b);
    if (lane == 0) { sh.wred[0][warp] = __float_as_uint(a); sh.wred[1][warp] = __float_as_uint(b); }
    __syncthreads();
    if (warp == 0) {
      a = warp_sum(lane < NW ? __uint_as_float(sh.wred[0][lane]) : 0.f);
      b = warp_sum(lane < NW ? __uint_as_float(sh.wred[1][lane]) : 0.f);
      if (lane < SAMP_CL) { cl_st(&sh.slot[par][0][rank], lane, __float_as_uint(a)); cl_st(&sh.slot[par][1][rank], lane, __float_as_uint(b)); }
    }
    cl_sync();
    a = b = 0.f;
#pragma unroll
    for (int r = 0; r < SAMP_CL; ++r) { a += __uint_as_float(sh.slot[par][0][r]); b += __uint_as_float(sh.slot[par][1][r]); }
    par ^= 1;                                                          // (the next writers of this half have passed the next barrier)
  };

  const float inv_t = 1.f / fmaxf(p.temperature[row], 1e-6f);
  const int topk = p.top_k[row];
  const bool greedy = topk == 1;
  const float top_p = p.top_p[row], min_p = p.min_p[row];
  const bool need_k = topk > 0 && topk < V, need_p = top_p < 1.f;
  const bool need_z = p.out_logprobs || (!greedy && need_p && !need_k);

  // ---- first pass: maximum, its lowest index (torch.argmax), and the partition sum over a running maximum
  float mx = -INFINITY, z = 0.f;
  int am = 0x7fffffff;
#pragma unroll 2
  for (int i = w0 + lane * 8; i < w1; i += 256) {
    float v[8];
    get8(i, v);
    const float before = mx;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (v[j] > mx) { mx = v[j]; am = i + j; }
    if (need_z && mx > -INFINITY) {
      if (mx > before) z *= __expf((before - mx) * inv_t);
      if (i + 8 <= V) {
#pragma unroll
        for (int j = 0; j < 8; ++j) z += __expf((v[j] - mx) * inv_t);
      } else {
        for (int j = 0; i + j < V; ++j) z += __expf((to_f<T>(lr[i + j]) - mx) * inv_t);
      }
    }
  }
  const float own_max = mx;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, mx, o);
    const int oi = __shfl_xor_sync(0xffffffffu, am, o);
    if (ov > mx || (ov == mx && oi < am)) { mx = ov; am = oi; }
  }
  if (lane == 0) { sh.wred[0][warp] = __float_as_uint(mx); sh.wred[1][warp] = (uint32_t)am; }
  __syncthreads();
  cl_all_started();                                                    // (long past by now: the pass over the row lies between)
  if (warp == 0) {
    mx = lane < NW ? __uint_as_float(sh.wred[0][lane]) : -INFINITY;
    am = lane < NW ? (int)sh.wred[1][lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, mx, o);
      const int oi = __shfl_xor_sync(0xffffffffu, am, o);
      if (ov > mx || (ov == mx && oi < am)) { mx = ov; am = oi; }
    }
    if (lane < SAMP_CL) { cl_st(&sh.slot[par][0][rank], lane, __float_as_uint(mx)); cl_st(&sh.slot[par][1][rank], lane, (uint32_t)am); }
  }
  cl_sync();
  float gmax = -INFINITY;
  int arg = 0x7fffffff;
#pragma unroll
  for (int r = 0; r < SAMP_CL; ++r) {                                  // ranks in index order: a strict comparison keeps the lowest index
    const float ov = __uint_as_float(sh.slot[par][0][r]);
    if (ov > gmax) { gmax = ov; arg = (int)sh.slot[par][1][r]; }
  }
  if (arg == 0x7fffffff) arg = 0;                                      // a row without a finite logit
  par ^= 1;
  float Z = 0.f;
  if (need_z) {
    float unused = 0.f;
    Z = own_max > -INFINITY ? z * __expf((own_max - gmax) * inv_t) : z;
    reduce2(Z, unused);
  }
  auto finish = [&](int token) {
    p.out_tokens[row] = token;
    if (p.next_token_buf && p.out_slots) p.next_token_buf[p.out_slots[row]] = token;
    if (p.out_logprobs) p.out_logprobs[row] = (to_f<T>(lr[token]) - gmax) * inv_t - __logf(Z);
  };
  if (greedy) {
    if (rank == 0 && tid == 0) finish(arg);
    return;                            // (nobody reads this CTA's shared memory after the barrier above)
  }
  // a seeded request draws from (its seed, ITS OWN output position): the stream does not depend on which step / row / batch it landed in
  const bool own_seed = p.seeds && p.seeds[2 * row + 1] >= 0;
  const long long step = p.step_ptr ? *p.step_ptr : p.step;
  const float u01 = own_seed ? rng_uniform((unsigned long long)p.seeds[2 * row], 0ull, (unsigned long long)p.seeds[2 * row + 1])
                             : rng_uniform(p.global_seed, (unsigned long long)row, (unsigned long long)step);

  // f(d) over this thread's logits
  auto each = [&](auto&& f) {
#pragma unroll 2
    for (int i = w0 + lane * 8; i < w1; i += 256) {
      float v[8];
      get8(i, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) f((gmax - v[j]) * inv_t);
    }
  };
  constexpr float W1 = 1.f / 64.f;
  const float scale = fminf(16384.f, floorf(4294967040.f / (float)V)), inv_scale = 1.f / scale;      // whole: V logits of a bin's largest r fit 32 bits
  auto bin1 = [](float d) { return min(SAMP_BINS - 1, (int)(d * (1.f / W1))); };
  auto fixed_mass = [&](float d, int b) { return (uint32_t)(__expf(b * W1 - d) * scale + 0.5f); };
  const auto count = [](int, uint32_t s) { return (float)s; };
  const auto mass = [&](int bin, uint32_t s) { return (float)s * inv_scale * __expf(-bin * W1); };
  auto clear = [&]() {
    for (int i = tid; i < SAMP_BINS; i += NT) sh.hist[i] = 0;
    __syncthreads();
  };
  auto flush_last = [&](uint32_t last) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) last += __shfl_xor_sync(0xffffffffu, last, o);
    if (lane == 0 && last) atomicAdd(&sh.hist[SAMP_BINS - 1], last);
  };
  // first bin whose inclusive prefix reaches the target (SAMP_BINS: none does) and the exclusive prefix before it.  value(bin, sum) weighs a bin.
  // The row's histogram is the sum of the CTAs'; each scans a segment of it
  auto find_row = [&](float target, float& before, auto&& value) -> int {
    if (tid == 0) sh.hit = SAMP_BINS;
    cl_sync();                                                         // every CTA's histogram is complete
    float li = 0.f;
    const int bin = rank * SAMP_SEG + tid;
    if (tid < SAMP_SEG) {
      uint32_t s = 0;
#pragma unroll
      for (int r = 0; r < SAMP_CL; ++r) s += cl_ld(&sh.hist[bin], r);
      li = value(bin, s);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, li, o);
        if (lane >= o) li += t;
      }
      if (lane == 31) sh.scan[warp] = li;
    }
    __syncthreads();
    float base = 0.f, total = 0.f;
#pragma unroll
    for (int w = 0; w < SAMP_SEG / 32; ++w) {
      if (w == warp) base = total;
      total += sh.scan[w];
    }
    if (tid < SAMP_CL) cl_st(&sh.seg_total[rank], tid, __float_as_uint(total));
    cl_sync();
    float seg = 0.f;
    for (int r = 0; r < rank; ++r) seg += sh.seg_total[r];
    float excl = 0.f;
    if (tid < SAMP_SEG) {
      const float prev = __shfl_up_sync(0xffffffffu, li, 1);
      excl = seg + (base + (lane ? prev : 0.f));
      if (seg + (base + li) >= target && (excl < target || bin == 0)) atomicMin(&sh.hit, bin);
    }
    __syncthreads();
    const int hit = sh.hit;
    if (hit == SAMP_BINS) {
      if (tid < SAMP_CL) cl_st(&sh.cand_bin[rank], tid, SAMP_BINS);
    } else if (bin == hit && tid < SAMP_SEG) {
      for (int r = 0; r < SAMP_CL; ++r) { cl_st(&sh.cand_before[rank], r, __float_as_uint(excl)); cl_st(&sh.cand_bin[rank], r, (uint32_t)hit); }
    }
    cl_sync();
    int found = SAMP_BINS;
#pragma unroll
    for (int r = SAMP_CL - 1; r >= 0; --r)
      if (sh.cand_bin[r] < SAMP_BINS) { found = (int)sh.cand_bin[r]; before = __uint_as_float(sh.cand_before[r]); }
    return found;
  };
  // the same inside one CTA (BPT consecutive bins a thread)
  auto find_list = [&](float target, float& before, auto&& value) -> int {
    constexpr int BPT = SAMP_BINS / NT;
    if (tid == 0) sh.hit = SAMP_BINS;
    __syncthreads();                                                   // the histogram is complete
    float v[BPT], own = 0.f;
#pragma unroll
    for (int k = 0; k < BPT; ++k) { v[k] = value(tid * BPT + k, sh.hist[tid * BPT + k]); own += v[k]; }
    float li = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, li, o);
      if (lane >= o) li += t;
    }
    if (lane == 31) sh.scan[warp] = li;
    __syncthreads();
    float base = 0.f;
    for (int w = 0; w < warp; ++w) base += sh.scan[w];
    const float prev = __shfl_up_sync(0xffffffffu, li, 1);
    float run = base + (lane ? prev : 0.f);
    const bool mine = base + li >= target && (run < target || tid == 0);
    if (mine) atomicMin(&sh.hit, tid);
    __syncthreads();
    const int hit = sh.hit;
    if (hit == SAMP_BINS) return SAMP_BINS;
    if (tid == hit) {
      int b = BPT - 1;
      for (int k = 0; k < BPT; ++k) {
        if (run + v[k] >= target) { b = k; break; }
        if (k < BPT - 1) run += v[k];
      }
      sh.cand_bin[0] = tid * BPT + b;
      sh.cand_before[0] = __float_as_uint(run);
    }
    __syncthreads();
    before = __uint_as_float(sh.cand_before[0]);
    return (int)sh.cand_bin[0];
  };
  // d_max of the kept set { d <= d_max }, given that it lies within { d <= lim }; every thread gets the same.  Over the row or over the list
  auto solve = [&](float lim, auto&& over, auto&& find, auto&& sums) -> float {
    float d_max = INFINITY;
    // refine bin b1: the smallest d edge whose kept count / mass reaches ``target``, given what lies before the bin
    auto refine = [&](int b1, float target, auto&& weigh) -> float {
      const float lo = b1 * W1, far = b1 == SAMP_BINS - 1 ? d_max : fminf(d_max, lo + W1);
      clear();
      uint32_t last = 0;
      over([&](float d) {
        if (d >= lo && d <= far && bin1(d) == b1) {
          const int b = min(SAMP_BINS - 1, (int)((d - lo) * (SAMP_BINS / W1)));
          if (b == SAMP_BINS - 1) ++last;
          else atomicAdd(&sh.hist[b], 1u);
        }
      });
      flush_last(last);
      float before = 0.f;
      const int b2 = find(target, before, weigh);
      if (b1 == SAMP_BINS - 1 && b2 >= SAMP_BINS - 1) return INFINITY;
      return lo + (float)(min(b2, SAMP_BINS - 1) + 1) * (W1 / SAMP_BINS);
    };
    float base_mass = Z;
    if (need_k) {
      clear();
      uint32_t last = 0;
      over([&](float d) {
        if (d >= 0.f && d <= lim) {
          const int b = bin1(d);
          if (b == SAMP_BINS - 1) ++last;
          else atomicAdd(&sh.hist[b], 1u);
        }
      });
      flush_last(last);
      float before = 0.f;
      const int b1 = find((float)topk, before, count);
      if (b1 < SAMP_BINS) d_max = refine(b1, (float)topk - before, count);
      if (need_p) {
        float m = 0.f, unused = 0.f;
        const float edge = d_max;
        over([&](float d) { if (d >= 0.f && d <= edge) m += __expf(-d); });
        sums(m, unused);
        base_mass = m;
      }
    }
    if (need_p) {
      const float target = top_p * base_mass;
      const float dm = d_max, reach = fminf(dm, lim);
      clear();
      uint32_t last = 0;
      over([&](float d) {
        if (d >= 0.f && d <= reach) {
          const int b = bin1(d);
          const uint32_t q = fixed_mass(d, b);
          if (b == SAMP_BINS - 1) last += q;
          else atomicAdd(&sh.hist[b], q);
        }
      });
      flush_last(last);
      float before = 0.f;
      int b1 = min(find(target, before, mass), SAMP_BINS - 1);
      float m_before, m_in;
      int first = 0, last_bin = SAMP_BINS - 1;                         // where the bin can be: the nominated one, its neighbour, then by halves
      bool nominated = true;
      while (true) {                                                   // (the same numbers in every thread)
        m_before = m_in = 0.f;
        const int b = b1;
        const float far = b == SAMP_BINS - 1 ? dm : fminf(dm, (b + 1) * W1);
        over([&](float d) {
          if (d >= 0.f && d <= far) {
            const int k = bin1(d);
            if (k <= b) {
              const float r = __expf(-d);
              if (k < b) m_before += r;
              else m_in += r;
            }
          }
        });
        sums(m_before, m_in);
        if (m_before >= target && b1 > first) {
          last_bin = b1 - 1;
          b1 = nominated ? last_bin : (first + last_bin) >> 1;
        } else if (m_before + m_in < target && b1 < last_bin) {
          first = b1 + 1;
          b1 = nominated ? first : (first + last_bin) >> 1;
        } else {
          break;
        }
        nominated = false;
      }
      if (last_bin < SAMP_BINS - 1 || m_before + m_in >= target)       // (else rounding holds the whole row below the target)
        d_max = fminf(d_max, refine(b1, target - m_before, [&](int b, uint32_t s) { return (float)s * __expf(-(b1 * W1 + (b + 0.5f) * (W1 / SAMP_BINS))); }));
    }
    return d_max;
  };
  // keep { r >= thr }, r = p / p_max; beyond d_far no r can reach thr, which saves the exponential
  auto threshold = [&](float d_max) { return d_max < INFINITY ? fmaxf(min_p, __expf(-d_max)) : min_p; };
  auto beyond = [](float thr) { return thr > 0.f ? -__logf(thr) + 0.01f : INFINITY; };

  float d_max = INFINITY;
  if (need_k || need_p) {
    // ---- a bound on the boundary: the k-th largest of the threads' own maxima, or the point where their mass alone reaches the nucleus; else what lies
    // so low (r below (1 - p) / V of the mass, halved for rounding) that all of it together cannot reach the mass that is cut off
    float lim = INFINITY;
    const float od = (gmax - own_max) * inv_t;
    if (need_k ? topk <= SAMP_CL * NT / 2 : true) {
      clear();
      if (od >= 0.f) {
        const int b = bin1(od);
        atomicAdd(&sh.hist[b], need_k ? 1u : fixed_mass(od, b));
      }
      float unused = 0.f;
      const int b = need_k ? find_row((float)topk, unused, count) : find_row(top_p * Z * 1.0002f, unused, mass);
      if (b < SAMP_BINS - 1) lim = (b + 1) * W1;
    }
    if (!need_k) {
      const float tail = 0.5f * (1.f - top_p) * Z / (float)V;
      if (tail > 0.f) lim = fminf(lim, -__logf(tail));
    }
    // ---- second pass: candidates { d <= lim } in index order, an equal part of the list per warp
    int mine = 0;
    for (int i0 = w0; i0 < w1; i0 += 256) {
      const int i = i0 + lane * 8;
      float d[8];
      unsigned bits = 0;
      if (i < w1) {
        get8(i, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          d[j] = (gmax - d[j]) * inv_t;
          if (d[j] >= 0.f && d[j] <= lim) bits |= 1u << j;
        }
      }
      if (!__any_sync(0xffffffffu, bits)) continue;
      int at = __popc(bits);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += t;
      }
      const int end = mine + __shfl_sync(0xffffffffu, at, 31);
      at += mine - __popc(bits);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (bits >> j & 1) {
          if (at < WCAP) { sh.own_d[warp * WCAP + at] = d[j]; sh.own_i[warp * WCAP + at] = i + j; }
          ++at;
        }
      mine = end;
      if (mine > WCAP) break;
    }
    if (lane < SAMP_CL) cl_st(&sh.kept[rank * NW + warp], lane, (uint32_t)(mine > WCAP ? SAMP_LIST + 1 : mine));
    cl_sync();
    int first = 0, total = 0;                                          // this warp's place in the row's list
    for (int k = lane; k < SAMP_CL * NW; k += 32) {
      const int c = min((int)sh.kept[k], SAMP_LIST + 1);
      total += c;
      if (k < rank * NW + warp) first += c;
    }
    first = warp_sum(first);
    total = warp_sum(total);
    if (total <= SAMP_LIST) {
      __syncwarp();
      for (int k = lane; k < mine; k += 32) {
        cl_st(&sh.all_d[first + k], 0, __float_as_uint(sh.own_d[warp * WCAP + k]));
        cl_st(&sh.all_i[first + k], 0, (uint32_t)sh.own_i[warp * WCAP + k]);
      }
      cl_sync();
      if (rank != 0) return;
      auto over = [&](auto&& f) {
        for (int k = tid; k < total; k += NT) f(sh.all_d[k]);
      };
      auto sums = [&](float& a, float& b) {
        a = warp_sum(a); b = warp_sum(b);
        __syncthreads();
        if (lane == 0) { sh.wred[0][warp] = __float_as_uint(a); sh.wred[1][warp] = __float_as_uint(b); }
        __syncthreads();
        a = b = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) { a += __uint_as_float(sh.wred[0][w]); b += __uint_as_float(sh.wred[1][w]); }
      };
      const float thr = threshold(solve(lim, over, find_list, sums));
      // an equal run of the list per thread, scanned in order
      constexpr int PER = SAMP_LIST / NT;
      float r[PER], own = 0.f;
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int e = tid * PER + k;
        const float v = e < total ? __expf(-sh.all_d[e]) : -1.f;
        r[k] = v >= thr && e < total ? v : 0.f;
        own += r[k];
      }
      float li = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, li, o);
        if (lane >= o) li += t;
      }
      __syncthreads();
      if (lane == 31) sh.scan[warp] = li;
      if (tid == 0) sh.hit = NT;
      __syncthreads();
      float base = 0.f, sum = 0.f;
      for (int w = 0; w < NW; ++w) {
        if (w == warp) base = sum;
        sum += sh.scan[w];
      }
      const float u = u01 * sum;
      const float prev = __shfl_up_sync(0xffffffffu, li, 1);
      if (own > 0.f && base + li > u) atomicMin(&sh.hit, tid);
      __syncthreads();
      int hit = sh.hit;
      if (hit == NT) {                                                 // rounding at the very end: the last kept candidate (or none: the maximum)
        __syncthreads();
        if (tid == 0) sh.hit = -1;
        __syncthreads();
        if (own > 0.f) atomicMax(&sh.hit, tid);
        __syncthreads();
        hit = sh.hit;
      }
      if (hit < 0) {
        if (tid == 0) finish(arg);
      } else if (tid == hit) {
        float run = base + (lane ? prev : 0.f);
        int e = -1;
#pragma unroll
        for (int k = 0; k < PER; ++k)
          if (r[k] > 0.f && (e < 0 || !(run > u))) { e = tid * PER + k; run += r[k]; }
        finish(sh.all_i[e]);
      }
      return;
    }
    d_max = solve(lim, each, find_row, reduce2);
  }
  const float thr = threshold(d_max), d_far = beyond(thr);

  // ---- whole row: kept mass of every warp (index order), the warp that holds the drawn point, then the token inside it
  float cm = 0.f;
  each([&](float d) {
    if (d <= d_far) {
      const float r = __expf(-d);
      if (r >= thr) cm += r;
    }
  });
  cm = warp_sum(cm);
  if (need_k || need_p) cl_sync();                                     // (the candidate counts in ``kept`` have been read)
  if (lane < SAMP_CL) cl_st(&sh.kept[rank * NW + warp], lane, __float_as_uint(cm));
  cl_sync();
  if (warp == 0) {
    constexpr int PER = SAMP_CL * NW / 32;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < PER; ++k) s += __uint_as_float(sh.kept[lane * PER + k]);
    float incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const float total = __shfl_sync(0xffffffffu, incl, 31);
    float u = u01 * total;
    const float up = __shfl_up_sync(0xffffffffu, incl, 1);
    unsigned who = __ballot_sync(0xffffffffu, incl > u && s > 0.f);
    if (who == 0) {                                                    // rounding at the very end: the last kept logit
      who = __ballot_sync(0xffffffffu, s > 0.f);
      who = who ? 1u << (31 - __clz(who)) : 0u;
      u = INFINITY;
    }
    if (who == 0) {
      if (lane == 0) sh.pick = -1;
    } else if (lane == __ffs(who) - 1) {
      float run = lane ? up : 0.f;
      int pick = -1;
      float pick_run = run;
      for (int k = 0; k < PER; ++k) {
        const float m = __uint_as_float(sh.kept[lane * PER + k]);
        if (m <= 0.f) continue;
        pick = lane * PER + k;
        pick_run = run;
        run += m;
        if (run > u) break;
      }
      sh.pick = pick; sh.pick_run = pick_run; sh.pick_u = u;
    }
  }
  __syncthreads();
  const int pick = sh.pick;
  if (pick < 0) {
    if (rank == 0 && tid == 0) finish(arg);
    return;
  }
  if (pick != rank * NW + warp) return;
  float run = sh.pick_run;
  const float u = sh.pick_u;
  int token = arg;
  for (int i0 = w0; i0 < w1; i0 += 256) {
    const int i = i0 + lane * 8;
    float v[8], r[8], s = 0.f;
    int mine = -1;                                                     // last kept logit of this lane
    if (i < w1) get8(i, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float e = i < w1 ? __expf((v[j] - gmax) * inv_t) : 0.f;
      const bool keep = i < w1 && e >= thr && e > 0.f;                 // (a masked logit has no mass, and what rounding leaves over is not its own)
      r[j] = keep ? e : 0.f;
      s += r[j];
      if (keep) mine = i + j;
    }
    float incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const float up = __shfl_up_sync(0xffffffffu, incl, 1);
    const unsigned who = __ballot_sync(0xffffffffu, run + incl > u && s > 0.f);
    if (who) {
      if (lane == __ffs(who) - 1) {
        float c = run + (lane ? up : 0.f);
        int tok = mine;
#pragma unroll
        for (int j = 7; j >= 0; --j) {                                 // the first kept logit whose running mass passes u (from the back: the lowest stays)
          float upto = c;
          for (int k = 0; k <= j; ++k) upto += r[k];
          if (r[j] > 0.f && upto > u) tok = i + j;
        }
        finish(tok);
      }
      return;
    }
    const int far = __reduce_max_sync(0xffffffffu, mine);
    if (far >= 0) token = far;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) finish(token);
}

template <typename T>
static void launch_sample(const void* logits, const SampleParams& p, int B, cudaStream_t stream) {
  constexpr int NW = SAMP_NT / 32;
  const int per_warp = ((p.V + SAMP_CL * NW - 1) / (SAMP_CL * NW) + 255) / 256 * 256;
  sample_kernel<T><<<B * SAMP_CL, SAMP_NT, 0, stream>>>((const T*)logits, p, per_warp);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

void sample(const void* logits, bool bf16, int B, int V, int stride, const float* temperature, const int* top_k,
            const float* top_p, const float* min_p, const long long* seeds, const int* out_slots, int* next_token_buf,
            int* out_tokens, float* out_logprobs, unsigned long long global_seed, const long long* step_ptr, long long step,
            cudaStream_t stream) {
  if (B <= 0) return;
  SampleParams p{temperature, top_k, top_p, min_p, seeds, out_slots, next_token_buf, out_tokens, out_logprobs, global_seed,
                 step_ptr, step, V, stride};
  if (bf16) launch_sample<__nv_bfloat16>(logits, p, B, stream);
  else launch_sample<float>(logits, p, B, stream);
}

// ---------------------------------------------------------------- grammar bitmask: logits[b, v] = -inf where bit == 0
// ---- vocab-parallel greedy decoding: no [B, V] logits all-gather on the TP decode path.
// Every rank takes the argmax of its own vocabulary shard and publishes 4 bf16 words per row — (max logit, idx byte 0, 1, 2), all exactly
// representable — into its own [rank] plane of a [tp, Bpad, 4] buffer whose other planes it zeroes; the arena all-reduce (a sum with
// zeros: exact) then is an all-gather of 8 bytes per (rank, row), and greedy_merge_kernel picks the winner (ties -> lowest global index,
// as torch.argmax on the gathered row would).  Reference counterpart: the full-logits all-gather in layers/logits_processor.py:877-905.
template <typename T>
__global__ void __launch_bounds__(SAMP_THREADS) greedy_shard_kernel(const T* __restrict__ logits, int stride, int v_valid, int v_offset,
                                                                    int rank, int tp, int b_pad, __nv_bfloat16* __restrict__ buf) {
  __shared__ float red[32];
  __shared__ int s_arg;
  const int row = blockIdx.x, tid = threadIdx.x;
  const T* lr = logits + (size_t)row * stride;
  float mx = -INFINITY; int am = 0x7fffffff;
  for (int i = tid; i < v_valid; i += SAMP_THREADS) {
    const float v = to_f<T>(lr[i]);
    if (v > mx) { mx = v; am = i; }
  }
  const float gmax = block_reduce_max(mx, red);
  if (tid == 0) s_arg = 0x7fffffff;
  __syncthreads();
  if (mx == gmax && am != 0x7fffffff) atomicMin(&s_arg, am);
  __syncthreads();
  if (tid < tp) {
    __nv_bfloat16* dst = buf + ((size_t)tid * b_pad + row) * 4;
    if (tid == rank) {
      const int g = (s_arg == 0x7fffffff) ? 0 : (s_arg + v_offset);
      // a shard with no valid column (padding past the real vocabulary) publishes the most negative finite bf16
      const float val = (s_arg == 0x7fffffff) ? -3.3e38f : fmaxf(gmax, -3.3e38f);
      dst[0] = __float2bfloat16(val);
      dst[1] = __float2bfloat16((float)(g & 255));
      dst[2] = __float2bfloat16((float)((g >> 8) & 255));
      dst[3] = __float2bfloat16((float)((g >> 16) & 255));
    } else {
      dst[0] = dst[1] = dst[2] = dst[3] = __float2bfloat16(0.f);
    }
  }
}

__global__ void greedy_merge_kernel(const __nv_bfloat16* __restrict__ buf, int tp, int b_pad, int B, const int* __restrict__ out_slots,
                                    int* __restrict__ next_token_buf, int* __restrict__ out_tokens) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= B) return;
  float best = -INFINITY; int tok = 0;
  for (int r = 0; r < tp; ++r) {
    const __nv_bfloat16* src = buf + ((size_t)r * b_pad + row) * 4;
    const float v = __bfloat162float(src[0]);
    if (v > best) {          // strict: equal maxima keep the lower rank = the lower global index
      best = v;
      tok = (int)__bfloat162float(src[1]) | ((int)__bfloat162float(src[2]) << 8) | ((int)__bfloat162float(src[3]) << 16);
    }
  }
  out_tokens[row] = tok;
  if (next_token_buf != nullptr && out_slots != nullptr) next_token_buf[out_slots[row]] = tok;
}

void greedy_shard(const void* logits, bool bf16, int B, int stride, int v_valid, int v_offset, int rank, int tp, int b_pad, void* buf,
                  cudaStream_t stream) {
  if (B <= 0) return;
  if (tp > 32) throw std::runtime_error("sglb greedy_shard: tp <= 32");
  if (bf16)
    greedy_shard_kernel<__nv_bfloat16><<<B, SAMP_THREADS, 0, stream>>>((const __nv_bfloat16*)logits, stride, v_valid, v_offset, rank, tp, b_pad,
                                                                       (__nv_bfloat16*)buf);
  else
    greedy_shard_kernel<float><<<B, SAMP_THREADS, 0, stream>>>((const float*)logits, stride, v_valid, v_offset, rank, tp, b_pad, (__nv_bfloat16*)buf);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

void greedy_merge(const void* buf, int tp, int b_pad, int B, const int* out_slots, int* next_token_buf, int* out_tokens, cudaStream_t stream) {
  if (B <= 0) return;
  greedy_merge_kernel<<<(B + 255) / 256, 256, 0, stream>>>((const __nv_bfloat16*)buf, tp, b_pad, B, out_slots, next_token_buf, out_tokens);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

template <typename T>
__global__ void apply_bitmask_kernel(T* __restrict__ logits, const int* __restrict__ bitmask, const int* __restrict__ row_idx,
                                     int V, int stride, int words) {
  const int r = blockIdx.y;
  const int row = row_idx ? row_idx[r] : r;
  T* lr = logits + (size_t)row * stride;
  const int* bm = bitmask + (size_t)r * words;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x) {
    const unsigned bits = (unsigned)bm[w];
    if (bits == 0xffffffffu) continue;
#pragma unroll 4
    for (int b = 0; b < 32; ++b) {
      const int v = w * 32 + b;
      if (v < V && !((bits >> b) & 1u)) lr[v] = T(-INFINITY);
    }
  }
}
void apply_token_bitmask(void* logits, bool bf16, const int* bitmask, const int* row_idx, int n_rows, int V, int stride,
                         cudaStream_t stream) {
  if (n_rows <= 0) return;
  const int words = (V + 31) / 32;
  dim3 grid(min((words + 255) / 256, 16), n_rows);
  if (bf16) apply_bitmask_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>((__nv_bfloat16*)logits, bitmask, row_idx, V, stride, words);
  else apply_bitmask_kernel<float><<<grid, 256, 0, stream>>>((float*)logits, bitmask, row_idx, V, stride, words);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------- penalties (frequency / presence / repetition) + logit bias
// counts: int32 [B, V] occurrences in the generated output; prompt_mask: uint8 [B, V] (optional)
__global__ void apply_penalties_kernel(float* __restrict__ logits, const int* __restrict__ counts,
                                       const unsigned char* __restrict__ prompt_mask, const float* __restrict__ freq,
                                       const float* __restrict__ pres, const float* __restrict__ rep, int V, int stride) {
  const int row = blockIdx.y;
  float* lr = logits + (size_t)row * stride;
  const int* cr = counts + (size_t)row * V;
  const float f = freq[row], pz = pres[row], rp = rep[row];
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const int c = cr[v];
    const bool seen = c > 0 || (prompt_mask && prompt_mask[(size_t)row * V + v]);
    if (!seen) continue;
    float x = lr[v];
    if (rp != 1.f) x = x > 0.f ? x / rp : x * rp;
    x -= f * (float)c + (c > 0 ? pz : 0.f);
    lr[v] = x;
  }
}
void apply_penalties(float* logits, const int* counts, const unsigned char* prompt_mask, const float* freq, const float* pres,
                     const float* rep, int B, int V, int stride, cudaStream_t stream) {
  if (B <= 0) return;
  dim3 grid(min((V + 255) / 256, 64), B);
  apply_penalties_kernel<<<grid, 256, 0, stream>>>(logits, counts, prompt_mask, freq, pres, rep, V, stride);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

__global__ void bump_counts_kernel(int* __restrict__ counts, const int* __restrict__ tokens, int V, int B) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < B) atomicAdd(&counts[(size_t)b * V + tokens[b]], 1);
}
void bump_counts(int* counts, const int* tokens, int B, int V, cudaStream_t stream) {
  if (B <= 0) return;
  bump_counts_kernel<<<(B + 127) / 128, 128, 0, stream>>>(counts, tokens, V, B);
  SGLB_CUDA_CHECK(cudaGetLastError());
}

}  // namespace sglb
