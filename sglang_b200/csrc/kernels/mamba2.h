// Arguments of the Mamba-2 recurrence, shared by its kernels (mamba.cu: token by token and eight tokens a step; mamba_chunk.cu: 64 tokens a step).
#pragma once
#include <cuda_runtime.h>

namespace sglb {

struct Mamba2Params {
  const float* u; int ldu;                       // conv outputs [T, ldu] = [x (H*P) | B (G*N) | C (G*N)]
  const void* z; int ldz;                        // gate rows (model dtype) or null
  const void* dt_raw; int lddt;                  // [T, >= H] (model dtype)
  const float* dt_bias; const float* A_log; const float* D;
  const float* decay;                            // non-null: step size 1 and the head's constant decay (dt_raw, dt_bias, A_log unused)
  const float* gates; int gstride;               // non-null: [T, H, gstride] with every token's decay at [0] and step at [1] (likewise)
  float* state;                                  // [slots, H, N, P]
  const int* req_slots; const int* seq_lens; const int* cu_q;
  float* out;                                    // [T, H*P]
  int H, P, N, G, pchunks;
};

__device__ __forceinline__ float m2_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// 64 tokens a step on the tensor cores.  The workspace's size; 0: not this form's sizes or alignment
size_t mamba2_chunk_workspace(const float* u, int ldu, int B, int T, int H, int P, int N, int G);
void mamba2_chunk_scan(const Mamba2Params& p, bool z_bf16, int B, int T, void* ws, cudaStream_t stream);

}  // namespace sglb
