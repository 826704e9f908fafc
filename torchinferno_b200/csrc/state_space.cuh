// What the kernels of the state-space scan share.
#pragma once

#include "common.cuh"

namespace tib {

__device__ __forceinline__ float ss_load(const void* p, int dtype, size_t i) {
  return dtype == TIB_F32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ __forceinline__ float ss_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

struct ScanArgs {
  const void* xbc; int xbc_dtype; int64_t ld_xbc;        // rows [x: heads * P | B: groups * N | C: groups * N]
  const void* dt; int dt_dtype; int64_t ld_dt; int dt_col;   // raw step sizes: column dt_col + h of a row
  const float* dt_bias; const float* a_log; const float* d_skip;   // [heads] each
  float* state; int64_t state_stride;                      // per slot: S [heads][N][P] at offset 0
  const int* q_start; const int* slots;
  float* y;                                                // [tokens, heads * P] fp32
  float* run_state; float* run_decay;                      // [runs][heads * N * P], [runs][heads]
  int heads, groups, N, P;
  int* error_word;
};

// Long portions of bf16 rows on the tensor cores (ssd_chunks.cu), where ssd_chunks_takes them: run_state [runs][heads * N * P] and
// run_decay [runs][heads] with n_tokens / kSsdChunk + n_entries runs.
constexpr int kSsdChunk = 128;
bool ssd_chunks_takes(const ScanArgs& a);
int ssd_chunks(const ScanArgs& a, int n_entries, int n_tokens, int max_q_len, cudaStream_t stream);
// The same for heads in whole tiles of 64 columns (ssd_tcgen05.cu), and what both run between sums and outputs.
int ssd_tcgen05(const ScanArgs& a, int n_entries, int n_tokens, int max_q_len, cudaStream_t stream);
int ssd_fold(const ScanArgs& a, int n_entries, cudaStream_t stream);

}  // namespace tib
