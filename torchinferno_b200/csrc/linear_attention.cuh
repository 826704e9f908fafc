// What the kernels of the decayed linear attention share.
#pragma once

#include "common.cuh"

namespace tib {

__device__ __forceinline__ float lin_act(float z, int activation) { return activation ? z / (1.f + expf(-z)) : z; }

constexpr int kLinRun = 128;            // tokens of a run

struct LinRunArgs {
  const int* q_start;
  const int* slots;
  const float* powers;    // [heads, kLinRun + 1]
  float* state;           // [slots, heads, D, value_dim]
  float* run_state;       // [runs, n_heads, D, value_dim]: L of a run, then the state at its start
  float* out;
  int64_t ldq, ldk, ldv;
  int heads, value_dim, activation;
  int head0, n_heads;     // the heads of these launches (the runs' states are made for some heads at a time)
  int shortest;           // portion that is cut into runs
  int* error_word;
};

// An entry's first run: entries' runs never overlap, since an entry of len tokens has at most len / kLinRun + 1 runs and the
// next entry starts len rows and one entry later.
__device__ __forceinline__ size_t lin_first_run(int row0, int entry) { return (size_t)(row0 / kLinRun) + entry; }

// Every run's own sum L and, once these are folded into the states at the runs' starts, every run's outputs (linear_tcgen05.cu).
int launch_lin_run_sums(const void* k, const void* v, const LinRunArgs& a, int dtype, int key_dim, int tile, dim3 grid, cudaStream_t stream);
int launch_lin_run_outs(const void* q, const void* k, const void* v, const LinRunArgs& a, int dtype, int key_dim, int tile, dim3 grid, cudaStream_t stream);

}  // namespace tib
