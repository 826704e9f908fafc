// What the kernels of the attention in a window share.
#pragma once

#include "common.cuh"

namespace tib {

struct PwaCache {
  void* keys; void* values;          // first key / value of the layer's first page
  const int* block_table; int table_stride;
  int page_size; int64_t page_stride; int num_pages;
};

__device__ __forceinline__ int pwa_page(const PwaCache& c, const int* table, int index, int* error_word, int code) {
  const int page = table[index / c.page_size];
  if (page >= 0 && page < c.num_pages) return page;
  if (error_word) atomicExch(error_word, code);
  return -1;
}

struct PwaArgs {
  const int* q_start; const int* kv_start; const int* slots;
  int heads, kv_heads, dim, vdim;
  int window, pool;                  // pool 0: no blocks, only the window
  int keep;                          // tokens 0 .. keep - 1 are seen from behind the window too (pool 0 only)
  float scale;
  const float* temp; const float* sink;                    // [heads] or null
  const float* vfreq;                                      // [vdim / 2] or null (values were not turned)
  const float* turns;                                      // [tokens, vdim / 2, 2] cosine and sine of vfreq's angles at the tokens, or null
  const void* gate; int gate_dtype; int64_t ld_gate;       // [tokens, heads * vdim] logits or null
  const float* rel_bias; int rel_span;                     // [heads, rel_span] or null: added to a token's score by distance
  PwaCache tokens, blocks;
  int group_chunk, q_tile;
  int* error_word;
  int shortest, longest;                                   // portions this launch takes (window_tcgen05 / the mma.sync kernel)
  float* partial; int n_splits; int n_tokens;              // a step of single tokens whose contexts are shared out over blocks
};

// Prompt portions on the 5th-generation tensor cores (window_tcgen05.cu), where window_tcgen05_takes them: those of `shortest` tokens
// and more, which is more rows (tokens x query heads of a key head) than kWtFewRows, a tile of the mma.sync kernel, which keeps
// the others.
constexpr int kWtFewRows = 64;
bool window_tcgen05_takes(const PwaArgs& a, const void* q, const void* out, int max_q_len);
int window_tcgen05(const void* q, void* out, const PwaArgs& a, int n_entries, int max_q_len, cudaStream_t stream);

}  // namespace tib
