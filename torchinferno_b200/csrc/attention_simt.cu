// Paged causal attention on CUDA cores, for any head size, group size, page
// size and window.  It serves the 32-bit path of the engine and every shape the
// tensor-core kernels refuse.
//
// Formula (src/torchinferno/models/llama3/raw_ops.py:44-51): s = (q . k) / sqrt(d)
// (the scale is an argument), a key is allowed iff key_pos <= query_pos (and,
// with a window w > 0, query_pos - key_pos < w), p = softmax(s) in fp32, o = p . v.
// Streaming form with running max / sum / accumulator as in
// src/torchinferno/kernels/triton_ops.py:2555-2574.
//
// Exactness: one warp owns one (query token, query head) row from start to end.
// It walks the keys in blocks of 32 that are aligned to absolute positions
// (block b = keys 32b .. 32b+31), in rising order, so the arithmetic of a row
// depends only on its own position and keys, never on how the batch was cut,
// which other rows share the block, or which pages hold the keys.
#include "common.cuh"
#include <math_constants.h>

namespace tib {

// What bounds it: chains of loads and shuffles with four blocks of 16 rows an SM (128 registers a thread).  A warp works on its rows together, so
// that a key's four numbers, read at once, serve all of them, and a value's, the next block's keys and values are on their way meanwhile, and the
// rows' maxima and sums cross the lanes side by side.  Row by row and number by number, two loads a multiply-add, two portions of 200 and 101
// tokens, 32 / 8 heads of 64, took 117 us, 37 now (44 with one row's maximum and sum after the other's and divisions for every piece's place);
// 12 single tokens at 300, 32 heads of 128: 40 (55).  Five blocks an SM, at 96 registers: 45 and 58.
constexpr int kAttnWarps = 4;
constexpr int kAttnKeys = 32;                              // keys per step = lanes

struct AttnArgs {
  const int* q_start;      // [n_entries + 1] first token row of each entry
  const int* kv_start;     // [n_entries] position of the entry's first query token
  const int* slots;        // [n_entries] row of the block table
  const int* block_table;  // [slots, table_stride]
  int table_stride;
  int heads, kv_heads, head_dim;
  int page_size;
  int64_t page_stride;     // elements between pages of this layer
  int num_pages;
  int window;              // 0: all earlier keys
  float scale;
  int group_chunk;         // query heads of one kv head handled by one block
  int q_tile;              // query tokens per block
  int* error_word;
};

__device__ __forceinline__ float4 attn_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 attn_load4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
}

// R rows a warp; VEC: heads in whole fours of numbers, queries and pages on boundaries of four
template <typename T, int DPL, int R, bool VEC>
__device__ __forceinline__ void paged_attention_simt(const T* __restrict__ q, const T* __restrict__ pool, T* __restrict__ out, const AttnArgs& a) {
  extern __shared__ __align__(16) float smem[];
  constexpr int ROWS = kAttnWarps * R;
  const int d = a.head_dim, kd = VEC ? d + 4 : d + 1;      // row stride of the keys: no bank conflicts between neighbouring lanes
  float* q_s = smem;                           // [ROWS][d]
  float* k_s = q_s + ROWS * d;                 // [32][kd]
  float* v_s = k_s + kAttnKeys * kd;           // [32][d]
  float* p_s = v_s + kAttnKeys * d;            // [ROWS][32]: a row's weights

  pdl_wait();
  pdl_trigger();
  const int entry = blockIdx.y;
  const int group = a.heads / a.kv_heads;
  const int chunks = (group + a.group_chunk - 1) / a.group_chunk;
  const int kvh = blockIdx.z / chunks;
  const int g0 = (blockIdx.z - kvh * chunks) * a.group_chunk;
  const int gc = min(a.group_chunk, group - g0);

  const int row0 = a.q_start[entry];
  const int q_len = a.q_start[entry + 1] - row0;
  const int t0 = blockIdx.x * a.q_tile;
  if (t0 >= q_len) return;
  const int nt = min(a.q_tile, q_len - t0);
  const int nrows = nt * gc;
  const int pos0 = a.kv_start[entry] + t0;     // position of the first query of the tile
  const int last_pos = pos0 + nt - 1;          // highest key any row may read
  const int* table = a.block_table + (size_t)a.slots[entry] * a.table_stride;

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q_width = a.heads * d;
  constexpr int W = VEC ? 4 : 1;
  const int pieces = d / W;

  // Stage the queries (fp32).
  for (int e = threadIdx.x; e < nrows * pieces; e += blockDim.x) {
    const int r = e / pieces, dd = (e - r * pieces) * W;
    const int t = r / gc, g = r - t * gc;
    const T* src = q + (size_t)(row0 + t0 + t) * q_width + (kvh * group + g0 + g) * d + dd;
    if constexpr (VEC) *reinterpret_cast<float4*>(q_s + r * d + dd) = attn_load4(src);
    else q_s[r * d + dd] = to_f32(*src);
  }

  float m[R], l[R], acc[R][DPL];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m[i] = -CUDART_INF_F;
    l[i] = 0.f;
#pragma unroll
    for (int j = 0; j < DPL; ++j) acc[i][j] = 0.f;
  }

  int first_key = 0;
  if (a.window > 0) first_key = max(0, pos0 - a.window + 1);
  const int b_lo = first_key / kAttnKeys, b_hi = last_pos / kAttnKeys;

  // Keys and values of block b.  Keys past last_pos are not yet written (or belong to nobody): they are filled with zeros and
  // always masked.
  const int shift = (a.page_size & (a.page_size - 1)) == 0 ? 31 - __clz(a.page_size) : -1;      // (a division is 20 instructions)
  auto row_of = [&](int b, int j, int dd) -> const T* {
    const int kp = b * kAttnKeys + j;
    if (kp > last_pos || kp < first_key) return nullptr;
    const int at = shift >= 0 ? kp >> shift : kp / a.page_size, page = table[at];
    if (page >= 0 && page < a.num_pages) return pool + (size_t)page * a.page_stride + ((size_t)kvh * a.page_size + (kp - at * a.page_size)) * d + dd;
    if (a.error_word) atomicExch(a.error_word, 0x10000 + entry);
    return nullptr;
  };
  const size_t values = (size_t)a.kv_heads * a.page_size * d;
  constexpr int AHEAD = VEC ? 2 * DPL : 1;              // pieces a thread holds: the next block's are on their way under this one's work
  float4 k_next[AHEAD], v_next[AHEAD];
  // The thread's pieces of every block, kept in registers but with one row a warp and heads of 32, where they would take a block off every SM.
  constexpr bool KEPT = VEC && !(R == 1 && DPL == 1);
  int own_j[AHEAD], own_dd[AHEAD];
  auto own = [&](int i, int& j, int& dd) {
    const int e = threadIdx.x + i * kAttnWarps * 32;
    j = e / pieces;
    dd = (e - j * pieces) * W;
  };
  if constexpr (KEPT) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) own(i, own_j[i], own_dd[i]);
  }
  auto piece = [&](int i, int& j, int& dd) {
    if constexpr (KEPT) j = own_j[i], dd = own_dd[i];
    else own(i, j, dd);
  };
  auto ask = [&](int b) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      int j, dd;
      piece(i, j, dd);
      const T* from = j < kAttnKeys ? row_of(b, j, dd) : nullptr;
      k_next[i] = v_next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (from) {
        k_next[i] = attn_load4(from);
        v_next[i] = attn_load4(from + values);
      }
    }
  };
  if constexpr (VEC) ask(b_lo);
  for (int b = b_lo; b <= b_hi; ++b) {
    __syncthreads();  // previous block's tiles are no longer read (and q_s is written)
    if constexpr (VEC) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        int j, dd;
        piece(i, j, dd);
        if (j >= kAttnKeys) break;
        *reinterpret_cast<float4*>(k_s + j * kd + dd) = k_next[i];
        *reinterpret_cast<float4*>(v_s + j * d + dd) = v_next[i];
      }
      if (b < b_hi) ask(b + 1);
    } else {
      for (int e = threadIdx.x; e < kAttnKeys * pieces; e += blockDim.x) {
        const int j = e / pieces, dd = (e - j * pieces) * W;
        const T* from = row_of(b, j, dd);
        k_s[j * kd + dd] = from ? to_f32(*from) : 0.f;
        v_s[j * d + dd] = from ? to_f32(from[values]) : 0.f;
      }
    }
    __syncthreads();
    if (warp * R >= nrows) continue;                  // uniform in the warp

    // Scores: a lane's key with every row (a row behind the last one reads what lies there; nothing of it is kept).
    float s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) s[i] = 0.f;
    const float* qr = q_s + warp * R * d;
    const float* kr = k_s + lane * kd;
    if constexpr (VEC) {
#pragma unroll(KEPT ? 4 : 2)
      for (int dd = 0; dd < d; dd += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(kr + dd);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float4 qv = *reinterpret_cast<const float4*>(qr + i * d + dd);
          s[i] = fmaf(qv.x, kv.x, s[i]); s[i] = fmaf(qv.y, kv.y, s[i]);
          s[i] = fmaf(qv.z, kv.z, s[i]); s[i] = fmaf(qv.w, kv.w, s[i]);
        }
      }
    } else {
      for (int dd = 0; dd < d; ++dd) {
        const float kv = kr[dd];
#pragma unroll
        for (int i = 0; i < R; ++i) s[i] = fmaf(qr[i * d + dd], kv, s[i]);
      }
    }
    // The rows' softmax side by side, so that their chains of shuffles run together; a row that may read no key of the block keeps what it has.
    bool live[R], allowed[R];
    float top[R], p[R], sum[R];
    float* pw = p_s + warp * R * kAttnKeys;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = warp * R + i, qpos = pos0 + r / gc, kp = b * kAttnKeys + lane;
      const int lo = a.window > 0 ? max(0, qpos - a.window + 1) : 0;
      live[i] = r < nrows && b * kAttnKeys <= qpos && b * kAttnKeys + kAttnKeys - 1 >= lo;
      allowed[i] = kp <= qpos && kp >= lo;
      s[i] = allowed[i] ? s[i] * a.scale : -CUDART_INF_F;
      top[i] = s[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < R; ++i) top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], o));
#pragma unroll
    for (int i = 0; i < R; ++i) {
      top[i] = fmaxf(m[i], top[i]);                   // (finite where the row is live: the block holds an allowed key)
      p[i] = allowed[i] ? expf(s[i] - top[i]) : 0.f;
      sum[i] = p[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < R; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (!live[i]) continue;                         // (uniform in the warp)
      const float alpha = m[i] == -CUDART_INF_F ? 0.f : expf(m[i] - top[i]);
      l[i] = l[i] * alpha + sum[i];
      m[i] = top[i];
#pragma unroll
      for (int j = 0; j < DPL; ++j) acc[i][j] *= alpha;
      pw[i * kAttnKeys + lane] = p[i];
    }
    __syncwarp();
#pragma unroll 2
    for (int kk = 0; kk < kAttnKeys; kk += 4) {
      float v[4][DPL];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int j = 0; j < DPL; ++j) {
          const int dd = lane + 32 * j;
          v[c][j] = dd < d ? v_s[(kk + c) * d + dd] : 0.f;
        }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (!live[i]) continue;
        const float4 p = *reinterpret_cast<const float4*>(pw + i * kAttnKeys + kk);
#pragma unroll
        for (int j = 0; j < DPL; ++j) {
          acc[i][j] = fmaf(p.x, v[0][j], acc[i][j]); acc[i][j] = fmaf(p.y, v[1][j], acc[i][j]);
          acc[i][j] = fmaf(p.z, v[2][j], acc[i][j]); acc[i][j] = fmaf(p.w, v[3][j], acc[i][j]);
        }
      }
    }
  }

#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = warp * R + i;
    if (r >= nrows) continue;
    const int t = r / gc, g = r - t * gc;
    T* dst = out + (size_t)(row0 + t0 + t) * q_width + (kvh * group + g0 + g) * d;
    const float inv = 1.f / l[i];
#pragma unroll
    for (int j = 0; j < DPL; ++j) {
      const int dd = lane + 32 * j;
      if (dd < d) dst[dd] = from_f32<T>(acc[i][j] * inv);
    }
  }
}

template <typename T, int DPL, int R, bool VEC>
__global__ void __launch_bounds__(kAttnWarps * 32) paged_attention_simt_kernel(const T* __restrict__ q, const T* __restrict__ pool, T* __restrict__ out, AttnArgs a) {
  paged_attention_simt<T, DPL, R, VEC>(q, pool, out, a);
}

// Single tokens in heads of 128 with four blocks an SM where the compiler would rather have 167 registers and three: 512 blocks (32 tokens at 1,500, 16
// heads) 214 us, 357 with three; but 8 tokens 36.7 and 33.6.
template <typename T>
__global__ void __launch_bounds__(kAttnWarps * 32, 4) paged_attention_simt_four_kernel(const T* __restrict__ q, const T* __restrict__ pool, T* __restrict__ out, AttnArgs a) {
  paged_attention_simt<T, 4, 1, true>(q, pool, out, a);
}

template <typename T, int DPL, int R, bool VEC>
static int launch_attention_rows(const void* q, const void* pool, void* out, AttnArgs a, int n_entries, int max_q_len, cudaStream_t stream) {
  constexpr int ROWS = kAttnWarps * R;
  const int d = a.head_dim, group = a.heads / a.kv_heads;
  a.group_chunk = group < ROWS ? group : ROWS;
  a.q_tile = ROWS / a.group_chunk;
  const int chunks = (group + a.group_chunk - 1) / a.group_chunk;
  if ((int64_t)a.kv_heads * chunks > 65535) return TIB_E_SIZE;
  const size_t smem = sizeof(float) * ((size_t)ROWS * d + (size_t)kAttnKeys * (VEC ? d + 4 : d + 1) + (size_t)kAttnKeys * d + 3 + (size_t)ROWS * kAttnKeys);
  if (smem > 227 * 1024) return TIB_E_SMEM;
  auto kern = paged_attention_simt_kernel<T, DPL, R, VEC>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
    if (e != cudaSuccess) return (int)e;
  }
  dim3 grid(ceil_div(max_q_len, a.q_tile), n_entries, a.kv_heads * chunks);
  if constexpr (VEC && DPL == 4 && R == 1) {
    const int64_t blocks = (int64_t)grid.x * grid.y * grid.z;
    if (ceil_div64(blocks, 4 * 148) < ceil_div64(blocks, 3 * 148)) kern = paged_attention_simt_four_kernel<T>;
  }
  TIB_LAUNCH_DEPENDENT(kern, grid, kAttnWarps * 32, smem, stream, (const T*)q, (const T*)pool, (T*)out, a);
  return TIB_OK;
}

template <typename T, int DPL>
static int launch_attention(const void* q, const void* pool, void* out, const AttnArgs& a, int n_entries, int max_q_len, cudaStream_t stream) {
  const bool vec = a.head_dim % 4 == 0 && a.page_stride % 4 == 0 && (((uintptr_t)q | (uintptr_t)pool) & (4 * sizeof(T) - 1)) == 0;
  // Rows (token, head) a warp owns: four (eight or two of a block of the 1B sizes on 301 tokens: 390 and 375 us against 367); in steps of single
  // tokens as few as share a key head's queries out over the block's warps.
#define TIB_ATTN_ROWS(R) \
  (vec ? launch_attention_rows<T, DPL, R, true>(q, pool, out, a, n_entries, max_q_len, stream) : launch_attention_rows<T, DPL, R, false>(q, pool, out, a, n_entries, max_q_len, stream))
  const int group = a.heads / a.kv_heads;
  if (max_q_len == 1 && group <= kAttnWarps) return TIB_ATTN_ROWS(1);
  return TIB_ATTN_ROWS(4);
#undef TIB_ATTN_ROWS
}

}  // namespace tib

using namespace tib;

// q, out: [n_tokens, heads * head_dim]; pool: this layer's pages
// [pages][2][kv_heads][page_size][head_dim]; q_start: [n_entries + 1];
// kv_start, slots: [n_entries]; max_q_len: the longest entry of the batch.
TIB_API int tib_paged_attention_simt(const void* q, const void* pool, void* out, const int* q_start,
                                     const int* kv_start, const int* slots, const int* block_table,
                                     int table_stride, int n_entries, int max_q_len, int heads,
                                     int kv_heads, int head_dim, int page_size, int64_t page_stride,
                                     int num_pages, int window, float scale, int* error_word,
                                     int dtype, cudaStream_t stream) {
  if (n_entries == 0 || max_q_len == 0) return TIB_OK;
  if (!q || !pool || !out || !q_start || !kv_start || !slots || !block_table) return TIB_E_ARG;
  if (heads < 1 || kv_heads < 1 || heads % kv_heads != 0 || head_dim < 1 || page_size < 1) return TIB_E_SIZE;
  if (head_dim > 256) return TIB_E_SIZE;
  if (n_entries > 65535) return TIB_E_SIZE;
  AttnArgs a;
  a.q_start = q_start; a.kv_start = kv_start; a.slots = slots; a.block_table = block_table;
  a.table_stride = table_stride; a.heads = heads; a.kv_heads = kv_heads; a.head_dim = head_dim;
  a.page_size = page_size; a.page_stride = page_stride; a.num_pages = num_pages; a.window = window;
  a.scale = scale; a.error_word = error_word;
  const int dpl = (head_dim + 31) / 32;
#define TIB_ATTN_DISPATCH(T)                                                                     \
  (dpl <= 1 ? launch_attention<T, 1>(q, pool, out, a, n_entries, max_q_len, stream)             \
   : dpl <= 2 ? launch_attention<T, 2>(q, pool, out, a, n_entries, max_q_len, stream)           \
   : dpl <= 4 ? launch_attention<T, 4>(q, pool, out, a, n_entries, max_q_len, stream)           \
              : launch_attention<T, 8>(q, pool, out, a, n_entries, max_q_len, stream))
  if (dtype == TIB_F32) return TIB_ATTN_DISPATCH(float);
  if (dtype == TIB_BF16) return TIB_ATTN_DISPATCH(__nv_bfloat16);
#undef TIB_ATTN_DISPATCH
  return TIB_E_DTYPE;
}

// The calls the Python parts make (common.cuh).
TIB_PACKED(tib_paged_attention_simt)
