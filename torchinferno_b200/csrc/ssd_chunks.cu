// The state-space scan of long portions in chunks of 128 tokens, as products (state-space duality).  With F_t the sum of the log
// decays from the chunk's start to token t, dt the step sizes and S the state at the chunk's start:
//     y_i  = exp(F_i) S^T C_i + sum_(j <= i) (C_i . B_j) exp(F_i - F_j) dt_j x_j + D x_i
//     S'   = exp(F_end) S + sum_j exp(F_end - F_j) dt_j B_j x_j^T
//
//   ssd_sums    every chunk's own sum (the last line's second term) and exp(F_end)
//   ssd_fold    S' = exp(F_end) S + sum over a request's chunks, an element a thread
//   ssd_outs    y from the state at the chunk's start
//
// x, B and C are bf16 as the convolution left them, so C . B is a product of exact operands with fp32 sums.  Whatever is 32-bit
// (the state, the weighted scores, the weighted x) enters its product as three bf16 terms, which hold all 24 bits of an fp32
// number; F is summed in double precision and kept as two floats, so that differences of long sums keep their last bits.  The
// tensor core's own sums are cut off rather than rounded, so only the 16 terms of a step (small ones first) are left to it, and
// the steps are added as ordinary fp32 numbers.  What is not finite stays with the tokens it concerns, as in the walk, though an
// infinity may come out as NaN (where it meets a term or a decay of zero).
//
// Heads in whole tiles of 64 columns run the first and the last on tcgen05 (ssd_tcgen05.cu); the kernels here, on mma.sync, take tiles of 32 (heads
// of 32 or 96 columns).  The walk of ssd_scan_kernel spends five fp32 operations per state element and token twice over (two prompts of 1,366
// and 682 tokens, 64 heads of 64 with a state of 128: 182 + 32 + 264 us, the fp32 pipe at 40 %), the products took 39 + 32 + 98 us
// cold here and take 30 + 32 + 66 there.  Error against 64 bits of such a scan: y 9.8e-8 in both, the walk 8.5e-8; with steps of e^-8 and less, where
// the walk adds a thousand small terms one by one, 1e-7 against 6e-6.  What bounds it: the legacy tensor path with operands from shared memory,
// and the states' way through the L2 (one of 32 KB a head of 64 and chunk, written twice and read twice).
#include "state_space.cuh"
#include "split_terms.cuh"
#include <type_traits>

namespace tib {

constexpr int kQ = kSsdChunk;
constexpr int kSsdThreads = 256;
constexpr int kSsdTile = 32;            // columns of a head a block takes
constexpr int kSsdRows = 32;            // rows of the state staged at a time

__device__ __forceinline__ size_t ssd_first_chunk(int row0, int entry) { return (size_t)(row0 / kQ) + entry; }

// d = a . b over eight of the sixteen k of a fragment (halves 0 and 1)
__device__ __forceinline__ void ssd_mma8(float (&d)[4], const uint32_t (&a)[4], uint32_t b, int half) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[2 * half]), "r"(a[2 * half + 1]), "r"(b));
}
__device__ __forceinline__ void ssd_add(float (&sum)[4], const float (&step)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) sum[c] += step[c];
}

// Step sizes and sums of log decays of a chunk's n tokens (tokens behind it: no step, the sum stays).  Called by the whole block;
// ends with a barrier.
struct SsdSteps {
  float dt[kQ], fh[kQ], fl[kQ], w[kQ];  // F = fh + fl; w: what a token weighs in the chunk's sum
  double warp_sum[4];
};
__device__ __forceinline__ void ssd_steps(SsdSteps& s, const ScanArgs& a, int h, size_t first_row, int n) {
  const int t = threadIdx.x, lane = t & 31;
  double f = 0.0;
  if (t < kQ) {
    float step = 0.f;
    if (t < n) {
      step = ss_softplus(ss_load(a.dt, a.dt_dtype, (first_row + t) * a.ld_dt + a.dt_col + h) + a.dt_bias[h]);
      const float log_decay = -expf(a.a_log[h]) * step;
      f = (double)(log_decay < -1e4f ? -1e4f : log_decay);      // (a decay of zero either way, and no infinity in the sums)
    }
    s.dt[t] = step;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, f, o);
      if (lane >= o) f += up;
    }
    if (lane == 31) s.warp_sum[t >> 5] = f;
  }
  __syncthreads();
  if (t < kQ) {
    for (int w = 0; w < (t >> 5); ++w) f += s.warp_sum[w];
    const float hi = (float)f;
    s.fh[t] = hi;
    s.fl[t] = (float)(f - (double)hi);
  }
  __syncthreads();
}
__device__ __forceinline__ float ssd_decay(const SsdSteps& s, int to, int from) { return expf((s.fh[to] - s.fh[from]) + (s.fl[to] - s.fl[from])); }

// 16-byte copies of n rows of WIDTH elements (row stride ld) into [kQ][WIDTH + 8]; rows behind them are zeroed.
template <int WIDTH>
__device__ __forceinline__ void ssd_rows(__nv_bfloat16* dst, const __nv_bfloat16* src, int64_t ld, int n) {
  for (int p = threadIdx.x; p < kQ * WIDTH / 8; p += kSsdThreads) {
    const int r = p / (WIDTH / 8), c = (p % (WIDTH / 8)) * 8;
    cp_async16(dst + r * (WIDTH + 8) + c, src + (r < n ? (size_t)r * ld : 0) + c, r < n);
  }
}

// grid (heads * column tiles, chunks, entries)
template <int N, int PT>
__global__ void __launch_bounds__(kSsdThreads, 2) ssd_sums_kernel(ScanArgs a) {
  extern __shared__ __align__(16) __nv_bfloat16 ssd_smem[];
  constexpr int NS = N + 8, PS = PT + 8;
  __nv_bfloat16* bs = ssd_smem;                 // [kQ][NS]
  __nv_bfloat16* wx = bs + kQ * NS;             // [3][kQ][PS]: weighted x in three terms
  __shared__ SsdSteps st;
  pdl_wait();
  pdl_trigger();
  const int entry = blockIdx.z, row0 = a.q_start[entry], len = a.q_start[entry + 1] - row0;
  const int t0 = blockIdx.y * kQ;
  if (t0 >= len) return;
  const int n = min(kQ, len - t0), tiles = a.P / PT, h = blockIdx.x / tiles, p0 = (blockIdx.x - h * tiles) * PT;
  const int inner = a.heads * a.P, g = h / (a.heads / a.groups);
  const size_t first = (size_t)(row0 + t0);
  const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(a.xbc) + first * a.ld_xbc;
  ssd_rows<N>(bs, rows + inner + g * N, a.ld_xbc, n);
  cp_async_commit();
  constexpr int XV = kQ * PT / 8 / kSsdThreads;      // 16-byte pieces of x a thread fetches (zeros behind the chunk's tokens)
  uint4 xv[XV];
#pragma unroll
  for (int i = 0; i < XV; ++i) {
    const int p = threadIdx.x + i * kSsdThreads, r = p / (PT / 8), c = (p % (PT / 8)) * 8;
    xv[i] = r < n ? *reinterpret_cast<const uint4*>(rows + (size_t)r * a.ld_xbc + h * a.P + p0 + c) : make_uint4(0u, 0u, 0u, 0u);
  }
  ssd_steps(st, a, h, first, n);
  if (threadIdx.x < kQ) st.w[threadIdx.x] = (int)threadIdx.x < n ? ssd_decay(st, n - 1, threadIdx.x) * st.dt[threadIdx.x] : 0.f;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < XV; ++i) {
    const int p = threadIdx.x + i * kSsdThreads, r = p / (PT / 8), c = (p % (PT / 8)) * 8;
    const float w = st.w[r];
    const uint32_t raw[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
    uint32_t term[3][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 v = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&raw[q]));
      ft_split2_finite(v.x * w, v.y * w, term[0][q], term[1][q], term[2][q]);
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) *reinterpret_cast<uint4*>(wx + (u * kQ + r) * PS + c) = make_uint4(term[u][0], term[u][1], term[u][2], term[u][3]);
  }
  cp_async_wait<0>();
  __syncthreads();
  // warps: N / 16 groups of 16 state rows, the rest of the warps share the columns
  constexpr int RG = N / 16, CH = 8 / RG, CW = PT / CH, NT = CW / 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m0 = (warp % RG) * 16, c0 = (warp / RG) * CW;
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
  const int steps = (n + 15) / 16;
  for (int ks = 0; ks < steps; ++ks) {
    uint32_t av[4];      // (state row, token), read transposed from [token][state row]
    ldmatrix_x4_trans(av, bs + (ks * 16 + (lane >> 4) * 8 + (lane & 7)) * NS + m0 + ((lane >> 3) & 1) * 8);
#pragma unroll
    for (int j = 0; j < NT / 2; ++j) {
      float step[2][4] = {};
#pragma unroll
      for (int u = 2; u >= 0; --u) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, wx + (u * kQ + ks * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * PS + c0 + j * 16 + ((lane >> 4) << 3));
        mma_bf16(step[0], av, b[0], b[1]);
        mma_bf16(step[1], av, b[2], b[3]);
      }
      ssd_add(acc[2 * j], step[0]);
      ssd_add(acc[2 * j + 1], step[1]);
    }
  }
  const size_t run = ssd_first_chunk(row0, entry) + blockIdx.y;
  float* dst = a.run_state + (run * a.heads + h) * (size_t)N * a.P + p0 + c0;
  const int gr = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int half = 0; half < 2; ++half)
      *reinterpret_cast<float2*>(dst + (size_t)(m0 + gr + half * 8) * a.P + i * 8 + 2 * t4) = make_float2(acc[i][2 * half], acc[i][2 * half + 1]);
  if (p0 == 0 && threadIdx.x == 0) a.run_decay[run * a.heads + h] = expf(st.fh[n - 1] + st.fl[n - 1]);
}

// grid (state elements / 1024, entries), four elements a thread: run_state turns from a chunk's sum into the state at its start.
template <int AHEAD>      // chunks whose sums a thread has on their way
__global__ void __launch_bounds__(256) ssd_fold_kernel(ScanArgs a) {
  pdl_wait();
  pdl_trigger();
  const int entry = blockIdx.y, row0 = a.q_start[entry], len = a.q_start[entry + 1] - row0;
  const size_t per_head = (size_t)a.N * a.P, width = per_head * a.heads;
  const size_t e = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (len <= 0 || e >= width) return;
  const int h = (int)(e / per_head), runs = (len + kQ - 1) / kQ;
  const size_t run0 = ssd_first_chunk(row0, entry);
  float* run = a.run_state + run0 * width + e;
  const float* decays = a.run_decay + run0 * a.heads + h;
  float4* slot = reinterpret_cast<float4*>(a.state + (size_t)a.slots[entry] * a.state_stride + e);
  float4 s = *slot;
  for (int r = 0; r < runs; r += AHEAD) {
    float4 sum[AHEAD];
    float decay[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (r + u < runs) {
        sum[u] = *reinterpret_cast<const float4*>(run + (size_t)(r + u) * width);
        decay[u] = decays[(size_t)(r + u) * a.heads];
      }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (r + u >= runs) break;
      *reinterpret_cast<float4*>(run + (size_t)(r + u) * width) = s;
      s = make_float4(fmaf(decay[u], s.x, sum[u].x), fmaf(decay[u], s.y, sum[u].y), fmaf(decay[u], s.z, sum[u].z), fmaf(decay[u], s.w, sum[u].w));
    }
  }
  *slot = s;
}

// grid (heads * column tiles, chunks, entries): a warp owns 16 tokens and all PT columns.
template <int N, int PT>
__global__ void __launch_bounds__(kSsdThreads, 2) ssd_outs_kernel(ScanArgs a) {
  extern __shared__ __align__(16) __nv_bfloat16 ssd_smem[];
  constexpr int NS = N + 8, PS = PT + 8, NT = PT / 8;
  __nv_bfloat16* cs = ssd_smem;                 // [kQ][NS]
  __nv_bfloat16* bs = cs + kQ * NS;             // [kQ][NS]
  __nv_bfloat16* xs = bs + kQ * NS;             // [kQ][PS]
  __nv_bfloat16* ss = xs + kQ * PS;             // [3][kSsdRows][PS]: rows of the state in three terms
  __shared__ SsdSteps st;
  pdl_wait();
  pdl_trigger();
  const int entry = blockIdx.z, row0 = a.q_start[entry], len = a.q_start[entry + 1] - row0;
  const int t0 = blockIdx.y * kQ;
  if (t0 >= len) return;
  const int n = min(kQ, len - t0), tiles = a.P / PT, h = blockIdx.x / tiles, p0 = (blockIdx.x - h * tiles) * PT;
  const int inner = a.heads * a.P, g = h / (a.heads / a.groups);
  const size_t first = (size_t)(row0 + t0);
  const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(a.xbc) + first * a.ld_xbc;
  ssd_rows<N>(cs, rows + inner + (a.groups + g) * N, a.ld_xbc, n);
  cp_async_commit();
  ssd_rows<N>(bs, rows + inner + g * N, a.ld_xbc, n);
  ssd_rows<PT>(xs, rows + h * a.P + p0, a.ld_xbc, n);
  cp_async_commit();
  const float* S = a.run_state + ((ssd_first_chunk(row0, entry) + blockIdx.y) * a.heads + h) * (size_t)N * a.P + p0;
  constexpr int SV = kSsdRows * PT / 4 / kSsdThreads;
  float4 sv[SV];
  auto ask = [&](int r0) {
#pragma unroll
    for (int i = 0; i < SV; ++i) {
      const int p = threadIdx.x + i * kSsdThreads;
      sv[i] = *reinterpret_cast<const float4*>(S + (size_t)(r0 + p / (PT / 4)) * a.P + (p % (PT / 4)) * 4);
    }
  };
  ask(0);
  ssd_steps(st, a, h, first, n);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m0 = warp * 16, gr = lane >> 2, t4 = lane & 3;
  cp_async_wait<1>();
  __syncthreads();                              // C has landed
  uint32_t cv[N / 16][4];
#pragma unroll
  for (int k = 0; k < N / 16; ++k) ldmatrix_x4(cv[k], cs + (m0 + (lane & 15)) * NS + k * 16 + (lane >> 4) * 8);
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
#pragma unroll
  for (int r0 = 0; r0 < N; r0 += kSsdRows) {
#pragma unroll
    for (int i = 0; i < SV; ++i) {
      const int p = threadIdx.x + i * kSsdThreads, r = p / (PT / 4), c = (p % (PT / 4)) * 4;
      uint32_t lo[3], hi[3];
      ft_split2_finite(sv[i].x, sv[i].y, lo[0], lo[1], lo[2]);
      ft_split2_finite(sv[i].z, sv[i].w, hi[0], hi[1], hi[2]);
#pragma unroll
      for (int u = 0; u < 3; ++u) *reinterpret_cast<uint2*>(ss + (u * kSsdRows + r) * PS + c) = make_uint2(lo[u], hi[u]);
    }
    __syncthreads();
    if (r0 + kSsdRows < N) ask(r0 + kSsdRows);
    if (m0 < n) {
#pragma unroll
      for (int k = 0; k < kSsdRows / 16; ++k)
#pragma unroll
        for (int j = 0; j < NT / 2; ++j) {
          float step[2][4] = {};
#pragma unroll
          for (int u = 2; u >= 0; --u) {
            uint32_t b[4];
            ldmatrix_x4_trans(b, ss + (u * kSsdRows + k * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * PS + j * 16 + ((lane >> 4) << 3));
            mma_bf16(step[0], cv[r0 / 16 + k], b[0], b[1]);
            mma_bf16(step[1], cv[r0 / 16 + k], b[2], b[3]);
          }
          ssd_add(acc[2 * j], step[0]);
          ssd_add(acc[2 * j + 1], step[1]);
        }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  __syncthreads();                              // B and x have landed
  if (m0 >= n) return;
  const int i0 = m0 + gr, i1 = i0 + 8;
  {
    const float f0 = expf(st.fh[i0] + st.fl[i0]), f1 = expf(st.fh[i1] + st.fl[i1]);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      acc[i][0] *= f0; acc[i][1] *= f0;
      acc[i][2] *= f1; acc[i][3] *= f1;
    }
  }
  // Among the warp's own tokens a later one weighs 0, which must not meet an infinity or NaN: what is not finite there stays out of the
  // product and is added below, to the tokens it does not come after.  (A prompt of 2,048 tokens, 64 heads of 64: the layer takes 254 us
  // without any look, 263 with the check and the repair in the loop, 258 so.)
  bool odd = false;
#pragma unroll
  for (int p = lane; p < 16 * PT / 8; p += 32) {
    const uint4 v = *reinterpret_cast<const uint4*>(xs + (m0 + p / (PT / 8)) * PS + (p % (PT / 8)) * 8);
    odd |= (ft_finite2(v.x) & ft_finite2(v.y) & ft_finite2(v.z) & ft_finite2(v.w)) != 0xffffffffu;
  }
  odd = __any_sync(0xffffffffu, odd);
  const auto within = [&](auto checked) {         // (the common case without the check)
    constexpr bool CHECKED = decltype(checked)::value;
    for (int j0 = 0; j0 <= m0; j0 += 16) {        // 16 tokens before (or among) the warp's own
      float s[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[i][c] = 0.f;
#pragma unroll
      for (int k = 0; k < N / 16; ++k) {
        uint32_t b[4];
        ldmatrix_x4(b, bs + (j0 + ((lane >> 4) << 3) + (lane & 7)) * NS + k * 16 + ((lane >> 3) & 1) * 8);
        float step[4][4] = {};
        ssd_mma8(step[0], cv[k], b[0], 0);
        ssd_mma8(step[1], cv[k], b[1], 1);
        ssd_mma8(step[2], cv[k], b[2], 0);
        ssd_mma8(step[3], cv[k], b[3], 1);
        ssd_add(step[0], step[1]);
        ssd_add(step[2], step[3]);
        ssd_add(s[0], step[0]);
        ssd_add(s[1], step[2]);
      }
      uint32_t w[3][4];
#pragma unroll
      for (int half = 0; half < 2; ++half)        // (tokens j0 + 8 half + 2 t4 and the next one)
#pragma unroll
        for (int r = 0; r < 2; ++r) {             // (rows i0, i1)
          const int i = r == 0 ? i0 : i1, j = j0 + half * 8 + 2 * t4;
          const float v0 = j <= i ? s[half][2 * r] * (ssd_decay(st, i, j) * st.dt[j]) : 0.f;
          const float v1 = j + 1 <= i ? s[half][2 * r + 1] * (ssd_decay(st, i, j + 1) * st.dt[j + 1]) : 0.f;
          ft_split2_finite(v0, v1, w[0][half * 2 + r], w[1][half * 2 + r], w[2][half * 2 + r]);
        }
#pragma unroll
      for (int j = 0; j < NT / 2; ++j) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, xs + (j0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * PS + j * 16 + ((lane >> 4) << 3));
        if (CHECKED && j0 == m0) {
#pragma unroll
          for (int q = 0; q < 4; ++q) b[q] &= ft_finite2(b[q]);
        }
        float step[2][4] = {};
#pragma unroll
        for (int u = 2; u >= 0; --u) {
          mma_bf16(step[0], w[u], b[0], b[1]);
          mma_bf16(step[1], w[u], b[2], b[3]);
        }
        ssd_add(acc[2 * j], step[0]);
        ssd_add(acc[2 * j + 1], step[1]);
      }
    }
  };
  if (odd) within(std::true_type{});
  else within(std::false_type{});
  if (odd) {
#pragma unroll 1
    for (int j = m0; j < m0 + 16; ++j)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = r == 0 ? i0 : i1;
        if (j > i) continue;
        float weight = 0.f;
        for (int k = 0; k < N; ++k) weight = fmaf(__bfloat162float(cs[i * NS + k]), __bfloat162float(bs[j * NS + k]), weight);
        weight *= ssd_decay(st, i, j) * st.dt[j];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const float2 x = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(xs + j * PS + t * 8 + 2 * t4));
          if (!isfinite(x.x)) acc[t][2 * r] = fmaf(weight, x.x, acc[t][2 * r]);
          if (!isfinite(x.y)) acc[t][2 * r + 1] = fmaf(weight, x.y, acc[t][2 * r + 1]);
        }
      }
  }
  const float skip = a.d_skip[h];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int i = r == 0 ? i0 : i1;
    if (i >= n) continue;
    float* dst = a.y + (first + i) * inner + h * a.P + p0;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const float2 x = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(xs + i * PS + t * 8 + 2 * t4));
      *reinterpret_cast<float2*>(dst + t * 8 + 2 * t4) = make_float2(fmaf(skip, x.x, acc[t][2 * r]), fmaf(skip, x.y, acc[t][2 * r + 1]));
    }
  }
}

int ssd_fold(const ScanArgs& a, int n_entries, cudaStream_t stream) {
  const dim3 grid((unsigned)ceil_div64((int64_t)a.heads * a.N * a.P, 1024), n_entries);
  // Four chunks' sums on their way a thread where there are five blocks an SM and more, which fill the memory with fewer registers a thread, else eight
  // (layers on 600 to 2,600 tokens, us with four and eight: 192 blocks 148 and 142, 512 103 and 102, 640 108 and 108, 1,024 174 and 177, 1,536 174
  // and 179, 2,560 303 and 311; two prompts of 1,366 and 682 tokens, 64 heads of 64: the fold 14.5 -> 11.4 behind the sums, with twelve 17, with two 19).
  if ((int64_t)grid.x * grid.y >= 5 * 148) TIB_LAUNCH_DEPENDENT(ssd_fold_kernel<4>, grid, 256, 0, stream, a);
  else TIB_LAUNCH_DEPENDENT(ssd_fold_kernel<8>, grid, 256, 0, stream, a);
  return TIB_OK;
}

template <int N>
static int launch_ssd_chunks(const ScanArgs& a, int n_entries, int max_q_len, cudaStream_t stream) {
  constexpr int PT = kSsdTile, sums = 2 * (kQ * (N + 8) + 3 * kQ * (PT + 8)), outs = 2 * (2 * kQ * (N + 8) + kQ * (PT + 8) + 3 * kSsdRows * (PT + 8));
  cudaError_t e = cudaFuncSetAttribute(ssd_sums_kernel<N, PT>, cudaFuncAttributeMaxDynamicSharedMemorySize, sums);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(ssd_outs_kernel<N, PT>, cudaFuncAttributeMaxDynamicSharedMemorySize, outs);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid(a.heads * (a.P / PT), ceil_div(max_q_len, kQ), n_entries);
  TIB_LAUNCH_DEPENDENT((ssd_sums_kernel<N, PT>), grid, kSsdThreads, sums, stream, a);
  const int status = ssd_fold(a, n_entries, stream);
  if (status != TIB_OK) return status;
  TIB_LAUNCH_DEPENDENT((ssd_outs_kernel<N, PT>), grid, kSsdThreads, outs, stream, a);
  return TIB_OK;
}

// bf16 rows on 16-byte boundaries, a state of 64 or 128, heads in whole tiles of 32 columns, states on 16-byte boundaries.
bool ssd_chunks_takes(const ScanArgs& a) {
  const int64_t inner = (int64_t)a.heads * a.P;
  return a.xbc_dtype == TIB_BF16 && (a.N == 64 || a.N == 128) && a.P % 32 == 0 && a.ld_xbc % 8 == 0 && inner % 8 == 0 && a.state_stride % 4 == 0 &&
         (((uintptr_t)a.xbc | (uintptr_t)a.state | (uintptr_t)a.run_state | (uintptr_t)a.y) & 15) == 0;
}

int ssd_chunks(const ScanArgs& a, int n_entries, int n_tokens, int max_q_len, cudaStream_t stream) {
  if (a.P % 64 == 0) return ssd_tcgen05(a, n_entries, n_tokens, max_q_len, stream);
  return a.N == 128 ? launch_ssd_chunks<128>(a, n_entries, max_q_len, stream) : launch_ssd_chunks<64>(a, n_entries, max_q_len, stream);
}

}  // namespace tib
