// The state-space scan in chunks of 128 tokens (the formulas are in ssd_chunks.cu) on the 5th-generation tensor cores, for heads in whole tiles of 64
// columns: every chunk's own sum and, once these are folded into the states at the chunks' starts, every chunk's outputs.
//
// x, B and C are bf16 as they come and are operands as they lie in memory; what is 32-bit (the state, the weighted scores, the weighted x)
// is three bf16 terms (split_terms.cuh).  The tensor core cuts its sums off, so the terms above 2^-8 of the whole are shared out over four
// accumulators, two instructions of 16 k each; the scores, made once for all heads of a block, over one for each 16 of the state.
//
// A block of 512 threads owns a chunk and several heads of a group, one after the other: B and C are fetched once, and a head's state and x are
// fetched and split while the products of the one before run.  Warp 0 issues them:
//     carried = C S                              (the scores are weighed, split and put into tensor memory meanwhile)
//     inside = weighted scores x                 (carried is read and scaled before; the next head's S and x are split meanwhile)
// A weight exp(F_i - F_j) dt_j is worked out by itself within a group of 32 tokens, by all four warps of the group; for earlier groups it is
// exp(F_i - F_r) times what j weighs at r, the last token of its group, both at most one.
//
// What bounds it: the threads' work around the products, 18,600 warp instructions a head and chunk for outputs and 8,000 for sums, at a third of the
// issue slots with one block of 16 warps an SM (tensor cores 12 %).  Two prompts of 1,366 and 682 tokens, 64 heads of 64, a state of 128: sums 29 us
// cold, outputs 65 (39 and 99 on mma.sync), the layer 230 (272), two of it for infinities that stay infinite.
// Weights of a group of 32 by two powers each, as between groups, made the outputs
// 55 us, and the scores in two accumulators of four instructions another 3 less, for errors of y of 1.3e-7 and 1.4e-7 where they are 9.8e-8 now and before.
#include "state_space.cuh"
#include "split_terms.cuh"

namespace tib {

constexpr int kQ = kSsdChunk, kStThreads = 512, kStItems = 12;      // (heads a block takes at most)
constexpr uint32_t kStSub = kQ * 128;                              // 128 rows of 64 bf16, 128-byte swizzle

// What a head's tokens weigh in this chunk.
struct __align__(16) StSteps {
  float dt[kQ], fh[kQ], fl[kQ];      // step sizes; the sums of log decays F = fh + fl
  float w[kQ];                       // outputs: dt and the decay to the last token of the token's group of 32; sums: to the chunk's last token
};

// A block's part: heads (or 64-column tiles of heads) first .. first + items - 1 of group g.
struct StBlock {
  int g, first, items, row0, t0, n, inner, tiles;
  size_t run;
  __device__ __forceinline__ int head(const ScanArgs& a, int it) const { return g * (a.heads / a.groups) + (first + it) / tiles; }
  __device__ __forceinline__ int column(int it) const { return (first + it) % tiles * 64; }
};
__device__ __forceinline__ bool st_block(const ScanArgs& a, int per_block, StBlock& b) {
  const int entry = blockIdx.z;
  b.row0 = a.q_start[entry];
  const int len = a.q_start[entry + 1] - b.row0;
  b.t0 = blockIdx.y * kQ;
  b.n = min(kQ, len - b.t0);
  b.inner = a.heads * a.P;
  b.tiles = a.P / 64;
  const int of_group = a.heads / a.groups * b.tiles, blocks = (of_group + per_block - 1) / per_block;
  b.g = blockIdx.x / blocks;
  b.first = (blockIdx.x - b.g * blocks) * per_block;
  b.items = min(per_block, of_group - b.first);
  b.run = (size_t)(b.row0 / kQ) + entry + blockIdx.y;
  return b.t0 < len;
}

// exp(F_a - F_b) to the last bits however far the two lie apart: what the difference of the upper parts loses is taken into account (rounded
// at 30 it would be off by a millionth).
__device__ __forceinline__ float st_power(float ah, float al, float bh, float bl) {
  const float d = ah - bh, back = ah - d;
  const float lost = (ah - (d + back)) + (back - bh);
  const float p = expf(d);
  return fmaf(p, lost + (al - bl), p);
}

// The terms of W numbers; an infinity has nothing in the lower two, where it would meet its opposite or a zero.
template <int W>
__device__ __forceinline__ void st_split(const float (&v)[W], uint32_t (&t)[3][W / 2]) {
  float largest = 0.f;
#pragma unroll
  for (int e = 0; e < W; ++e) largest = fmaxf(largest, fabsf(v[e]));
  if (largest < 3e38f) {
#pragma unroll
    for (int e = 0; e < W / 2; ++e) ft_split2(v[2 * e], v[2 * e + 1], t[0][e], t[1][e], t[2][e]);
  } else {
#pragma unroll
    for (int e = 0; e < W / 2; ++e) ft_split2_finite(v[2 * e], v[2 * e + 1], t[0][e], t[1][e], t[2][e]);
  }
}

// A warp fills in the steps of one item: four tokens a lane, F summed in double precision (tokens behind the chunk's: no step, the sum stays).
template <bool SUMS>
__device__ __forceinline__ void st_steps(StSteps& s, const ScanArgs& a, const StBlock& b, int h, int lane) {
  const size_t first = (size_t)(b.row0 + b.t0);
  float dt[4], fh[4], fl[4];
  double f[4];
  const float rate = -expf(a.a_log[h]), bias = a.dt_bias[h];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int t = lane * 4 + k;
    dt[k] = t < b.n ? ss_softplus(ss_load(a.dt, a.dt_dtype, (first + t) * a.ld_dt + a.dt_col + h) + bias) : 0.f;
    const float log_decay = t < b.n ? rate * dt[k] : 0.f;
    f[k] = (double)(log_decay < -1e4f ? -1e4f : log_decay) + (k ? f[k - 1] : 0.0);      // (a decay of zero either way, and no infinity in the sums)
  }
  double up = f[3];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double from = __shfl_up_sync(0xffffffffu, up, o);
    if (lane >= o) up += from;
  }
  const double below = __shfl_up_sync(0xffffffffu, up, 1), before = lane ? below : 0.0;      // (not up - f[3]: a NaN step is not its earlier neighbours')
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double sum = before + f[k];
    fh[k] = (float)sum;
    fl[k] = (float)(sum - (double)fh[k]);
  }
  // (the last token of the group of 32 is the fourth of the group's eighth lane)
  const int from = SUMS ? 31 : lane | 7;
  const float rh = __shfl_sync(0xffffffffu, fh[3], from), rl = __shfl_sync(0xffffffffu, fl[3], from);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int t = lane * 4 + k;
    s.dt[t] = dt[k];
    s.fh[t] = fh[k];
    s.fl[t] = fl[k];
    s.w[t] = (SUMS ? expf((rh - fh[k]) + (rl - fl[k])) : st_power(rh, rl, fh[k], fl[k])) * dt[k];
  }
}

// n rows of WIDTH bf16 (row stride ld) by cp.async into a tile of 128 rows; rows behind them are zeroed.
template <int WIDTH>
__device__ __forceinline__ void st_rows(unsigned char* dst, const __nv_bfloat16* src, int64_t ld, int n) {
#pragma unroll
  for (int p = threadIdx.x; p < kQ * WIDTH / 8; p += kStThreads) {
    const int r = p / (WIDTH / 8), c8 = p % (WIDTH / 8);
    cp_async16(dst + ft_place(r, c8, kQ), src + (r < n ? (size_t)r * ld : 0) + c8 * 8, r < n);
  }
}

// A thread's two pieces of a chunk's x.
struct StX {
  uint4 v[2];
  __device__ __forceinline__ void ask(const __nv_bfloat16* src, int64_t ld, int n) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int p = threadIdx.x + i * kStThreads, r = p >> 3;
      v[i] = r < n ? *reinterpret_cast<const uint4*>(src + (size_t)r * ld + (p & 7) * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
};

template <int N> struct StSums {
  static constexpr uint32_t kB = N / 64 * kStSub, kX = 3 * kStSub;      // B; the weighted x, twice
  static constexpr uint32_t kSmem = 1024 + kB + 2 * kX + 64;
};

// grid (groups * blocks of a group, chunks, entries)
template <int N>
__global__ void __launch_bounds__(kStThreads, 1) ssd_sums_tcgen05_kernel(ScanArgs a, int per_block) {
  using S = StSums<N>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ StSteps steps[kStItems];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  pdl_wait();
  StBlock b;
  if (!st_block(a, per_block, b)) return;
  const uint32_t bar = base + S::kB + 2 * S::kX, xs = base + S::kB;
  const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(a.xbc) + (size_t)(b.row0 + b.t0) * a.ld_xbc;
  st_rows<N>(smem, rows + b.inner + b.g * N, a.ld_xbc, b.n);
  cp_async_commit();
  StX x;
  x.ask(rows + b.head(a, 0) * a.P + b.column(0), a.ld_xbc, b.n);
  const uint32_t tmem = ft_setup(bar, 1, bar + 8, reinterpret_cast<volatile uint32_t*>(smem + (bar + 8 - base)), warp, 512);
  pdl_trigger();
  if (warp < b.items) st_steps<true>(steps[warp], a, b, b.head(a, warp), lane);
  cp_async_wait<0>();
  __syncthreads();
  const auto put = [&](int it) {
    unsigned char* tile = smem + S::kB + (it & 1) * S::kX;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int p = tid + i * kStThreads, r = p >> 3;
      const float w = steps[it].w[r];
      const uint32_t raw[4] = {x.v[i].x, x.v[i].y, x.v[i].z, x.v[i].w};
      float wx[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        wx[2 * e] = __uint_as_float(raw[e] << 16) * w;
        wx[2 * e + 1] = __uint_as_float(raw[e] & 0xffff0000u) * w;
      }
      uint32_t t[3][4];
      st_split(wx, t);
#pragma unroll
      for (int u = 0; u < 3; ++u) *reinterpret_cast<uint4*>(tile + u * kStSub + ft_place(r, p & 7, kQ)) = make_uint4(t[u][0], t[u][1], t[u][2], t[u][3]);
    }
  };
  put(0);
  if (b.items > 1) x.ask(rows + b.head(a, 1) * a.P + b.column(1), a.ld_xbc, b.n);
  const uint32_t leader = warp == 0 ? umma_leader() : 0;
  const int quarter = warp & 3, part = warp >> 2, state_row = quarter * 32 + lane;
  for (int it = 0; it < b.items; ++it) {
    ft_hand_over();
    if (warp == 0) {
      // both operands have the tokens as rows; the small terms side by side (of a state of 64 the upper half of the 128 rows is never stored)
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | (8u << 24);
      const uint32_t tile = xs + (it & 1) * S::kX;
#pragma unroll
      for (int k = 0; k < kQ / 16; ++k) {
        const uint64_t rows_b = umma_desc_mn128(base + k * 2048, kStSub);
        umma_warp(leader, tmem, rows_b, umma_desc_mn128(tile + kStSub + k * 2048, kStSub), idesc | ((128u >> 3) << 17), k != 0);
        umma_warp(leader, tmem + 128 + (k >> 1) * 64, rows_b, umma_desc_mn128(tile + k * 2048, kStSub), idesc | ((64u >> 3) << 17), (k & 1) != 0);
      }
      if (leader) umma_commit(bar);
      __syncwarp();
    }
    if (it + 1 < b.items) put(it + 1);
    if (it + 2 < b.items) x.ask(rows + b.head(a, it + 2) * a.P + b.column(it + 2), a.ld_xbc, b.n);
    ft_wait(bar, it & 1, a.error_word, 0x7C00B1);
    const int h = b.head(a, it);
    float sum[16];
#pragma unroll
    for (int u = 0; u < 3; ++u) {      // (the small terms, then the tokens' fourths)
      uint32_t v[16], w[16];
      tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + u * 128 + part * 16, v);
      tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + u * 128 + 64 + part * 16, w);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const float both = __uint_as_float(v[c]) + __uint_as_float(w[c]);
        sum[c] = u == 0 ? both : sum[c] + both;
      }
    }
    if (N == 128 || state_row < N) {
      float* dst = a.run_state + (b.run * a.heads + h) * (size_t)N * a.P + (size_t)state_row * a.P + b.column(it) + part * 16;
#pragma unroll
      for (int e = 0; e < 16; e += 8) {
        const float o[8] = {sum[e], sum[e + 1], sum[e + 2], sum[e + 3], sum[e + 4], sum[e + 5], sum[e + 6], sum[e + 7]};
        ft_store8(dst + e, o);
      }
    }
    if (b.column(it) == 0 && tid == 0) a.run_decay[b.run * a.heads + h] = expf(steps[it].fh[b.n - 1] + steps[it].fl[b.n - 1]);
  }
  ft_release(warp, tmem, 512);
}

// Shared memory: C; B, whose place the scores take (the ten blocks of 32 x 32 on and below the diagonal); the state's terms; x, twice; the decays
// between tokens of a group of 32; barriers.
template <int N> struct StOuts {
  static constexpr uint32_t kRows = N / 64 * kStSub, kTerm = N * 128, kScores = 10 * 4096;
  static constexpr uint32_t kB = kRows, kState = kB + (kRows > kScores ? kRows : kScores), kX = kState + 3 * kTerm, kNear = kX + 2 * kStSub;
  static constexpr uint32_t kBars = kNear + 4 * 4096, kSmem = 1024 + kBars + 64;
};

template <int N>
__global__ void __launch_bounds__(kStThreads, 1) ssd_outs_tcgen05_kernel(ScanArgs a, int per_block) {
  using S = StOuts<N>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ StSteps steps[kStItems];
  __shared__ int odd[kStItems];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  pdl_wait();
  StBlock b;
  if (!st_block(a, per_block, b)) return;
  const size_t first = (size_t)(b.row0 + b.t0);
  const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(a.xbc) + first * a.ld_xbc;
  st_rows<N>(smem, rows + b.inner + (a.groups + b.g) * N, a.ld_xbc, b.n);
  st_rows<N>(smem + S::kB, rows + b.inner + b.g * N, a.ld_xbc, b.n);
  cp_async_commit();
  constexpr int SV = N * 64 / 8 / kStThreads;      // pieces of eight of the state a thread fetches
  float4 held[SV][2];
  StX x;
  const auto ask = [&](int it) {
    const int h = b.head(a, it), p0 = b.column(it);
    const float* src = a.run_state + (b.run * a.heads + h) * (size_t)N * a.P + p0;
#pragma unroll
    for (int i = 0; i < SV; ++i) {
      const int p = tid + i * kStThreads;
      const float4* from = reinterpret_cast<const float4*>(src + (size_t)(p >> 3) * a.P + (p & 7) * 8);
      held[i][0] = from[0];
      held[i][1] = from[1];
    }
    x.ask(rows + h * a.P + p0, a.ld_xbc, b.n);
  };
  const auto put = [&](int it) {
    unsigned char* tile = smem + S::kState;
#pragma unroll
    for (int i = 0; i < SV; ++i) {
      const int p = tid + i * kStThreads;
      const float v[8] = {held[i][0].x, held[i][0].y, held[i][0].z, held[i][0].w, held[i][1].x, held[i][1].y, held[i][1].z, held[i][1].w};
      uint32_t t[3][4];
      st_split(v, t);
#pragma unroll
      for (int u = 0; u < 3; ++u) *reinterpret_cast<uint4*>(tile + u * S::kTerm + ft_place(p >> 3, p & 7, N)) = make_uint4(t[u][0], t[u][1], t[u][2], t[u][3]);
    }
    // (an infinity or NaN of x must not meet the weight 0 of the tokens before it: it stays out of the product and is added below)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int p = tid + i * kStThreads;
      uint4 keep = x.v[i];
      const uint32_t exponents = 0x7f807f80u, one = 0x00800080u;      // (an exponent of ones carries into the sign's place)
      if ((((keep.x & exponents) + one) | ((keep.y & exponents) + one) | ((keep.z & exponents) + one) | ((keep.w & exponents) + one)) & 0x80008000u) {
        odd[it] = 1;
        keep.x &= ft_finite2(keep.x);
        keep.y &= ft_finite2(keep.y);
        keep.z &= ft_finite2(keep.z);
        keep.w &= ft_finite2(keep.w);
      }
      *reinterpret_cast<uint4*>(smem + S::kX + (it & 1) * kStSub + ft_place(p >> 3, p & 7, kQ)) = keep;
    }
  };
  ask(0);
  if (tid < kStItems) odd[tid] = 0;
  const uint32_t bar = base + S::kBars;
  const uint32_t tmem = ft_setup(bar, 3, bar + 24, reinterpret_cast<volatile uint32_t*>(smem + S::kBars + 24), warp, 512);
  pdl_trigger();
  if (warp < b.items) st_steps<false>(steps[warp], a, b, b.head(a, warp), lane);
  put(0);
  cp_async_wait<0>();
  const uint32_t leader = warp == 0 ? umma_leader() : 0;
  // token i: a lane; the warp's fourth of the tokens before it, then of the columns
  const int quarter = warp & 3, part = warp >> 2, i = quarter * 32 + lane;
  const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
  constexpr int STEPS = N / 16;
  const auto c_at = [&](int k) { return umma_desc_k128(base + (k >> 2) * kStSub + (k & 3) * 32); };
  // Scores, the same for every head of the group: an accumulator for each 16 of the state, four at a time.
  float* scores = reinterpret_cast<float*>(smem + S::kB) + (quarter * (quarter + 1) / 2 + part) * 1024 + lane;      // [token j of its group][lane]
  {
    float s[32];
#pragma unroll
    for (int k0 = 0; k0 < STEPS; k0 += 4) {
      ft_hand_over();
      if (warp == 0) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kQ >> 3) << 17) | (8u << 24);
#pragma unroll
        for (int k = k0; k < k0 + 4; ++k)
          umma_warp(leader, tmem + (k - k0) * 128, c_at(k), umma_desc_k128(base + S::kB + (k >> 2) * kStSub + (k & 3) * 32), idesc, 0);
        if (leader) umma_commit(bar);
        __syncwarp();
      }
      ft_wait(bar, (k0 >> 2) & 1, a.error_word, 0x7C00B2);
      if (part <= quarter) {
#pragma unroll
        for (int k = 0; k < 4; k += 2)
#pragma unroll
          for (int c0 = 0; c0 < 32; c0 += 16) {
            uint32_t v[16], w[16];
            tmem_ld16(tmem + k * 128 + lanes + part * 32 + c0, v);
            tmem_ld16(tmem + k * 128 + 128 + lanes + part * 32 + c0, w);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const float both = __uint_as_float(v[c]) + __uint_as_float(w[c]);
              s[c0 + c] = k0 + k == 0 ? both : s[c0 + c] + both;
            }
          }
      }
    }
    __syncthreads();      // (B is no longer needed)
    if (part <= quarter) {
#pragma unroll
      for (int c = 0; c < 32; ++c) scores[c * 32] = s[c];
    }
  }
  float* near = reinterpret_cast<float*>(smem + S::kNear) + quarter * 1024 + lane;      // [token j][lane]: from j to the lane's token
  // tensor memory from here on: the weighted scores' three terms of 64 columns; one accumulator of 64 columns for small terms and four for the large
  const uint32_t small = tmem + 192, wide = tmem + 256;
  constexpr uint32_t idesc_v = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((64u >> 3) << 17) | (8u << 24);
  for (int it = 0; it < b.items; ++it) {
    ft_hand_over();
    if (warp == 0) {
#pragma unroll
      for (int u = 2; u >= 0; --u)
#pragma unroll
        for (int k = 0; k < STEPS; ++k)
          umma_warp(leader, u == 0 ? wide + k * 4 / STEPS * 64 : small, c_at(k), umma_desc_mn128(base + S::kState + u * S::kTerm + k * 2048, N * 128), idesc_v,
                        u == 0 ? k % (STEPS / 4) != 0 : !(u == 2 && k == 0));
      if (leader) umma_commit(bar + 8);
      __syncwarp();
    }
    const StSteps& st = steps[it];
    if (it + 1 < b.items) ask(it + 1);
    {
      const float ih = st.fh[i], il = st.fl[i];
#pragma unroll
      for (int c = 0; c < 8; c += 4) {      // (each of the four warps of a group of 32 tokens works out the decays from eight of them)
        const int j = quarter * 32 + part * 8 + c;
        const float4 jh = *reinterpret_cast<const float4*>(st.fh + j), jl = *reinterpret_cast<const float4*>(st.fl + j);
        const float4 dt = *reinterpret_cast<const float4*>(st.dt + j);
        float* to = near + (part * 8 + c) * 32;
        to[0] = expf((ih - jh.x) + (il - jl.x)) * dt.x;
        to[32] = expf((ih - jh.y) + (il - jl.y)) * dt.y;
        to[64] = expf((ih - jh.z) + (il - jl.z)) * dt.z;
        to[96] = expf((ih - jh.w) + (il - jl.w)) * dt.w;
      }
      asm volatile("bar.sync %0, 128;\n" ::"r"(1 + quarter) : "memory");
      float s[32];
      if (part < quarter) {
        const int r = part * 32 + 31;
        const float e = st_power(ih, il, st.fh[r], st.fl[r]);
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          const float4 w = *reinterpret_cast<const float4*>(st.w + part * 32 + c);
          s[c] = scores[c * 32] * (e * w.x);
          s[c + 1] = scores[c * 32 + 32] * (e * w.y);
          s[c + 2] = scores[c * 32 + 64] * (e * w.z);
          s[c + 3] = scores[c * 32 + 96] * (e * w.w);
        }
      } else if (part == quarter) {
#pragma unroll
        for (int c = 0; c < 32; ++c) s[c] = c <= lane ? scores[c * 32] * near[c * 32] : 0.f;
      }
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += 16) {
        uint32_t t[3][8] = {};
        if (part <= quarter) {
          float half[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) half[c] = s[c0 + c];
          st_split(half, t);
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 3; ++u) ft_tmem_st8(tmem + lanes + u * 64 + part * 16 + c0 / 2, t[u]);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
    }
    ft_wait(bar + 8, it & 1, a.error_word, 0x7C00B3);
    float sum[16];
    const auto add_up = [&](float (&sum)[16]) {      // the five accumulators of the warp's columns, small terms first
#pragma unroll
      for (int e = 0; e < 16; e += 8) {
        uint32_t v[5][8];
        tmem_ld8(small + lanes + part * 16 + e, v[0]);
#pragma unroll
        for (int q = 0; q < 4; ++q) tmem_ld8(wide + q * 64 + lanes + part * 16 + e, v[q + 1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
          const auto pair = [&](int q) { return f2_pack(__uint_as_float(v[q][c]), __uint_as_float(v[q][c + 1])); };
          f2_unpack(f2_add(f2_add(f2_add(pair(1), pair(2)), f2_add(pair(3), pair(4))), pair(0)), sum[e + c], sum[e + c + 1]);
        }
      }
    };
    add_up(sum);
    {
      const float decay = expf(st.fh[i] + st.fl[i]);
#pragma unroll
      for (int c = 0; c < 16; ++c) sum[c] *= decay;
    }
    ft_hand_over();
    const uint32_t tile = S::kX + (it & 1) * kStSub;
    if (warp == 0) {
      // (the weighted scores: tensor memory, 64 columns a term)
#pragma unroll
      for (int u = 2; u >= 0; --u)
#pragma unroll
        for (int k = 0; k < kQ / 16; ++k) {
          const uint32_t to = u == 0 ? wide + k / 2 * 64 : small;
          umma_warp_tmem(leader, to, tmem + u * 64 + k * 8, umma_desc_mn128(base + tile + k * 2048, kStSub), idesc_v, u == 0 ? k % 2 != 0 : !(u == 2 && k == 0));
        }
      if (leader) umma_commit(bar + 16);
      __syncwarp();
    }
    if (it + 1 < b.items) put(it + 1);
    ft_wait(bar + 16, it & 1, a.error_word, 0x7C00B4);
    {
      float own[16];
      add_up(own);
#pragma unroll
      for (int c = 0; c < 16; ++c) sum[c] += own[c];
    }
    const int h = b.head(a, it);
    const float skip = a.d_skip[h];
    float* dst = a.y + (first + i) * b.inner + h * a.P + b.column(it) + part * 16;
    if (i < b.n) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint4 raw = *reinterpret_cast<const uint4*>(smem + tile + ft_place(i, part * 2 + e, kQ));
        const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
        float o[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          o[2 * c] = fmaf(skip, __uint_as_float(r[c] << 16), sum[8 * e + 2 * c]);
          o[2 * c + 1] = fmaf(skip, __uint_as_float(r[c] & 0xffff0000u), sum[8 * e + 2 * c + 1]);
        }
        ft_store8(dst + 8 * e, o);
      }
    }
    __syncwarp();
    if (odd[it]) {      // what stayed out, from its own token on
      const __nv_bfloat16* all = rows + h * a.P + b.column(it) + part * 16;
#pragma unroll 1
      for (int j = 0; j < b.n; ++j) {
        uint32_t term[3];
#pragma unroll
        for (int u = 0; u < 3; ++u)
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(term[u]) : "r"(tmem + lanes + u * 64 + (j >> 1)));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        float w = 0.f;
#pragma unroll
        for (int u = 2; u >= 0; --u) w += __uint_as_float(j & 1 ? term[u] & 0xffff0000u : term[u] << 16);
        if (i >= j && i < b.n)
          for (int c = 0; c < 16; ++c) {
            const float v = __bfloat162float(all[(size_t)j * a.ld_xbc + c]);
            if (!isfinite(v)) dst[c] = fmaf(w, v, i == j ? fmaf(skip, v, dst[c]) : dst[c]);
          }
        __syncwarp();
      }
    }
  }
  ft_release(warp, tmem, 512);
}

template <int N>
static int launch_ssd_tcgen05(const ScanArgs& a, int n_entries, int n_tokens, int max_q_len, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(ssd_sums_tcgen05_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)StSums<N>::kSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(ssd_outs_tcgen05_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)StOuts<N>::kSmem);
  if (e != cudaSuccess) return (int)e;
  // Heads a block takes one after the other: whole rounds of blocks over the SMs times a block's heads and a start of one and a half.  (80 heads of
  // 64 in four groups, 2,600 tokens: 12 heads a block, in two rounds, 413 us, 4 heads in three 356.)  Chunks: half a one more a request than the
  // tokens fill.
  const int of_group = a.heads / a.groups * (a.P / 64), chunks = n_tokens / kQ + (n_entries + 1) / 2;
  int per_block = 1;
  double least = 1e30;
  for (int p = 1; p <= kStItems && p <= of_group; ++p) {
    const double cost = (double)ceil_div64((int64_t)a.groups * ceil_div(of_group, p) * chunks, 148) * (p + 1.5);
    if (cost < least) {
      least = cost;
      per_block = p;
    }
  }
  const dim3 grid(a.groups * ceil_div(of_group, per_block), ceil_div(max_q_len, kQ), n_entries);
  TIB_LAUNCH_DEPENDENT(ssd_sums_tcgen05_kernel<N>, grid, kStThreads, StSums<N>::kSmem, stream, a, per_block);
  const int status = ssd_fold(a, n_entries, stream);
  if (status != TIB_OK) return status;
  TIB_LAUNCH_DEPENDENT(ssd_outs_tcgen05_kernel<N>, grid, kStThreads, StOuts<N>::kSmem, stream, a, per_block);
  return TIB_OK;
}

int ssd_tcgen05(const ScanArgs& a, int n_entries, int n_tokens, int max_q_len, cudaStream_t stream) {
  return a.N == 128 ? launch_ssd_tcgen05<128>(a, n_entries, n_tokens, max_q_len, stream) : launch_ssd_tcgen05<64>(a, n_entries, n_tokens, max_q_len, stream);
}

}  // namespace tib
