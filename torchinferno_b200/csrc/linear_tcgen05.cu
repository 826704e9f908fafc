// The two kernels of the decayed linear attention's runs that multiply, on the tensor cores in 32 bits.  For the n <= 128 tokens of a run
//     L        = sum_j lambda^(n-1-j) k_j v_j^T                                                          lin_run_sums
//     o_i      = lambda^(i+1) S^T q_i + sum_(j<=i) (q_i . k_j) lambda^(i-j) v_j       (S: state at its start)   lin_run_outs
// q, k and v are fp32 numbers (activated), as are S and the weighted scores: each is three bf16 terms, and the six products of terms above
// 2^-24 of the whole are made (split_terms.cuh).  The tensor core cuts its sums off, so the largest group of products is shared out over
// several accumulators (L: four or eight, an instruction or two of 16 k each; else two); the small groups come first in the last one.
//
// A block owns a run, a head and 64 or 128 value columns; its 512 threads load, activate and split, warp 0 issues the products:
//     q, k -> shared memory        scores = q k^T                       (S is fetched meanwhile)
//     S -> k's place               carried = q S                        (scores are weighed, split and put back into tensor memory meanwhile)
//     v -> q's place               inside = scores v                    (carried is read and scaled before)
// One launch a run and head keeps no chain between runs but the fold's.  A value that is not finite would meet the weight 0 of the tokens
// before it: it stays out of the product and is added to its own column from its own token on.  Any other infinity, and a number that rounds to
// one in bf16, makes NaN of what it meets in three terms: a sum or output that is not finite is made again by multiply-adds in order.
//
// What bounds it: the threads' activations and conversions (27 instructions an element) between the products, with one block of 16 warps an SM (192 KB
// of terms): issue slots a third full, tensor cores 17 and 25 %.  Blocks of 8 warps took 117 us in all where these take 68.  Figures: linear_attention.cu.
#include "linear_attention.cuh"
#include "split_terms.cuh"

namespace tib {

constexpr int kLtThreads = 512;
constexpr uint32_t kLtSub = kLinRun * 128;      // 128 rows of 64 bf16, 128-byte swizzle

// A tile's terms: [3][width / 64][rows][64].
__device__ __forceinline__ void lt_put(unsigned char* tile, uint32_t term_bytes, uint32_t at, const float (&x)[8]) {
  uint32_t t[3][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) ft_split2(x[2 * e], x[2 * e + 1], t[0][e], t[1][e], t[2][e]);
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(tile + p * term_bytes + at) = make_uint4(t[p][0], t[p][1], t[p][2], t[p][3]);
}

// The activation, with the reciprocal to a unit in the last place (an IEEE division is a third of these kernels' instructions; a Newton step
// behind it changes nothing in the outputs' error).  Below -87.3 it is zero instead of less than 1.1e-36.
__device__ __forceinline__ float lt_act(float z, int activation) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + expf(-z)));
  return activation ? z * r : z;
}

// Eight elements of a row as they lie in memory, and activated.
template <typename T> struct LtRaw;
template <> struct LtRaw<__nv_bfloat16> {
  uint4 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void zero() { v = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ void activated(int activation, float (&x)[8]) const {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[2 * i] = lt_act(__uint_as_float(w[i] << 16), activation);
      x[2 * i + 1] = lt_act(__uint_as_float(w[i] & 0xffff0000u), activation);
    }
  }
};
template <> struct LtRaw<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) {
    a = reinterpret_cast<const float4*>(p)[0];
    b = reinterpret_cast<const float4*>(p)[1];
  }
  __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void activated(int activation, float (&x)[8]) const {
    const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = lt_act(w[i], activation);
  }
};

// A thread's pieces of n rows of WIDTH columns (zeros behind them): all asked for first, then activated, changed by f(row, values) and left as terms.
template <typename T, int WIDTH> struct LtRows {
  static constexpr int kPieces = kLinRun * WIDTH / 8 / kLtThreads;
  LtRaw<T> raw[kPieces];
  __device__ __forceinline__ void ask(const T* src, int64_t ld, int n) {
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
      const int p = threadIdx.x + i * kLtThreads, r = p / (WIDTH / 8), c8 = p % (WIDTH / 8);
      if (r < n) raw[i].load(src + (size_t)r * ld + c8 * 8);
      else raw[i].zero();
    }
  }
  template <typename F> __device__ __forceinline__ void put(unsigned char* tile, int activation, F f) {
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
      const int p = threadIdx.x + i * kLtThreads, r = p / (WIDTH / 8), c8 = p % (WIDTH / 8);
      float x[8];
      raw[i].activated(activation, x);
      f(r, x);
      lt_put(tile, WIDTH / 64 * kLtSub, ft_place(r, c8, kLinRun), x);
    }
  }
};

// The six products of terms over STEPS instructions of 16 k into ACC accumulators of `columns` columns: the last takes the small groups first,
// and each its share of the largest; a(p, k) and b(p, k) describe term p at step k.
template <int STEPS, int ACC, typename A, typename B>
__device__ __forceinline__ void lt_products(uint32_t leader, uint32_t d, uint32_t columns, uint32_t idesc, A a, B b) {
  const uint32_t last = d + (ACC - 1) * columns;
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    umma_warp(leader, last, a(0, k), b(2, k), idesc, k != 0);
    umma_warp(leader, last, a(1, k), b(1, k), idesc, 1);
    umma_warp(leader, last, a(2, k), b(0, k), idesc, 1);
  }
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    umma_warp(leader, last, a(0, k), b(1, k), idesc, 1);
    umma_warp(leader, last, a(1, k), b(0, k), idesc, 1);
  }
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    const int share = k * ACC / STEPS;
    umma_warp(leader, d + share * columns, a(0, k), b(0, k), idesc, share == ACC - 1 || k % (STEPS / ACC) != 0);
  }
}

// What the two kernels' blocks begin with; false: the block has no run.
struct LtBlock {
  int head, own, col0, row0, t0, n;
  size_t run;
};
template <int TV>
__device__ __forceinline__ bool lt_block(const LinRunArgs& a, LtBlock& b) {
  const int tiles = a.value_dim / TV, entry = blockIdx.z;
  b.own = blockIdx.x / tiles;
  b.head = a.head0 + b.own;
  b.col0 = (blockIdx.x - b.own * tiles) * TV;
  b.row0 = a.q_start[entry];
  const int len = a.q_start[entry + 1] - b.row0;
  b.t0 = blockIdx.y * kLinRun;
  b.n = min(kLinRun, len - b.t0);
  b.run = lin_first_run(b.row0, entry) + blockIdx.y;
  return b.t0 < len && len >= a.shortest;
}
template <int D, int TV, int ACC> struct LtSums {
  static constexpr uint32_t kKeyTerm = D / 64 * kLtSub, kValueTerm = TV / 64 * kLtSub;
  static constexpr uint32_t kSmem = 1024 + 3 * (kKeyTerm + kValueTerm) + 64;
  static constexpr uint32_t kColumns = ACC * TV;
};

// An element of L by multiply-adds: k and v at the run's first token.
template <typename T>
__device__ __noinline__ float lt_plain_sum(const T* k, int64_t ldk, const T* v, int64_t ldv, const float* pw, int n, int activation) {
  float s = 0.f;
  for (int j = 0; j < n && s == s; ++j)
    s = fmaf(pw[n - 1 - j] * lt_act(to_f32(k[(size_t)j * ldk]), activation), lt_act(to_f32(v[(size_t)j * ldv]), activation), s);
  return s;
}

// grid (heads * column tiles, runs, entries).  How many accumulators there are is the value heads' width's alone, not the tile's, which the step
// chooses: a request's bits do not depend on its neighbours.
template <typename T, int D, int TV, int ACC>
__global__ void __launch_bounds__(kLtThreads, 1) lin_run_sums_kernel(const T* __restrict__ k, const T* __restrict__ v, LinRunArgs a) {
  using S = LtSums<D, TV, ACC>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ float pw[kLinRun + 1];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  pdl_wait();
  LtBlock b;
  if (!lt_block<TV>(a, b)) return;
  const uint32_t bar = base + 3 * (S::kKeyTerm + S::kValueTerm);
  if (threadIdx.x <= kLinRun) pw[threadIdx.x] = a.powers[b.head * (kLinRun + 1) + threadIdx.x];
  const uint32_t tmem = ft_setup(bar, 1, bar + 8, reinterpret_cast<volatile uint32_t*>(smem + (bar + 8 - base)), warp, S::kColumns);
  pdl_trigger();
  const size_t first = (size_t)(b.row0 + b.t0);
  LtRows<T, D> keys_of;
  LtRows<T, TV> values_of;
  keys_of.ask(k + first * a.ldk + b.head * D, a.ldk, b.n);
  values_of.ask(v + first * a.ldv + b.head * a.value_dim + b.col0, a.ldv, b.n);
  keys_of.put(smem, a.activation, [&](int r, float (&x)[8]) {
    const float w = pw[max(b.n - 1 - r, 0)];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] *= w;
  });
  values_of.put(smem + 3 * S::kKeyTerm, a.activation, [](int, float (&)[8]) {});
  ft_hand_over();
  if (warp == 0) {
    const uint32_t leader = umma_leader();
    // both operands have the tokens as rows (of heads of 64 the upper half of the 128 rows is the next tile's, and never stored)
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(TV >> 3) << 17) | (8u << 24);
    const uint32_t keys = base, values = base + 3 * S::kKeyTerm;
    lt_products<kLinRun / 16, ACC>(leader, tmem, TV, idesc, [&](int p, int s) { return umma_low_mn128(keys + p * S::kKeyTerm + s * 2048, kLtSub); },
                              [&](int p, int s) { return umma_low_mn128(values + p * S::kValueTerm + s * 2048, kLtSub); });
    if (leader) umma_commit(bar);
    __syncwarp();
  }
  ft_wait(bar, 0, a.error_word, 0x7C00A1);
  const int quarter = warp & 3, part = warp >> 2, d = quarter * 32 + lane;
  const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + part * (TV / 4);
  float* dst = a.run_state + (b.run * a.n_heads + b.own) * (size_t)D * a.value_dim + (size_t)d * a.value_dim + b.col0 + part * (TV / 4);
  uint32_t again = 0;      // columns to be made again
#pragma unroll
  for (int c0 = 0; c0 < TV / 4; c0 += 16) {
    float sum[16];
#pragma unroll
    for (int i = 0; i < ACC; i += 2) {
      uint32_t x[16], y[16];
      tmem_ld16(at + i * TV + c0, x);
      tmem_ld16(at + (i + 1) * TV + c0, y);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float both = __uint_as_float(x[e]) + __uint_as_float(y[e]);
        sum[e] = i == 0 ? both : sum[e] + both;
      }
    }
    if (D < 128 && d >= D) continue;
#pragma unroll
    for (int e = 0; e < 16; ++e) again |= isfinite(sum[e]) ? 0u : 1u << (c0 + e);
#pragma unroll
    for (int e = 0; e < 16; e += 8) {
      const float o[8] = {sum[e], sum[e + 1], sum[e + 2], sum[e + 3], sum[e + 4], sum[e + 5], sum[e + 6], sum[e + 7]};
      ft_store8(dst + c0 + e, o);
    }
  }
  for (; again; again &= again - 1) {
    const int c = __ffs(again) - 1;
    dst[c] = lt_plain_sum(k + first * a.ldk + b.head * D + d, a.ldk, v + first * a.ldv + b.head * a.value_dim + b.col0 + part * (TV / 4) + c, a.ldv, pw, b.n,
                          a.activation);
  }
  ft_release(warp, tmem, S::kColumns);
}

template <int D, int TV> struct LtOuts {
  static constexpr uint32_t kKeyTerm = D / 64 * kLtSub, kValueTerm = TV / 64 * kLtSub, kStateTerm = TV / 64 * D * 128;
  static constexpr uint32_t kFirst = 3 * (kKeyTerm > kValueTerm ? kKeyTerm : kValueTerm);      // q, then v
  static constexpr uint32_t kSecond = 3 * (kKeyTerm > kStateTerm ? kKeyTerm : kStateTerm);     // k, then S
  static constexpr uint32_t kSmem = 1024 + kFirst + kSecond + 64;
};

// The columns `again` of token i's outputs by multiply-adds: query is its own row, k and v lie at the run's first token, v, state and dst at the
// thread's columns.
template <typename T, int D>
__device__ __noinline__ void lt_plain_outs(uint32_t again, int i, const T* query, const T* k, int64_t ldk, const T* v, int64_t ldv, const float* state,
                                           int value_dim, float* dst, const float* pw, int activation) {
  for (uint32_t left = again; left; left &= left - 1) {
    const int c = __ffs(left) - 1;
    float s = 0.f;
    for (int d = 0; d < D && s == s; ++d) s = fmaf(state[(size_t)d * value_dim + c], lt_act(to_f32(query[d]), activation), s);
    dst[c] = s * pw[i + 1];
  }
  for (int j = 0; j <= i && again; ++j) {
    float w = 0.f;
    for (int d = 0; d < D && w == w; ++d) w = fmaf(lt_act(to_f32(query[d]), activation), lt_act(to_f32(k[(size_t)j * ldk + d]), activation), w);
    w *= pw[i - j];
    for (uint32_t left = again; left; left &= left - 1) {
      const int c = __ffs(left) - 1;
      const float s = fmaf(w, lt_act(to_f32(v[(size_t)j * ldv + c]), activation), dst[c]);
      dst[c] = s;
      if (s != s) again ^= 1u << c;      // (it stays NaN)
    }
  }
}

template <typename T, int D, int TV>
__global__ void __launch_bounds__(kLtThreads, 1) lin_run_outs_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, LinRunArgs a) {
  using S = LtOuts<D, TV>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ float pw[kLinRun + 1];
  __shared__ int odd;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  pdl_wait();
  LtBlock b;
  if (!lt_block<TV>(a, b)) return;
  const uint32_t bar = base + S::kFirst + S::kSecond;
  if (tid <= kLinRun) pw[tid] = a.powers[b.head * (kLinRun + 1) + tid];
  if (tid == 0) odd = 0;
  // tensor memory: scores (two accumulators), later their three terms; carried, later inside
  const uint32_t tmem = ft_setup(bar, 3, bar + 24, reinterpret_cast<volatile uint32_t*>(smem + (bar + 24 - base)), warp, 512);
  pdl_trigger();
  const size_t first = (size_t)(b.row0 + b.t0);
  const uint32_t one = base, two = base + S::kFirst;
  {
    LtRows<T, D> rows_q, rows_k;
    rows_q.ask(q + first * a.ldq + b.head * D, a.ldq, b.n);
    rows_k.ask(k + first * a.ldk + b.head * D, a.ldk, b.n);
    rows_q.put(smem, a.activation, [](int, float (&)[8]) {});
    rows_k.put(smem + S::kFirst, a.activation, [](int, float (&)[8]) {});
  }
  ft_hand_over();
  const uint32_t leader = warp == 0 ? umma_leader() : 0;
  if (warp == 0) {
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kLinRun >> 3) << 17) | (8u << 24);
    const auto at = [](uint32_t tile, int p, int s) { return umma_low_k128(tile + p * S::kKeyTerm + (s >> 2) * kLtSub + (s & 3) * 32); };
    lt_products<D / 16, 2>(leader, tmem, 128, idesc, [&](int p, int s) { return at(one, p, s); }, [&](int p, int s) { return at(two, p, s); });
    if (leader) umma_commit(bar);
    __syncwarp();
  }
  constexpr int SV = D * TV / 8 / kLtThreads;      // pieces of eight of S a thread fetches
  const float* state = a.run_state + (b.run * a.n_heads + b.own) * (size_t)D * a.value_dim + b.col0;
  float4 held[SV][2];
#pragma unroll
  for (int i = 0; i < SV; ++i) {
    const int p = tid + i * kLtThreads;
    const float4* src = reinterpret_cast<const float4*>(state + (size_t)(p / (TV / 8)) * a.value_dim + (p % (TV / 8)) * 8);
    held[i][0] = src[0];
    held[i][1] = src[1];
  }
  ft_wait(bar, 0, a.error_word, 0x7C00A2);
#pragma unroll
  for (int i = 0; i < SV; ++i) {
    const int p = tid + i * kLtThreads;
    const float x[8] = {held[i][0].x, held[i][0].y, held[i][0].z, held[i][0].w, held[i][1].x, held[i][1].y, held[i][1].z, held[i][1].w};
    lt_put(smem + S::kFirst, S::kStateTerm, ft_place(p / (TV / 8), p % (TV / 8), D), x);
  }
  ft_hand_over();
  const uint32_t carried = tmem + 256;
  constexpr uint32_t idesc_v = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(TV >> 3) << 17) | (8u << 24);
  if (warp == 0) {
    lt_products<D / 16, 2>(leader, carried, TV, idesc_v,
                        [&](int p, int s) { return umma_low_k128(one + p * S::kKeyTerm + (s >> 2) * kLtSub + (s & 3) * 32); },
                        [&](int p, int s) { return umma_low_mn128(two + p * S::kStateTerm + s * 2048, D * 128); });
    if (leader) umma_commit(bar + 8);
    __syncwarp();
  }
  const T* values = v + first * a.ldv + b.head * a.value_dim + b.col0;
  LtRows<T, TV> rows_v;
  rows_v.ask(values, a.ldv, b.n);
  // token i: a lane; the warp's fourth of the tokens before it, then of the columns
  const int quarter = warp & 3, part = warp >> 2, i = quarter * 32 + lane;
  const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
  {
    float s[32];
#pragma unroll
    for (int c0 = 0; c0 < 32; c0 += 16) {
      uint32_t x[16], y[16];
      tmem_ld16(tmem + lanes + part * 32 + c0, x);
      tmem_ld16(tmem + lanes + 128 + part * 32 + c0, y);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
      for (int c = 0; c < 16; ++c) s[c0 + c] = __uint_as_float(x[c]) + __uint_as_float(y[c]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    asm volatile("bar.sync %0, 128;\n" ::"r"(1 + quarter) : "memory");      // (all four warps of these lanes have read them)
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
    for (int c0 = 0; c0 < 32; c0 += 16) {
      uint32_t t[3][8];
#pragma unroll
      for (int c = 0; c < 16; c += 2) {
        const int back = i - (part * 32 + c0 + c);
        const float w0 = back >= 0 ? s[c0 + c] * pw[max(back, 0)] : 0.f, w1 = back >= 1 ? s[c0 + c + 1] * pw[max(back - 1, 0)] : 0.f;
        ft_split2(w0, w1, t[0][c / 2], t[1][c / 2], t[2][c / 2]);
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) ft_tmem_st8(tmem + lanes + p * 64 + part * 16 + c0 / 2, t[p]);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
  }
  ft_wait(bar + 8, 0, a.error_word, 0x7C00A3);
  float sum[TV / 4];
  const float decay = pw[i + 1];
#pragma unroll
  for (int c0 = 0; c0 < TV / 4; c0 += 16) {
    uint32_t x[16], y[16];
    tmem_ld16(carried + lanes + part * (TV / 4) + c0, x);
    tmem_ld16(carried + TV + lanes + part * (TV / 4) + c0, y);
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int c = 0; c < 16; ++c) sum[c0 + c] = (__uint_as_float(x[c]) + __uint_as_float(y[c])) * decay;
  }
  rows_v.put(smem, a.activation, [&](int, float (&x)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (!isfinite(x[e])) {
        odd = 1;
        x[e] = 0.f;
      }
  });
  ft_hand_over();
  if (warp == 0) {
    // (the weighted scores: tensor memory, 64 columns a term)
    const auto b_at = [&](int p, int s) { return umma_low_mn128(one + p * S::kValueTerm + s * 2048, kLtSub); };
    const uint32_t d0 = carried, d1 = carried + TV;
#pragma unroll
    for (int s = 0; s < kLinRun / 16; ++s) {
      umma_warp_tmem(leader, d1, tmem + s * 8, b_at(2, s), idesc_v, s != 0);
      umma_warp_tmem(leader, d1, tmem + 64 + s * 8, b_at(1, s), idesc_v, 1);
      umma_warp_tmem(leader, d1, tmem + 128 + s * 8, b_at(0, s), idesc_v, 1);
    }
#pragma unroll
    for (int s = 0; s < kLinRun / 16; ++s) {
      umma_warp_tmem(leader, d1, tmem + s * 8, b_at(1, s), idesc_v, 1);
      umma_warp_tmem(leader, d1, tmem + 64 + s * 8, b_at(0, s), idesc_v, 1);
    }
#pragma unroll
    for (int s = 0; s < kLinRun / 16; ++s) umma_warp_tmem(leader, s < kLinRun / 32 ? d0 : d1, tmem + s * 8, b_at(0, s), idesc_v, s != 0);
    if (leader) umma_commit(bar + 16);
    __syncwarp();
  }
  ft_wait(bar + 16, 0, a.error_word, 0x7C00A4);
#pragma unroll
  for (int c0 = 0; c0 < TV / 4; c0 += 16) {
    uint32_t x[16], y[16];
    tmem_ld16(carried + lanes + part * (TV / 4) + c0, x);
    tmem_ld16(carried + TV + lanes + part * (TV / 4) + c0, y);
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int c = 0; c < 16; ++c) sum[c0 + c] += __uint_as_float(x[c]) + __uint_as_float(y[c]);
  }
  uint32_t again = 0;      // columns to be made again
#pragma unroll
  for (int c = 0; c < TV / 4; ++c) again |= isfinite(sum[c]) ? 0u : 1u << c;
  float* dst = a.out + (first + i) * a.heads * a.value_dim + b.head * a.value_dim + b.col0 + part * (TV / 4);
  if (i < b.n) {
#pragma unroll
    for (int c0 = 0; c0 < TV / 4; c0 += 8) {
      const float o[8] = {sum[c0], sum[c0 + 1], sum[c0 + 2], sum[c0 + 3], sum[c0 + 4], sum[c0 + 5], sum[c0 + 6], sum[c0 + 7]};
      ft_store8(dst + c0, o);
    }
  }
  __syncwarp();
  if (odd) {      // what stayed out, from its own token on
#pragma unroll 1
    for (int j = 0; j < b.n; ++j) {
      uint32_t term[3];
#pragma unroll
      for (int p = 0; p < 3; ++p)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(term[p]) : "r"(tmem + lanes + p * 64 + (j >> 1)));
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      float w = 0.f;
#pragma unroll
      for (int p = 2; p >= 0; --p) w += __uint_as_float(j & 1 ? term[p] & 0xffff0000u : term[p] << 16);
      if (i >= j && i < b.n)
        for (int c = 0; c < TV / 4; ++c) {
          const float x = lt_act(to_f32(values[(size_t)j * a.ldv + part * (TV / 4) + c]), a.activation);
          if (!isfinite(x)) dst[c] = fmaf(w, x, dst[c]);
        }
      __syncwarp();
    }
  }
  if (again && i < b.n)
    lt_plain_outs<T, D>(again, i, q + (first + i) * a.ldq + b.head * D, k + first * a.ldk + b.head * D, a.ldk, values + part * (TV / 4), a.ldv,
                        state + part * (TV / 4), a.value_dim, dst, pw, a.activation);
  ft_release(warp, tmem, 512);
}

template <typename T, int D, int TV, int ACC>
static int lt_run_sums(const void* k, const void* v, const LinRunArgs& a, dim3 grid, cudaStream_t stream) {
  auto kern = lin_run_sums_kernel<T, D, TV, ACC>;
  constexpr int smem = LtSums<D, TV, ACC>::kSmem;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  TIB_LAUNCH_DEPENDENT(kern, grid, kLtThreads, smem, stream, (const T*)k, (const T*)v, a);
  return TIB_OK;
}
template <typename T, int D, int TV>
static int lt_go_sums(const void* k, const void* v, const LinRunArgs& a, dim3 grid, cudaStream_t stream) {
  if constexpr (TV == 64) {
    if (a.value_dim % 128 != 0) return lt_run_sums<T, D, 64, 8>(k, v, a, grid, stream);
  }
  return lt_run_sums<T, D, TV, 4>(k, v, a, grid, stream);
}
template <typename T, int D, int TV>
static int lt_go_outs(const void* q, const void* k, const void* v, const LinRunArgs& a, dim3 grid, cudaStream_t stream) {
  auto kern = lin_run_outs_kernel<T, D, TV>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LtOuts<D, TV>::kSmem);
  if (e != cudaSuccess) return (int)e;
  TIB_LAUNCH_DEPENDENT(kern, grid, kLtThreads, (LtOuts<D, TV>::kSmem), stream, (const T*)q, (const T*)k, (const T*)v, a);
  return TIB_OK;
}

#define TIB_LT_PICK(T, go, ...)                                                             \
  (key_dim == 64 ? (tile == 64 ? go<T, 64, 64>(__VA_ARGS__) : go<T, 64, 128>(__VA_ARGS__))   \
                 : (tile == 64 ? go<T, 128, 64>(__VA_ARGS__) : go<T, 128, 128>(__VA_ARGS__)))

int launch_lin_run_sums(const void* k, const void* v, const LinRunArgs& a, int dtype, int key_dim, int tile, dim3 grid, cudaStream_t stream) {
  return dtype == TIB_F32 ? TIB_LT_PICK(float, lt_go_sums, k, v, a, grid, stream) : TIB_LT_PICK(__nv_bfloat16, lt_go_sums, k, v, a, grid, stream);
}
int launch_lin_run_outs(const void* q, const void* k, const void* v, const LinRunArgs& a, int dtype, int key_dim, int tile, dim3 grid, cudaStream_t stream) {
  return dtype == TIB_F32 ? TIB_LT_PICK(float, lt_go_outs, q, k, v, a, grid, stream) : TIB_LT_PICK(__nv_bfloat16, lt_go_outs, q, k, v, a, grid, stream);
}
#undef TIB_LT_PICK

}  // namespace tib
