// Prompt portions of the attention over a low-rank latent, with per-head keys and values made for the step.
//
// The cache holds one row per token: the normed latent c (rank wide) and the rotated key part r all heads share.  For single tokens
// the folded form (latent_attention.cu) reads that row once for all heads.  A prompt pays for it: every head multiplies keys of
// rank + rot and values of rank numbers.  Here the step's keys and values are made once from the cached rows,
//     K_j = W_uk_j c,   V_j = W_uv_j c        (one library product over some or all heads, [keys, heads * (dim + value_dim)])
// and attention runs at its own head sizes, a quarter of the products at rank 512, heads of 128 and 64 rotated.
//
//   latent_gather    the cached rows of every entry, dense: latents [rows, rank] and rotated parts [rows, rot]; an entry's rows
//                    start at a multiple of 128 and are padded with zeros to one, so that a tile of keys is one entry's
//   latent_prefill   a block owns 128 tokens of one head and walks its keys in tiles of 128 up to the causal edge, as
//                    attention_tcgen05.cu does (its softmax halves, slack and merge at the end); what differs: the score is a
//                    product over dim + rot (Q and K in sub-tiles of 64, the last one from the shared rotated parts), and the
//                    weights enter the second product as two bf16 terms (high part and remainder: 16 bits), which together fill
//                    the columns of S they come from.  A head's sink and the output gate are applied at the end.
//
// What bounds it: the tensor core (two products, the second twice) at two stages of 80 KB of keys and values.  Two prompts of 1,667
// and 833 tokens, 16 heads of 128 + 64 over a rank of 512: gather 3 us, product 14, attention 45, where the folded form took 20 for
// folding, 1,094 for the attention, 21 for a cast, 12 for unfolding and 20 for the gate.
#include "tcgen05.cuh"
#include <math_constants.h>

namespace tib {

constexpr int kLpTile = 128;                        // tokens of a block, keys of a tile
constexpr int kLpWarps = 8;                         // softmax warps: two threads per row, 64 keys each
constexpr int kLpThreads = 64 + 32 * kLpWarps + 32;
constexpr int kLpValueWarp = 2 + kLpWarps;
constexpr int kLpStages = 2;
constexpr float kLpSlack = 8.f;
constexpr uint32_t kLpSub = kLpTile * 64 * 2;       // bytes of a [128][64] sub-tile

struct LpArgs {
  const int* q_start;
  const int* kv_start;
  const float* sink;               // [heads] or null
  const __nv_bfloat16* gate;       // rows of heads or heads * value_dim numbers, or null
  int64_t ld_gate;
  int gate_per_head;
  __nv_bfloat16* out;              // [tokens, heads, value_dim]
  int heads, dim, head0;           // head0: the first of the launch's heads
  int shortest;                    // shorter portions are left alone
  float scale_log2;
  int* error_word;
};

// First dense row of an entry's keys: the padded lengths of the entries before it.  Called by a whole warp.
__device__ __forceinline__ int lp_first_row(const int* q_start, const int* kv_start, int entry, int lane) {
  int sum = 0;
  for (int e = lane; e < entry; e += 32) sum += (kv_start[e] + q_start[e + 1] - q_start[e] + kLpTile - 1) / kLpTile * kLpTile;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum;
}

// grid (runs of eight rows, entries), 256 threads: 16 bytes a lane, a warp a row (longer runs of rows a block, four rows a warp one after the other:
// 12 us where this takes 3.1 on the call of the header).
constexpr int kGatherRows = 8;
__global__ void __launch_bounds__(256)
latent_gather_kernel(const uint4* __restrict__ pool, int64_t page_stride, int page_size, int num_pages, const int* __restrict__ block_table,
                     int table_stride, const int* __restrict__ q_start, const int* __restrict__ kv_start, const int* __restrict__ slots,
                     uint4* __restrict__ latent, uint4* __restrict__ rotated, int rows, int rank8, int rot8, int* __restrict__ error_word) {
  pdl_wait();
  pdl_trigger();
  const int entry = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * kGatherRows + warp, slot = slots[entry];
  const int keys = kv_start[entry] + q_start[entry + 1] - q_start[entry];
  const int padded = (keys + kLpTile - 1) / kLpTile * kLpTile;
  if (r >= padded) return;
  const int page = r < keys ? block_table[(size_t)slot * table_stride + r / page_size] : -1;
  const int first = lp_first_row(q_start, kv_start, entry, lane);
  const int pieces = rank8 + rot8;
  const bool have = page >= 0 && page < num_pages;
  if (r < keys && !have && error_word && lane == 0) atomicExch(error_word, 0x30000 + entry);
  if (first + r >= rows) {      // (the entries need more rows than there are: reported, nothing is written behind the last one)
    if (error_word && lane == 0) atomicExch(error_word, 0x60000 + entry);
    return;
  }
  const uint4* src = pool + (size_t)(have ? page : 0) * page_stride + (size_t)(r % page_size) * pieces;
  constexpr int AHEAD = 4;
  for (int c0 = lane; c0 < pieces; c0 += 32 * AHEAD) {
    uint4 v[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) v[u] = have && c0 + 32 * u < pieces ? src[c0 + 32 * u] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int c = c0 + 32 * u;
      if (c < rank8) latent[(size_t)(first + r) * rank8 + c] = v[u];
      else if (c < pieces) rotated[(size_t)(first + r) * rot8 + c - rank8] = v[u];
    }
  }
}

// DQ: sub-tiles of a query's unrotated part (dim / 64); DV: of a value (value_dim / 64).
template <int DQ, int DV>
struct LpSmem {
  static constexpr uint32_t kQ = (DQ + 1) * kLpSub;
  static constexpr uint32_t kK = (DQ + 1) * kLpSub;
  static constexpr uint32_t kV = DV * kLpSub;
  static constexpr uint32_t kTotal = 1024 + kQ + kLpStages * (kK + kV) + 256;
};

template <int DQ, int DV>
__global__ void __launch_bounds__(kLpThreads, 1)
latent_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                      const __grid_constant__ CUtensorMap map_r, LpArgs a) {
  using L = LpSmem<DQ, DV>;
  constexpr int D = DV * 64;                        // width of a value
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_s = base;
  auto k_s = [&](int s) { return base + L::kQ + s * (L::kK + L::kV); };
  auto v_s = [&](int s) { return base + L::kQ + s * (L::kK + L::kV) + L::kK; };
  const uint32_t bars = base + L::kQ + kLpStages * (L::kK + L::kV);
  const uint32_t q_full = bars;
  auto k_full = [&](int s) { return bars + 8u * (1 + s); };
  auto k_empty = [&](int s) { return bars + 8u * (1 + kLpStages + s); };
  auto v_full = [&](int s) { return bars + 8u * (1 + 2 * kLpStages + s); };
  auto v_empty = [&](int s) { return bars + 8u * (1 + 3 * kLpStages + s); };
  auto s_full = [&](int b) { return bars + 8u * (1 + 4 * kLpStages + b); };
  auto p_full = [&](int b) { return bars + 8u * (3 + 4 * kLpStages + b); };
  const uint32_t pv_done = bars + 8u * (5 + 4 * kLpStages);
  const uint32_t o_final = bars + 8u * (6 + 4 * kLpStages);
  const uint32_t tmem_slot = bars + 8u * (7 + 4 * kLpStages);
  unsigned char* smem_gen = smem_raw + (base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - base));

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int own = blockIdx.x, head = a.head0 + own, entry = blockIdx.y;      // own: among the heads that kv holds
  // (the first block may be placed while the kernel before drains: the entries' arrays were uploaded before the step began,
  // what the step's kernels write is only touched behind pdl_wait below)
  const int row0 = a.q_start[entry];
  const int q_len = a.q_start[entry + 1] - row0;
  const int t0 = (gridDim.z - 1 - blockIdx.z) * kLpTile;      // longest first
  if (t0 >= q_len || q_len < a.shortest) return;
  const int nt = min(kLpTile, q_len - t0);
  const int pos0 = a.kv_start[entry] + t0, last_pos = pos0 + nt - 1;
  const int n_tiles = last_pos / kLpTile + 1;
  constexpr uint32_t kTmemCols = 512;               // S (two buffers): columns 0..255; O_0, O_1: D columns each from 256

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < kLpStages; ++s) {
      mbar_init(k_full(s), 1);
      mbar_init(k_empty(s), 1);
      mbar_init(v_full(s), 1);
      mbar_init(v_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(s_full(b), 1);
      mbar_init(p_full(b), 32 * kLpWarps);
    }
    mbar_init(pv_done, 1);
    mbar_init(o_final, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tmem_slot), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem_base = *tmem_slot_ptr;
  const uint32_t tmem_s = tmem_base, tmem_o = tmem_base + 256;
  pdl_wait();
  pdl_trigger();

  if (warp == 0 || warp == kLpValueWarp) {
    const bool values = warp == kLpValueWarp;
    const int first = lp_first_row(a.q_start, a.kv_start, entry, lane);
    if (lane == 0) {
      if (!values) {      // (rows behind the portion belong to the next one, or to nobody: their results are not stored)
        mbar_expect_tx(q_full, L::kQ);
#pragma unroll
        for (int i = 0; i <= DQ; ++i) tma_load_3d(q_s + i * kLpSub, &map_q, i * 64, head, row0 + t0, q_full);
      }
      for (int it = 0; it < n_tiles; ++it) {
        const int s = it % kLpStages;
        if (!mbar_wait(values ? v_empty(s) : k_empty(s), ((it / kLpStages) & 1) ^ 1)) {
          if (a.error_word) atomicExch(a.error_word, values ? 0x7C0078 : 0x7C0071);
          break;
        }
        const int row = first + it * kLpTile;
        if (values) {
          mbar_expect_tx(v_full(s), L::kV);
#pragma unroll
          for (int i = 0; i < DV; ++i) tma_load_2d(v_s(s) + i * kLpSub, &map_kv, own * (a.dim + D) + a.dim + i * 64, row, v_full(s));
        } else {
          mbar_expect_tx(k_full(s), L::kK);
#pragma unroll
          for (int i = 0; i < DQ; ++i) tma_load_2d(k_s(s) + i * kLpSub, &map_kv, own * (a.dim + D) + i * 64, row, k_full(s));
          tma_load_2d(k_s(s) + DQ * kLpSub, &map_r, 0, row, k_full(s));      // (rot below 64: the box's last columns are zeros, as Q's are)
        }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kLpTile >> 3) << 17) | ((uint32_t)(kLpTile >> 4) << 24);
    constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) /* B is MN-major */ | ((uint32_t)(D >> 3) << 17) |
                                 ((uint32_t)(kLpTile >> 4) << 24);
    const uint32_t leader = umma_leader();
    auto note = [&](int code) {
      if (a.error_word && leader) atomicExch(a.error_word, code);
      return false;
    };
    bool ok = mbar_wait_warp(q_full, 0) || note(0x7C0072);
    // O_half += P . V of tile j: of each half's 64 columns of S, the first 32 hold the high terms, the others the remainders
    auto issue_pv = [&](int j) {
      const int s = j % kLpStages;
      if (!mbar_wait_warp(v_full(s), (j / kLpStages) & 1)) {
        note(0x7C0079);
        return;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t values = umma_low_mn128(v_s(s), kLpSub), p = tmem_s + (j & 1) * kLpTile;
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        const int half = kk >> 3, term = (kk >> 2) & 1, k = kk & 3;
        umma_warp_tmem(leader, tmem_o + half * D, p + half * 64 + term * 32 + k * 8, values + (half * 64 + k * 16) * 8, idesc_o, (j | (kk & 7)) != 0);
      }
      if (leader) {
        umma_commit(v_empty(s));
        umma_commit(pv_done);
      }
    };
    const uint32_t queries = umma_low_k128(q_s);
    for (int it = 0; it < n_tiles && ok; ++it) {
      const int s = it % kLpStages;
      if (!mbar_wait_warp(k_full(s), (it / kLpStages) & 1)) {
        ok = note(0x7C0073);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t keys = umma_low_k128(k_s(s));
#pragma unroll
      for (int kk = 0; kk < (DQ + 1) * 4; ++kk) {
        const uint32_t off = ((kk >> 2) * kLpSub + (kk & 3) * 32) >> 4;
        umma_warp(leader, tmem_s + (it & 1) * kLpTile, queries + off, keys + off, idesc_s, kk != 0);
      }
      if (leader) {
        umma_commit(k_empty(s));
        umma_commit(s_full(it & 1));
      }
      if (it > 0) {
        if (!mbar_wait_warp(p_full((it - 1) & 1), ((it - 1) >> 1) & 1)) {
          ok = note(0x7C0074);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        issue_pv(it - 1);
      }
    }
    if (ok) {
      const int last = n_tiles - 1;
      if (mbar_wait_warp(p_full(last & 1), (last >> 1) & 1)) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        issue_pv(last);
      } else {
        note(0x7C0074);
      }
    }
    if (leader) umma_commit(o_final);
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    const int qpos = r < nt ? pos0 + r : last_pos;
    constexpr int HC = kLpTile / 2;                 // score columns of a thread
    constexpr int OC = D / 2;                       // output columns of a thread at the end
    const uint32_t tmem_mine = tmem_o + half * D;
    float m = -CUDART_INF_F, l = 0.f;               // of this half's keys; m in log2 units (scaled)
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
      if (ok && !mbar_wait(s_full(it & 1), (it >> 1) & 1)) {
        if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0075);
        ok = false;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int key_base = it * kLpTile + half * HC;
      if (ok) {
        uint32_t sv[HC];
        const uint32_t mine = tmem_s + lane_sel + (it & 1) * kLpTile + half * HC;
        {
          uint32_t (&lo)[32] = *reinterpret_cast<uint32_t (*)[32]>(&sv[0]);
          uint32_t (&hi)[32] = *reinterpret_cast<uint32_t (*)[32]>(&sv[32]);
          tmem_ld32(mine, lo);
          tmem_ld32(mine + 32, hi);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        }
        float mx = -CUDART_INF_F;
        if (key_base + HC - 1 > pos0) {
#pragma unroll
          for (int j = 0; j < HC; ++j) {
            if (key_base + j > qpos) sv[j] = __float_as_uint(-CUDART_INF_F);
            mx = fmaxf(mx, __uint_as_float(sv[j]));
          }
        } else {
#pragma unroll
          for (int j = 0; j < HC; ++j) mx = fmaxf(mx, __uint_as_float(sv[j]));
        }
        // (the running maximum bounds the scores loosely, as in attention_tcgen05.cu: the weights stay below 2^kLpSlack and
        // rescaling O is rare)
        float m_new = fmaxf(m, mx == -CUDART_INF_F ? -CUDART_INF_F : mx * a.scale_log2);
        if (m_new - m <= kLpSlack) m_new = m;
        const float basev = m_new == -CUDART_INF_F ? 0.f : m_new;
        float alpha;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(alpha) : "f"(m - basev));
        m = m_new;
        const bool rescale = it > 0 && __any_sync(0xffffffffu, alpha != 1.f);
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < 2; ++c) {               // 32 keys at a time: 16 columns of high terms, 16 of remainders
          uint32_t ph[16], pl[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float e0, e1;
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(fmaf(__uint_as_float(sv[c * 32 + 2 * j]), a.scale_log2, -basev)));
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(fmaf(__uint_as_float(sv[c * 32 + 2 * j + 1]), a.scale_log2, -basev)));
            sum += e0 + e1;
            const __nv_bfloat162 pair = __floats2bfloat162_rn(e0, e1);
            const float2 back = bf16x2_floats(pair);
            const __nv_bfloat162 rest = __floats2bfloat162_rn(e0 - back.x, e1 - back.y);
            ph[j] = *reinterpret_cast<const uint32_t*>(&pair);
            pl[j] = *reinterpret_cast<const uint32_t*>(&rest);
          }
          tmem_st16(mine + c * 16, ph);
          tmem_st16(mine + 32 + c * 16, pl);
        }
        l = l * alpha + sum;
        if (rescale && !mbar_wait(pv_done, (it - 1) & 1)) {
          if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0077);
          ok = false;
        }
        if (ok && rescale) {
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            uint32_t v[32];
            tmem_ld32(tmem_mine + lane_sel + c * 32, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
            tmem_st32(tmem_mine + lane_sel + c * 32, v);
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      mbar_arrive(p_full(it & 1));
    }
    // Eight columns of the row at a time, the next ones' gates on their way (the first while the last products run).  The loop is not
    // unrolled: its code runs once a block and waits for its own fetch.
    const bool store = r < nt;
    const size_t row = (size_t)(row0 + t0 + (store ? r : 0));
    const __nv_bfloat16* gates = a.gate && !a.gate_per_head ? a.gate + row * a.ld_gate + head * D + half * OC : nullptr;
    uint4 gate = make_uint4(0u, 0u, 0u, 0u);
    if (gates) gate = *reinterpret_cast<const uint4*>(gates);
    if (ok && !mbar_wait(o_final, 0)) {
      if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0076);
      ok = false;
    }
    // the two halves of a row pass each other (maximum, sum) through the first key stage, which no MMA reads any more
    float2* fin = reinterpret_cast<float2*>(smem_gen + (k_s(0) - base));   // [2][128]
    fin[half * 128 + r] = make_float2(m, l);
    asm volatile("bar.sync 1, %0;\n" ::"n"(32 * kLpWarps) : "memory");
    const float2 other = fin[(half ^ 1) * 128 + r];
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const float sink2 = a.sink ? a.sink[head] * 1.4426950408889634f : -CUDART_INF_F;
      const float mm = fmaxf(fmaxf(m, other.x), sink2);    // (finite: every row sees at least one key)
      const float w_mine = exp2f(m - mm), w_other = exp2f(other.x - mm);
      const float inv = 1.f / (l * w_mine + other.y * w_other + (a.sink ? exp2f(sink2 - mm) : 0.f));
      const float w0 = (half == 0 ? w_mine : w_other) * inv, w1 = (half == 0 ? w_other : w_mine) * inv;
      __nv_bfloat16* dst = a.out + (row * a.heads + head) * D + half * OC;
      const float head_gate = a.gate && a.gate_per_head ? sigmoid_newton(__bfloat162float(a.gate[row * a.ld_gate + head])) : 1.f;
#pragma unroll 1
      for (int c = 0; c < OC; c += 8) {
        const uint32_t g[4] = {gate.x, gate.y, gate.z, gate.w};
        if (gates && c + 8 < OC) gate = *reinterpret_cast<const uint4*>(gates + c + 8);
        uint32_t v0[8], v1[8];
        tmem_ld8(tmem_o + lane_sel + half * OC + c, v0);          // O_0
        tmem_ld8(tmem_o + D + lane_sel + half * OC + c, v1);      // O_1
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (__uint_as_float(v0[j]) * w0 + __uint_as_float(v1[j]) * w1) * head_gate;
        if (gates) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&g[j]));
            o[2 * j] *= sigmoid_newton(f.x);
            o[2 * j + 1] *= sigmoid_newton(f.y);
          }
        }
        uint4 packed;
        __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
        for (int j = 0; j < 4; ++j) p2[j] = __floats2bfloat162_rn(o[2 * j], o[2 * j + 1]);
        if (store) *reinterpret_cast<uint4*>(dst + c) = packed;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// A bf16 tensor read in 128-byte-swizzled boxes of 64 x 128 rows (dims and strides from the innermost; 2 or 3 dimensions).
static int lp_map(CUtensorMap* map, const void* ptr, int rank, const cuuint64_t* dims, const cuuint64_t* strides) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return TIB_E_ARG;
  const cuuint32_t box2[2] = {64, kLpTile}, box3[3] = {64, 1, kLpTile}, elem[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(ptr), dims, strides, rank == 2 ? box2 : box3, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? TIB_OK : TIB_E_ARG;
}

template <int DQ, int DV>
static int launch_lp(const CUtensorMap& map_q, const CUtensorMap& map_kv, const CUtensorMap& map_r, const LpArgs& a, int n_heads, int n_entries,
                     int max_q_len, cudaStream_t stream) {
  auto kern = latent_prefill_kernel<DQ, DV>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LpSmem<DQ, DV>::kTotal);
  if (e != cudaSuccess) return (int)e;
  TIB_LAUNCH_DEPENDENT(kern, dim3(n_heads, n_entries, ceil_div(max_q_len, kLpTile)), kLpThreads, (LpSmem<DQ, DV>::kTotal), stream, map_q, map_kv,
                       map_r, a);
  return TIB_OK;
}

}  // namespace tib

using namespace tib;

// Whether the two kernels here take these sizes (bf16): heads of 64 or 128 unrotated and 8 .. 64 rotated elements with values of 64 or 128.
TIB_API int tib_latent_prefill_supports(int dim, int value_dim, int rank, int rot) {
  return (dim == 64 || dim == 128) && (value_dim == 64 || value_dim == 128) && rank >= 8 && rank % 8 == 0 && rot >= 8 && rot <= 64 && rot % 8 == 0;
}

// pool: this layer's pages of [page_size][rank + rot] bf16; latent [rows, rank] and rotated [rows, rot]: every entry's keys padded to a
// multiple of 128 rows (zeros), entry after entry; rows: how many there are.  What the entries need beyond that is reported in
// error_word (0x60000 + entry) and not written.
TIB_API int tib_latent_gather(const void* pool, int64_t page_stride, int page_size, int num_pages, const int* block_table, int table_stride,
                              const int* q_start, const int* kv_start, const int* slots, int n_entries, int max_kv_len, void* latent,
                              void* rotated, int rows, int rank, int rot, int* error_word, cudaStream_t stream) {
  if (n_entries == 0 || max_kv_len == 0) return TIB_OK;
  if (!pool || !block_table || !q_start || !kv_start || !slots || !latent || !rotated || page_size < 1 || rows < 0) return TIB_E_ARG;
  if (rank % 8 || rot % 8 || page_stride % 8 || (((uintptr_t)pool | (uintptr_t)latent | (uintptr_t)rotated) & 15)) return TIB_E_ALIGN;
  if (n_entries > 65535) return TIB_E_SIZE;
  TIB_LAUNCH_DEPENDENT(latent_gather_kernel, dim3(ceil_div(max_kv_len, kLpTile) * (kLpTile / kGatherRows), n_entries), 256, 0, stream, (const uint4*)pool,
                       page_stride / 8, page_size, num_pages, block_table, table_stride, q_start, kv_start, slots, (uint4*)latent,
                       (uint4*)rotated, rows, rank / 8, rot / 8, error_word);
  return TIB_OK;
}

// q: [tokens, heads, dim + rot] (row stride ldq) with the rotation applied; kv: [rows, n_heads * (dim + value_dim)], key and value of the
// heads head0 .. head0 + n_heads - 1, head by head, which are the ones this call works; rotated: [rows, rot]; gate: rows of heads (per head) or heads * value_dim numbers (row stride ld_gate) or null;
// out: [tokens, heads, value_dim].  All bf16; sink: [heads] fp32 or null; scale > 0.  Portions of fewer than `shortest` tokens are left
// alone (their keys have their rows all the same).
TIB_API int tib_latent_prefill(const void* q, int64_t ldq, const void* kv, const void* rotated, int rows, const int* q_start,
                               const int* kv_start, int n_entries, int max_q_len, int shortest, int n_tokens, int heads, int head0, int n_heads, int dim, int value_dim, int rot,
                               float scale, const float* sink, const void* gate, int64_t ld_gate, int gate_per_head, void* out,
                               int* error_word, cudaStream_t stream) {
  if (n_entries == 0 || max_q_len == 0) return TIB_OK;
  if (!q || !kv || !rotated || !q_start || !kv_start || !out || rows < 1 || !(scale > 0.f)) return TIB_E_ARG;
  if (!tib_latent_prefill_supports(dim, value_dim, 8, rot) || heads < 1 || head0 < 0 || n_heads < 1 || head0 > heads - n_heads || n_entries > 65535 || ceil_div(max_q_len, kLpTile) > 65535) return TIB_E_SIZE;
  if (ldq % 8 || (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)rotated | (uintptr_t)out) & 15)) return TIB_E_ALIGN;
  if (gate && !gate_per_head && (ld_gate % 8 || ((uintptr_t)gate & 15))) return TIB_E_ALIGN;
  CUtensorMap map_q, map_kv, map_r;
  const cuuint64_t qd[3] = {(cuuint64_t)(dim + rot), (cuuint64_t)heads, (cuuint64_t)n_tokens}, qs[2] = {(cuuint64_t)(dim + rot) * 2, (cuuint64_t)ldq * 2};
  const cuuint64_t width = (cuuint64_t)n_heads * (dim + value_dim);
  const cuuint64_t kd[2] = {width, (cuuint64_t)rows}, ks[1] = {width * 2}, rd[2] = {(cuuint64_t)rot, (cuuint64_t)rows}, rs[1] = {(cuuint64_t)rot * 2};
  int rc = lp_map(&map_q, q, 3, qd, qs);
  if (rc == TIB_OK) rc = lp_map(&map_kv, kv, 2, kd, ks);
  if (rc == TIB_OK) rc = lp_map(&map_r, rotated, 2, rd, rs);
  if (rc != TIB_OK) return rc;
  LpArgs a;
  a.q_start = q_start; a.kv_start = kv_start; a.sink = sink; a.gate = (const __nv_bfloat16*)gate; a.ld_gate = ld_gate;
  a.gate_per_head = gate_per_head; a.out = (__nv_bfloat16*)out; a.heads = heads; a.dim = dim; a.head0 = head0; a.shortest = shortest; a.scale_log2 = scale * 1.4426950408889634f;
  a.error_word = error_word;
  if (dim == 128)
    return value_dim == 128 ? launch_lp<2, 2>(map_q, map_kv, map_r, a, n_heads, n_entries, max_q_len, stream)
                            : launch_lp<2, 1>(map_q, map_kv, map_r, a, n_heads, n_entries, max_q_len, stream);
  return value_dim == 128 ? launch_lp<1, 2>(map_q, map_kv, map_r, a, n_heads, n_entries, max_q_len, stream)
                          : launch_lp<1, 1>(map_q, map_kv, map_r, a, n_heads, n_entries, max_q_len, stream);
}

// The calls the Python parts make (common.cuh).
TIB_PACKED(tib_latent_gather)
TIB_PACKED(tib_latent_prefill)
TIB_PACKED(tib_latent_prefill_supports)
