// Prompt portions of the attention in a sliding window (with averaged blocks behind it, or with the first tokens kept in sight) on the
// 5th-generation tensor cores.  Contract and exactness as pooled_window_attention.cu; the structure is attention_tcgen05.cu's:
// a block owns 128 rows (tokens x query heads of a key head), one warp copies queries and keys, one the values, one
// issues the products, eight warps do the softmax with two threads a row, whose halves merge exactly at the end.
//
//   tiles      first the 128-entry tiles of block means any row sees, then those of kept tokens, then the window's 128-key
//              tiles, all aligned to absolute numbers and walked in rising order
//   scores     times the head's factor (scale and temperature) in fp32, masked by one range of indices per row and tile
//   weights    fp32, fed to the second product as a high bf16 part and the remainder (16 bits), which together take the
//              columns of S they come from
//   the end    sink, division, the turn of the sum back by the query's position, the gate
//
// What bounds it: a block's chain of some six tiles of 1.4 us (the softmax's eight warps, one behind the other's products), 3 us before the first and 6
// behind the last (the division, turns and gates, whose code each block fetches anew), two blocks an SM one after the other: two portions
// of 1,366 and 682 tokens, 16 / 8 heads of 128, window 512, blocks of 64: 44 us, where it took 81 with cosines and sines made here, masks compared
// key by key and a lone lane issuing (mma.sync kernel, 64 x 64 tiles: 173).
// Every wait is bounded and reports in error_word.
#include "tcgen05.cuh"
#include "window_attention.cuh"
#include <math_constants.h>

namespace tib {

constexpr int kWtTile = 128;                       // rows of a block, keys of a tile
constexpr int kWtWarps = 8;
constexpr int kWtThreads = 64 + 32 * kWtWarps + 32;
constexpr int kWtValueWarp = 2 + kWtWarps;
constexpr int kWtStages = 3;
constexpr float kWtSlack = 8.f;
constexpr uint32_t kWtSub = kWtTile * 64 * 2;      // bytes of a [128][64] sub-tile

template <int D>
struct WtSmem {
  static constexpr uint32_t kQ = kWtTile * D * 2;
  static constexpr uint32_t kKV = kWtTile * D * 2;
  static constexpr uint32_t kTotal = 1024 + kQ + kWtStages * 2 * kKV + 256;
};

__device__ __forceinline__ float wt_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int D>
__global__ void __launch_bounds__(kWtThreads, 1)
window_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                      const __grid_constant__ CUtensorMap map_bk, const __grid_constant__ CUtensorMap map_bv, __nv_bfloat16* __restrict__ out,
                      PwaArgs a) {
  using L = WtSmem<D>;
  constexpr int DH = D / 64;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_s = base;
  auto k_s = [&](int s) { return base + L::kQ + s * 2 * L::kKV; };
  auto v_s = [&](int s) { return base + L::kQ + s * 2 * L::kKV + L::kKV; };
  const uint32_t bars = base + L::kQ + kWtStages * 2 * L::kKV;
  const uint32_t q_full = bars;
  auto k_full = [&](int s) { return bars + 8u * (1 + s); };
  auto k_empty = [&](int s) { return bars + 8u * (1 + kWtStages + s); };
  auto v_full = [&](int s) { return bars + 8u * (1 + 2 * kWtStages + s); };
  auto v_empty = [&](int s) { return bars + 8u * (1 + 3 * kWtStages + s); };
  auto s_full = [&](int b) { return bars + 8u * (1 + 4 * kWtStages + b); };
  auto p_full = [&](int b) { return bars + 8u * (3 + 4 * kWtStages + b); };
  const uint32_t pv_done = bars + 8u * (5 + 4 * kWtStages);
  const uint32_t o_final = bars + 8u * (6 + 4 * kWtStages);
  const uint32_t tmem_slot = bars + 8u * (7 + 4 * kWtStages);
  unsigned char* smem_gen = smem_raw + (base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - base));

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int entry = blockIdx.y, kvh = blockIdx.x, group = a.heads / a.kv_heads;
  const int row0 = a.q_start[entry];
  const int q_len = a.q_start[entry + 1] - row0;
  const int q_tile = kWtTile / group;
  const int t0 = (gridDim.z - 1 - blockIdx.z) * q_tile;
  if (t0 >= q_len || q_len < a.shortest) return;
  const int nt = min(q_tile, q_len - t0), nrows = nt * group;
  const int pos0 = a.kv_start[entry] + t0, last_pos = pos0 + nt - 1;
  // block means any row sees, kept tokens' tiles ahead of the window's first, the window's tiles
  const int n_blocks = a.pool > 0 ? max(0, last_pos - a.window + 1) / a.pool : 0;
  const int first_key = max(0, pos0 - a.window + 1);
  const int s_lo = first_key / kWtTile, s_hi = last_pos / kWtTile;
  const int steps_b = (n_blocks + kWtTile - 1) / kWtTile;
  const int steps_k = min(s_lo, (a.keep + kWtTile - 1) / kWtTile);
  const int n_tiles = steps_b + steps_k + s_hi - s_lo + 1;
  auto tile_base = [&](int it) {
    if (it < steps_b) return it * kWtTile;
    it -= steps_b;
    return (it < steps_k ? it : s_lo + it - steps_k) * kWtTile;
  };
  constexpr uint32_t kTmemCols = 512;              // S (two buffers): columns 0..255; O_0, O_1: D columns each from 256

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < kWtStages; ++s) {
      mbar_init(k_full(s), 1);
      mbar_init(k_empty(s), 1);
      mbar_init(v_full(s), 1);
      mbar_init(v_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(s_full(b), 1);
      mbar_init(p_full(b), 32 * kWtWarps);
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

  if (warp == 0 || warp == kWtValueWarp) {
    // lane 0 waits and arms the barrier, then lane p copies page p of the tile (at most sixteen of them)
    const bool values = warp == kWtValueWarp;
    const int slot = a.slots[entry];
    const int* ttable = a.tokens.block_table + (size_t)slot * a.tokens.table_stride;
    const int* btable = a.pool > 0 ? a.blocks.block_table + (size_t)slot * a.blocks.table_stride : nullptr;
    if (!values && lane == 0) {
      mbar_expect_tx(q_full, (uint32_t)(q_tile * group * D * 2));
#pragma unroll
      for (int h = 0; h < DH; ++h) tma_load_3d(q_s + h * kWtSub, &map_q, h * 64, kvh * group, row0 + t0, q_full);
    }
    for (int it = 0; it < n_tiles; ++it) {
      const int s = it % kWtStages;
      const bool pooled = it < steps_b;
      const PwaCache& c = pooled ? a.blocks : a.tokens;
      const int idx = tile_base(it) + lane * c.page_size;
      const bool mine = lane * c.page_size < kWtTile;
      // (a page is wanted if a row of it is seen; what it holds besides is masked, or zeroed below)
      const bool wanted = mine && (pooled ? idx < n_blocks : idx <= last_pos && (idx + c.page_size > first_key || idx < a.keep));
      int page = -1;
      if (wanted) {
        page = (pooled ? btable : ttable)[idx / c.page_size];
        if ((page < 0 || page >= c.num_pages) && a.error_word) atomicExch(a.error_word, 0x10000 + entry);
      }
      const bool have = page >= 0 && page < c.num_pages;
      const uint32_t full = values ? v_full(s) : k_full(s);
      int ok = 1;
      if (lane == 0) {
        ok = mbar_wait(values ? v_empty(s) : k_empty(s), ((it / kWtStages) & 1) ^ 1) ? 1 : 0;
        if (!ok && a.error_word) atomicExch(a.error_word, values ? 0x7C0088 : 0x7C0081);
        if (ok) mbar_expect_tx(full, L::kKV);
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      if (mine) {
        const CUtensorMap* map = pooled ? (values ? &map_bv : &map_bk) : (values ? &map_v : &map_k);
        const uint32_t dst = (values ? v_s(s) : k_s(s)) + (uint32_t)(lane * c.page_size) * 128u;
#pragma unroll
        for (int h = 0; h < DH; ++h)      // (a page beyond the pool's last reads zeros)
          tma_load_3d(dst + h * kWtSub, map, h * 64, kvh * c.page_size, have ? page : c.num_pages, full);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kWtTile >> 3) << 17) | ((uint32_t)(kWtTile >> 4) << 24);
    constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) /* B is MN-major */ | ((uint32_t)(D >> 3) << 17) |
                                 ((uint32_t)(kWtTile >> 4) << 24);
    const uint32_t leader = umma_leader();
    auto note = [&](int code) {
      if (a.error_word && leader) atomicExch(a.error_word, code);
      return false;
    };
    bool ok = mbar_wait_warp(q_full, 0) || note(0x7C0082);
    // O_half += P . V of tile j: of each half's 64 columns of S, the first 32 hold the high terms, the others the remainders
    auto issue_pv = [&](int j) {
      const int s = j % kWtStages;
      if (!mbar_wait_warp(v_full(s), (j / kWtStages) & 1)) {
        note(0x7C0089);
        return;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t values = umma_low_mn128(v_s(s), kWtSub), p = tmem_s + (j & 1) * kWtTile;
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
      const int s = it % kWtStages;
      if (!mbar_wait_warp(k_full(s), (it / kWtStages) & 1)) {
        ok = note(0x7C0083);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t keys = umma_low_k128(k_s(s));
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t off = ((kk >> 2) * kWtSub + (kk & 3) * 32) >> 4;
        umma_warp(leader, tmem_s + (it & 1) * kWtTile, queries + off, keys + off, idesc_s, kk != 0);
      }
      if (leader) {
        umma_commit(k_empty(s));
        umma_commit(s_full(it & 1));
      }
      if (it > 0) {
        if (!mbar_wait_warp(p_full((it - 1) & 1), ((it - 1) >> 1) & 1)) {
          ok = note(0x7C0084);
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
        note(0x7C0084);
      }
    }
    if (leader) umma_commit(o_final);
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    const int rr = min(r, nrows - 1), t = rr / group, head = kvh * group + rr - t * group;
    const int qpos = pos0 + t, lo = max(0, qpos - a.window + 1);
    const int seen = a.pool > 0 ? lo / a.pool : 0;        // blocks 0 .. seen - 1 lie wholly behind the row's window
    const float factor = a.scale * (a.temp ? a.temp[head] : 1.f) * 1.4426950408889634f;
    constexpr int HC = kWtTile / 2;
    const uint32_t tmem_mine = tmem_o + half * D;
    float m = -CUDART_INF_F, l = 0.f;                     // of this half's keys, in log2 units
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
      if (ok && !mbar_wait(s_full(it & 1), (it >> 1) & 1)) {
        if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0085);
        ok = false;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const bool pooled = it < steps_b;
      const int tile0 = tile_base(it), key_base = tile0 + half * HC;
      if (ok) {
        uint32_t sv[HC];
        const uint32_t mine = tmem_s + lane_sel + (it & 1) * kWtTile + half * HC;
        {
          uint32_t (&s_lo32)[32] = *reinterpret_cast<uint32_t (*)[32]>(&sv[0]);
          uint32_t (&s_hi32)[32] = *reinterpret_cast<uint32_t (*)[32]>(&sv[32]);
          tmem_ld32(mine, s_lo32);
          tmem_ld32(mine + 32, s_hi32);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        }
        // what this row sees of the tile, a bit a key: indices from .. from + span - 1, and the kept tokens up to its own
        const int from = pooled ? 0 : lo, span = pooled ? seen : qpos - lo + 1;
        float mx = -CUDART_INF_F;
        if (__all_sync(0xffffffffu, key_base >= from && key_base + HC <= from + span)) {
#pragma unroll
          for (int j = 0; j < HC; ++j) {
            const float v = __uint_as_float(sv[j]) * factor;
            sv[j] = __float_as_uint(v);
            mx = fmaxf(mx, v);
          }
        } else {
          auto bits = [&](int first, int end) -> unsigned long long {      // of indices first .. end - 1
            const int b0 = min(max(first - key_base, 0), HC), b1 = min(max(end - key_base, 0), HC);
            return b1 > b0 ? (~0ull >> (64 - (b1 - b0))) << b0 : 0ull;
          };
          const unsigned long long allowed = bits(from, from + span) | (pooled ? 0ull : bits(0, min(a.keep, qpos + 1)));
          const uint32_t allow[2] = {(uint32_t)allowed, (uint32_t)(allowed >> 32)};
#pragma unroll
          for (int j = 0; j < HC; ++j) {
            const float v = allow[j >> 5] & (1u << (j & 31)) ? __uint_as_float(sv[j]) * factor : -CUDART_INF_F;
            sv[j] = __float_as_uint(v);
            mx = fmaxf(mx, v);
          }
        }
        // (the running maximum bounds the scores loosely, as in attention_tcgen05.cu)
        float m_new = fmaxf(m, mx);
        if (m_new - m <= kWtSlack) m_new = m;
        const float basev = m_new == -CUDART_INF_F ? 0.f : m_new;
        const float alpha = wt_exp2(m - basev);
        m = m_new;
        const bool rescale = it > 0 && __any_sync(0xffffffffu, alpha != 1.f);
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < 2; ++c) {                     // 32 keys at a time: 16 columns of high terms, 16 of remainders
          uint32_t ph[16], pl[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float e0 = wt_exp2(__uint_as_float(sv[c * 32 + 2 * j]) - basev), e1 = wt_exp2(__uint_as_float(sv[c * 32 + 2 * j + 1]) - basev);
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
          if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0087);
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
        // values of entries no row sees may never have been written: they must not be NaN
        const int end = pooled ? n_blocks : last_pos + 1;
        if (tile0 + kWtTile > end) {
          const int s = it % kWtStages;
          if (!mbar_wait(v_full(s), (it / kWtStages) & 1)) {
            if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C008A);
            ok = false;
          }
          for (int key = max(end - tile0, 0) + (warp - 2); key < kWtTile; key += kWtWarps)
            for (int cb = lane; cb < D / 8; cb += 32)
              *reinterpret_cast<uint4*>(smem_gen + (v_s(s) - base) + (cb >> 3) * kWtSub + key * 128 + ((cb & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      mbar_arrive(p_full(it & 1));
    }
    // A thread's columns: a quarter of the row's first half and the same quarter of its second, so that the pairs a value's turn goes over
    // lie in one thread; eight of each at a time, the next ones' gates and turns on their way (the first while the last products run).
    // The turns come from the table that the append made of them: cosines and sines worked out here took 18 us of a block's 39.  The loop
    // is not unrolled: its code runs four times a block, and four copies of it, fetched once each, take 16 us where it takes 5.
    constexpr int W = D / 4;
    const bool store = r < nrows;
    const size_t token = (size_t)(row0 + t0 + t);
    const __nv_bfloat16* gates = a.gate ? reinterpret_cast<const __nv_bfloat16*>(a.gate) + token * a.ld_gate + head * D + half * W : nullptr;
    const float4* turns = a.turns ? reinterpret_cast<const float4*>(a.turns + token * D) + half * (W / 2) : nullptr;      // (two pairs each)
    uint4 gate[2];
    float4 turn[4];
    auto ask = [&](int c) {
#pragma unroll
      for (int part = 0; part < 2; ++part)
        if (gates) gate[part] = *reinterpret_cast<const uint4*>(gates + part * (D / 2) + c * 8);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (turns) turn[j] = turns[4 * c + j];
    };
    ask(0);
    if (ok && !mbar_wait(o_final, 0)) {
      if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0086);
      ok = false;
    }
    float2* fin = reinterpret_cast<float2*>(smem_gen + (k_s(0) - base));   // [2][128]: no MMA reads this stage any more
    fin[half * 128 + r] = make_float2(m, l);
    asm volatile("bar.sync 1, %0;\n" ::"n"(32 * kWtWarps) : "memory");
    const float2 other = fin[(half ^ 1) * 128 + r];
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const float sink2 = a.sink ? a.sink[head] * 1.4426950408889634f : -CUDART_INF_F;
      const float mm = fmaxf(fmaxf(m, other.x), sink2);    // (finite: every row sees its own position)
      const float w_mine = exp2f(m - mm), w_other = exp2f(other.x - mm);
      const float inv = 1.f / (l * w_mine + other.y * w_other + (a.sink ? exp2f(sink2 - mm) : 0.f));
      const float w0 = (half == 0 ? w_mine : w_other) * inv, w1 = (half == 0 ? w_other : w_mine) * inv;
      __nv_bfloat16* dst = out + token * a.heads * D + (size_t)head * D + half * W;
#pragma unroll 1
      for (int c = 0; c < W / 8; ++c) {
        const uint4 g0 = gate[0], g1 = gate[1];
        const float4 turn_now[4] = {turn[0], turn[1], turn[2], turn[3]};
        if (c + 1 < W / 8) ask(c + 1);
        uint32_t u0[8], u1[8], v0[8], v1[8];
        const uint32_t at = tmem_o + lane_sel + half * W + c * 8;
        tmem_ld8(at, u0);
        tmem_ld8(at + D, u1);
        tmem_ld8(at + D / 2, v0);
        tmem_ld8(at + D + D / 2, v1);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        float w[2][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          w[0][j] = __uint_as_float(u0[j]) * w0 + __uint_as_float(u1[j]) * w1;
          w[1][j] = __uint_as_float(v0[j]) * w0 + __uint_as_float(v1[j]) * w1;
        }
        // turned back by the query's position: (u, v) -> (u cos + v sin, v cos - u sin)
        auto turn_back = [&](int j, float cs, float sn) {
          const float x = rope_lo(w[0][j], w[1][j], cs, -sn), y = rope_hi(w[0][j], w[1][j], cs, -sn);
          w[0][j] = x;
          w[1][j] = y;
        };
        if (turns) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            turn_back(2 * j, turn_now[j].x, turn_now[j].y);
            turn_back(2 * j + 1, turn_now[j].z, turn_now[j].w);
          }
        } else if (a.vfreq) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float angle = (float)qpos * a.vfreq[half * W + c * 8 + j];
            turn_back(j, cosf(angle), sinf(angle));
          }
        }
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          if (gates) {
            const uint32_t g[4] = {part ? g1.x : g0.x, part ? g1.y : g0.y, part ? g1.z : g0.z, part ? g1.w : g0.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&g[j]));
              w[part][2 * j] *= sigmoid_newton(f.x);
              w[part][2 * j + 1] *= sigmoid_newton(f.y);
            }
          }
          uint4 packed;
          __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
          for (int j = 0; j < 4; ++j) p2[j] = __floats2bfloat162_rn(w[part][2 * j], w[part][2 * j + 1]);
          if (store) *reinterpret_cast<uint4*>(dst + part * (D / 2) + c * 8) = packed;
        }
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

static int wt_map(CUtensorMap* map, const void* ptr, const cuuint64_t (&dims)[3], const cuuint64_t (&strides)[2], const cuuint32_t (&box)[3]) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return TIB_E_ARG;
  const cuuint32_t elem[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? TIB_OK : TIB_E_ARG;
}

static bool wt_pages_suit(const PwaCache& c) {
  const bool pow2 = (c.page_size & (c.page_size - 1)) == 0;
  return pow2 && c.page_size >= 8 && c.page_size <= kWtTile && c.page_stride % 8 == 0 && (((uintptr_t)c.keys | (uintptr_t)c.values) & 15) == 0;
}

// Heads of 64 or 128, keys and values alike, groups of up to 64, pages of 8 .. 128 tokens, no distance bias; and portions with more
// than kWtFewRows rows in the step.
bool window_tcgen05_takes(const PwaArgs& a, const void* q, const void* out, int max_q_len) {
  const int group = a.heads / a.kv_heads;
  if (a.dim != a.vdim || (a.dim != 64 && a.dim != 128) || group > 64 || a.rel_bias || a.n_splits > 1) return false;
  if ((int64_t)max_q_len * group <= kWtFewRows || !wt_pages_suit(a.tokens) || (a.pool > 0 && !wt_pages_suit(a.blocks))) return false;
  if (a.gate && (a.gate_dtype != TIB_BF16 || a.ld_gate % 8 || ((uintptr_t)a.gate & 15))) return false;
  return (((uintptr_t)q | (uintptr_t)out) & 15) == 0 && ceil_div(max_q_len, kWtTile / group) <= 65535;
}

template <int D>
static int launch_wt(const void* q, void* out, const PwaArgs& a, int n_entries, int max_q_len, cudaStream_t stream) {
  const int group = a.heads / a.kv_heads, q_tile = kWtTile / group;
  CUtensorMap map_q, map_k, map_v, map_bk, map_bv;
  int rc = wt_map(&map_q, q, {(cuuint64_t)D, (cuuint64_t)a.heads, (cuuint64_t)a.n_tokens}, {(cuuint64_t)D * 2, (cuuint64_t)a.heads * D * 2},
                  {64, (cuuint32_t)group, (cuuint32_t)q_tile});
  auto pages = [&](CUtensorMap* map, const void* ptr, const PwaCache& c) {      // (D, rows of all key heads of a page, pages)
    return wt_map(map, ptr, {(cuuint64_t)D, (cuuint64_t)a.kv_heads * c.page_size, (cuuint64_t)c.num_pages},
                  {(cuuint64_t)D * 2, (cuuint64_t)c.page_stride * 2}, {64, (cuuint32_t)c.page_size, 1});
  };
  const PwaCache& blocks = a.pool > 0 ? a.blocks : a.tokens;      // (not read without blocks)
  if (rc == TIB_OK) rc = pages(&map_k, a.tokens.keys, a.tokens);
  if (rc == TIB_OK) rc = pages(&map_v, a.tokens.values, a.tokens);
  if (rc == TIB_OK) rc = pages(&map_bk, blocks.keys, blocks);
  if (rc == TIB_OK) rc = pages(&map_bv, blocks.values, blocks);
  if (rc != TIB_OK) return rc;
  auto kern = window_tcgen05_kernel<D>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WtSmem<D>::kTotal);
  if (e != cudaSuccess) return (int)e;
  TIB_LAUNCH_DEPENDENT(kern, dim3(a.kv_heads, n_entries, ceil_div(max_q_len, q_tile)), kWtThreads, WtSmem<D>::kTotal, stream, map_q, map_k, map_v,
                       map_bk, map_bv, (__nv_bfloat16*)out, a);
  return TIB_OK;
}

int window_tcgen05(const void* q, void* out, const PwaArgs& a, int n_entries, int max_q_len, cudaStream_t stream) {
  return a.dim == 128 ? launch_wt<128>(q, out, a, n_entries, max_q_len, stream) : launch_wt<64>(q, out, a, n_entries, max_q_len, stream);
}

}  // namespace tib
