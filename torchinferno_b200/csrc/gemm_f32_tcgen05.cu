// The 32-bit matrix product out[M, N] = x[M, K] . w[N, K]^T on the tensor cores, with 32-bit operands and sums.
//
// A float is the sum of three bf16 numbers (8 bits of its 24 each, rounded to nearest): a = a0 + a1 + a2.  The product of two
// floats is then nine products of bf16 numbers, each exact in fp32; the six of them that are above 2^-24 of the whole are made,
//     a0 b0   |   a0 b1 + a1 b0   |   a0 b2 + a1 b1 + a2 b0
// each group in an accumulator of its own, for the tensor core cuts sums off where an fp32 addition rounds: the small terms lose
// nothing that way, and a0 b0 is only summed over 128 k there (eight instructions), then added to the output's sum in registers as an
// ordinary fp32 number.  The terms of the rows lie behind one another in shared memory, so that four instructions make the six products: a0 with
// b0, a0 with b1 and b2 side by side, a1 with b0 and b1, a2 with b0.  Every output is summed over k in the same order whatever the number of rows, so a row's bits do not depend on its
// neighbours or on the tile's width.
//
// The weights are the 128-row operand, from tensor memory; rows of x are the other (a tile takes up to 80 of them, in sixteens):
//   warps 0..15   turn the step's 128 x 64 weights, as they came into shared memory, into three terms in tensor memory
//   warp 16       one lane: TMA of the weights and of the rows' three terms (made by split_rows_kernel once a call: every tile of features
//                 reads them)
//   warp 17       issues the MMAs (the whole warp walks the loop, one lane issues: descriptors then stay in uniform registers); owns tensor
//                 memory, all of it: a step's terms of the weights twice, the accumulator of a0 b0 twice, the small ones once
//   warps 18..25  add the accumulators of 128 k up in registers while the next ones are made, and store the rows
//
// What bounds it: the warp that issues the MMAs, which waits once and issues 16 instructions a step of 64 k (0.95 us at 80 rows, of which 0.5 are
// products), and for the last round of tiles the SMs that have none.  A wait for the rows, one for each half of the weights' terms and one
// commit each made it 1.15 us; a lane issuing alone takes 45 cycles an instruction instead of 8.  301 rows, us, against gemm_f32.cu's fused
// multiply-adds: 16,384 x 2,048 117 (536), 2,048 x 8,192 66 (431), 2,048 x 2,048 25 (111); 8 rows: 30 (68), 33 (146), 20 (39).
// Error against 64 bits (2-norm): 1.4e-7 at 2,048 k and 1.5e-7 at 8,192, where multiply-adds in order have 8.1e-7 and 1.6e-6; numbers of one
// sign 1.6e-7 (6.3e-7); sums over 256 k 2.4e-7, for a tenth off the time.
// An output that is not finite is worked out again with fused multiply-adds in order (an infinity's terms make NaN of it).
#include "split_terms.cuh"
#include "cluster.cuh"

namespace tib {

constexpr int kFtM = 128, kFtK = 64, kFtRows = 80, kFtThreads = 832, kFtChunk = 2;      // (steps of 64 k in a chunk)
constexpr int kFtGroups = (kFtRows / 16 + 1) / 2;               // groups of 16 rows a warp adds up
constexpr uint32_t kFtW = kFtM * kFtK * 4;                      // a step's weights in shared memory
constexpr uint32_t kFtTermCols = 3 * kFtK / 2;                  // in tensor memory: a step's terms of the weights, twice
constexpr uint32_t kFtSums = 2 * kFtTermCols;                   // a0 b0 twice, then the two small groups

// The three terms of x, [3][rows][K]; grid-stride, four elements a thread.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, int64_t ldx, int rows, int K, __nv_bfloat16* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  const int64_t quarters = (int64_t)rows * (K / 4), plane = (int64_t)rows * K;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < quarters; e += (int64_t)gridDim.x * 256) {
    const int64_t r = e / (K / 4);
    const int c = (int)(e - r * (K / 4)) * 4;
    const float4 v = *reinterpret_cast<const float4*>(x + r * ldx + c);
    uint2 t[3];
    ft_split2(v.x, v.y, t[0].x, t[1].x, t[2].x);
    ft_split2(v.z, v.w, t[0].y, t[1].y, t[2].y);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(out + i * plane + r * K + c) = t[i];
  }
}

// An output whose terms did not add up to a finite number.
__device__ __noinline__ float ft_plain_sum(const float* __restrict__ x, const float* __restrict__ w, int K) {
  float s = 0.f;
  for (int k = 0; k < K && s == s; ++k) s = fmaf(x[k], w[k], s);
  return s;
}

struct FtArgs {
  const float* x;
  const float* w;
  float* out;
  int64_t ldx, ldw, ldo;
  int M, N, K;
  int rows;               // rows of a tile (a multiple of 16, at most kFtRows)
  int parts;              // of k, each summed by itself
  float* partial;         // [parts][M][N]: the parts' sums go there, a block takes any part of any tile; null: a block takes all parts of a tile, one after the other
  int w_stages, x_stages;
  int* error_word;
};

// A thread's sums of one feature into out, fetched and added to where `onto`; where `last`, what is not finite is made again, in a second pass over what was
// stored (a call with the sums still in registers would spill them).
__device__ __forceinline__ void ft_put(float (&sum)[kFtGroups][16], float* out, int64_t ld, bool onto, bool last, int m0, int feature, int half, const FtArgs& a) {
  if (feature >= a.N) return;
  bool finite = true;
#pragma unroll
  for (int g = 0; g < kFtGroups; ++g) {
    const int j0 = (2 * g + half) * 16, left = min(a.rows - j0, a.M - m0 - j0);
    if (left <= 0) break;
    float* to = out + (size_t)(m0 + j0) * ld + feature;
    if (onto) {
      float before[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) before[c] = c < left ? to[c * ld] : 0.f;
#pragma unroll
      for (int c = 0; c < 16; ++c) sum[g][c] = before[c] + sum[g][c];
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      if (c >= left) break;
      finite = finite && isfinite(sum[g][c]);
      to[c * ld] = sum[g][c];
    }
  }
  if (!last || finite) return;
#pragma unroll 1
  for (int g = 0; g < kFtGroups; ++g)
#pragma unroll 1
    for (int c = 0; c < 16; ++c) {
      const int row = (2 * g + half) * 16 + c;
      if (row >= a.rows || m0 + row >= a.M) break;
      float* to = out + (size_t)(m0 + row) * ld + feature;
      if (!isfinite(*to)) *to = ft_plain_sum(a.x + (size_t)(m0 + row) * a.ldx, a.w + (size_t)feature * a.ldw, a.K);
    }
}

__global__ void __launch_bounds__(kFtThreads, 1)
gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, FtArgs a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* smem_gen = smem_raw + (base - smem_u32(smem_raw));
  // Two rings: the weights' places are free again once they are converted, the rows' once they are multiplied.
  const uint32_t xplane = (uint32_t)a.rows * kFtK * 2, xring = base + a.w_stages * kFtW;
  const uint32_t bars = xring + a.x_stages * 3 * xplane;
  auto w_full_bar = [&](int s) { return bars + 8u * s; };
  auto w_empty_bar = [&](int s) { return bars + 8u * (8 + s); };
  auto x_full_bar = [&](int s) { return bars + 8u * (16 + s); };
  auto x_empty_bar = [&](int s) { return bars + 8u * (24 + s); };
  auto acc_full_bar = [&](int b) { return bars + 8u * (32 + b); };
  auto acc_empty_bar = [&](int b) { return bars + 8u * (34 + b); };
  const uint32_t small_empty_bar = bars + 8u * 36, tmem_slot = bars + 8u * 37;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - base));

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 8; ++s) {
      mbar_init(w_full_bar(s), 1);
      mbar_init(w_empty_bar(s), 16);
      mbar_init(x_full_bar(s), 1 + 16);      // (the rows' copies, and the weights' terms)
      mbar_init(x_empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full_bar(b), 1);
      mbar_init(acc_empty_bar(b), 8);
    }
    mbar_init(small_empty_bar, 8);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 17) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tmem_slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  pdl_wait();
  pdl_trigger();
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem_base = *tmem_slot_ptr;

  const int m_tiles = (a.M + a.rows - 1) / a.rows, f_tiles = (a.N + kFtM - 1) / kFtM, num_tiles = m_tiles * f_tiles;
  const int k_steps = a.K / kFtK;
  // This block's pieces of work: parts of tiles, steps first .. end - 1 of k.
  struct Piece { int tile, part, first, end; };
  const int of_tile = a.partial ? 1 : a.parts, stride = (int)gridDim.x, all = a.partial ? num_tiles * a.parts : num_tiles;
  const int pieces = (int)blockIdx.x < all ? (all - (int)blockIdx.x + stride - 1) / stride * of_tile : 0;
  const auto piece_of = [&](int i) {
    Piece u;
    if (a.partial) {
      const int at = (int)blockIdx.x + i * stride;
      u.tile = at / a.parts;
      u.part = at - u.tile * a.parts;
    } else {
      u.tile = (int)blockIdx.x + i / a.parts * stride;
      u.part = i % a.parts;
    }
    u.first = k_steps * u.part / a.parts;
    u.end = k_steps * (u.part + 1) / a.parts;
    return u;
  };
  int total = 0;
  for (int i = 0; i < pieces; ++i) {
    const Piece u = piece_of(i);
    total += u.end - u.first;
  }

  if (warp < 16) {
    // lane: a feature; the warp's 16 of the step's 64 k (which come as two copies of 32 k: rows of 128 bytes, swizzled)
    const int quarter = warp & 3, part = warp >> 2, r = quarter * 32 + lane;
    int ws = 0, xs = 0, before = 0;      // (places of this step, and of the one that used these terms' columns before)
    uint32_t wphase = 0, bphase = 0;
    const uint32_t dst = tmem_base + ((uint32_t)(quarter * 32) << 16) + part * 8;
    for (int it = 0; it < total; ++it) {
      if (!mbar_wait(w_full_bar(ws), wphase)) {
        if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0091);
        break;
      }
      const unsigned char* src = smem_gen + (size_t)ws * kFtW + (part >> 1) * (kFtW / 2) + r * 128;
      uint32_t t[3][8];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float4 v = *reinterpret_cast<const float4*>(src + ((((part & 1) * 4 + c) ^ (r & 7)) << 4));
        ft_split2(v.x, v.y, t[0][2 * c], t[1][2 * c], t[2][2 * c]);
        ft_split2(v.z, v.w, t[0][2 * c + 1], t[1][2 * c + 1], t[2][2 * c + 1]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(w_empty_bar(ws));
      if (it >= 2) {      // (the products of two steps ago are done)
        if (!mbar_wait(x_empty_bar(before), bphase)) {
          if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0096);
          break;
        }
        if (++before == a.x_stages) {
          before = 0;
          bphase ^= 1;
        }
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
      for (int p = 0; p < 3; ++p) ft_tmem_st8(dst + (it & 1) * kFtTermCols + p * (kFtK / 2), t[p]);
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(x_full_bar(xs));
      if (++ws == a.w_stages) {
        ws = 0;
        wphase ^= 1;
      }
      if (++xs == a.x_stages) xs = 0;
    }
  } else if (warp == 16) {
    if (lane == 0) {
      int ws = 0, xs = 0;
      uint32_t wphase = 1, xphase = 1;
      bool ok = true;
      for (int i = 0; i < pieces && ok; ++i) {
        const Piece u = piece_of(i);
        const int m0 = u.tile % m_tiles * a.rows, f0 = u.tile / m_tiles * kFtM;
        for (int ks = u.first; ks < u.end; ++ks) {
          ok = mbar_wait(w_empty_bar(ws), wphase);
          if (ok) {
            mbar_expect_tx(w_full_bar(ws), kFtW);
            for (int half = 0; half < 2; ++half)      // (features behind the last one: zeros)
              tma_load_2d(base + ws * kFtW + half * (kFtW / 2), &map_w, ks * kFtK + half * 32, f0, w_full_bar(ws));
            ok = mbar_wait(x_empty_bar(xs), xphase);
          }
          if (!ok) {
            if (a.error_word) atomicExch(a.error_word, 0x7C0092);
            break;
          }
          mbar_expect_tx(x_full_bar(xs), 3 * xplane);
          for (int p = 0; p < 3; ++p)      // (rows behind the last one: another term's, or zeros; never stored)
            tma_load_2d(xring + (xs * 3 + p) * xplane, &map_x, ks * kFtK, p * a.M + m0, x_full_bar(xs));
          if (++ws == a.w_stages) {
            ws = 0;
            wphase ^= 1;
          }
          if (++xs == a.x_stages) {
            xs = 0;
            xphase ^= 1;
          }
        }
      }
    }
  } else if (warp == 17) {
    const uint32_t leader = umma_leader(), idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kFtM >> 4) << 24);
    const uint32_t n1 = (uint32_t)(a.rows >> 4) << 18;      // (an instruction's columns, in sixteens)
    int s = 0;
    uint32_t phase = 0, chunk = 0, it = 0;
    bool ok = true;
    const uint32_t small = tmem_base + kFtSums + 2 * kFtRows;      // (behind each other: a.rows columns a group)
    for (int i = 0; i < pieces && ok; ++i) {
      const Piece u = piece_of(i);
      for (int ks = u.first; ks < u.end && ok; ks += kFtChunk, ++chunk) {
        const int ab = chunk & 1;
        const bool free = mbar_wait(acc_empty_bar(ab), ((chunk >> 1) & 1) ^ 1) && (ks > u.first || mbar_wait(small_empty_bar, (i & 1) ^ 1));
        if (!__all_sync(0xffffffffu, free)) {
          if (a.error_word && leader) atomicExch(a.error_word, 0x7C0094);
          ok = false;
          break;
        }
        const uint32_t large = tmem_base + kFtSums + ab * kFtRows;
        for (int kc = 0; kc < kFtChunk && ks + kc < u.end && ok; ++kc, ++it) {
          const uint32_t xs = xring + s * 3 * xplane, wt = tmem_base + (it & 1) * kFtTermCols;
          if (!__all_sync(0xffffffffu, mbar_wait(x_full_bar(s), phase))) {
            if (a.error_word && leader) atomicExch(a.error_word, 0x7C0093);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
          for (int k = 0; k < kFtK / 16; ++k) {
            const uint32_t x0 = umma_low_k128(xs + k * 32), x1 = umma_low_k128(xs + xplane + k * 32);
            const uint32_t w0 = wt + k * 8, w1 = w0 + kFtK / 2, w2 = w1 + kFtK / 2;
            umma_warp_tmem(leader, small, w0, x1, idesc0 | 2 * n1, (ks - u.first | kc | k) != 0);
            umma_warp_tmem(leader, small, w1, x0, idesc0 | 2 * n1, 1);
            umma_warp_tmem(leader, small + a.rows, w2, x0, idesc0 | n1, 1);
            umma_warp_tmem(leader, large, w0, x0, idesc0 | n1, (kc | k) != 0);
          }
          if (leader) umma_commit(x_empty_bar(s));
          if (++s == a.x_stages) {
            s = 0;
            phase ^= 1;
          }
        }
        if (leader) umma_commit(acc_full_bar(ab));      // (also on failure, so that the sums' warps do not wait in vain)
      }
    }
  } else {
    const int quarter = warp & 3, half = (warp - 18) >> 2;      // 32 features; groups of 16 rows half, half + 2, ...
    uint32_t chunk = 0;
    bool ok = true;
    for (int i = 0; i < pieces && ok; ++i) {
      const Piece u = piece_of(i);
      float sum[kFtGroups][16];
#pragma unroll
      for (int g = 0; g < kFtGroups; ++g)
#pragma unroll
        for (int c = 0; c < 16; ++c) sum[g][c] = 0.f;
      for (int ks = u.first; ks < u.end; ks += kFtChunk, ++chunk) {
        const int b = chunk & 1;
        if (!mbar_wait(acc_full_bar(b), (chunk >> 1) & 1)) {
          if (a.error_word && lane == 0) atomicExch(a.error_word, 0x7C0095);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const bool last = ks + kFtChunk >= u.end;
        const uint32_t at = tmem_base + ((uint32_t)(quarter * 32) << 16) + kFtSums;
#pragma unroll
        for (int g = 0; g < kFtGroups; ++g) {
          const int c0 = (2 * g + half) * 16;
          if (c0 >= a.rows) break;
          uint32_t v[16];
          tmem_ld16(at + b * kFtRows + c0, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
          for (int c = 0; c < 16; ++c) sum[g][c] += __uint_as_float(v[c]);
        }
        if (last) {
#pragma unroll
          for (int e = 0; e < 2 * kFtGroups; ++e) {
            const int c0 = (2 * (e >> 1) + half) * 16 + (e & 1) * 8;
            if (c0 >= a.rows) break;
            uint32_t m[8], n[8];
            tmem_ld8(at + 2 * kFtRows + c0, m);
            tmem_ld8(at + 2 * kFtRows + a.rows + c0, n);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int c = 0; c < 8; ++c) sum[e >> 1][(e & 1) * 8 + c] += __uint_as_float(m[c]) + __uint_as_float(n[c]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(acc_empty_bar(b));
          if (last) mbar_arrive(small_empty_bar);
        }
      }
      if (!ok) break;
      const int m0 = u.tile % m_tiles * a.rows, feature = u.tile / m_tiles * kFtM + quarter * 32 + lane;
      const bool last = u.part == a.parts - 1;
      // (a part's sum: by itself, or on top of the parts' before it)
      ft_put(sum, a.partial ? a.partial + (size_t)u.part * a.M * a.N : a.out, a.partial ? a.N : a.ldo, !a.partial && u.part > 0, !a.partial && last, m0, feature, half, a);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 17) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// The parts' sums, in their order: four outputs a thread.
__global__ void __launch_bounds__(256) add_parts_kernel(FtArgs a) {
  pdl_wait();
  pdl_trigger();
  const int64_t outputs = (int64_t)a.M * a.N, first = (int64_t)blockIdx.x * 1024 + threadIdx.x;
  float v[4], next[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = first + i * 256 < outputs ? a.partial[first + i * 256] : 0.f;
  for (int p = 1; p < a.parts; ++p) {
#pragma unroll
    for (int i = 0; i < 4; ++i) next[i] = first + i * 256 < outputs ? a.partial[p * outputs + first + i * 256] : 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = v[i] + next[i];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t e = first + i * 256;
    if (e >= outputs) break;
    const int64_t row = e / a.N, f = e - row * a.N;
    a.out[row * a.ldo + f] = isfinite(v[i]) ? v[i] : ft_plain_sum(a.x + row * a.ldx, a.w + f * a.ldw, a.K);
  }
}

// Into how many parts of k a product is summed, each by itself: by the weight's sizes alone, so that a row's bits do not depend on how many rows
// there are.  A weight of few features leaves SMs without a tile (2,048 features, 301 rows: 64 to 112 tiles), and these parts are work for them, while with
// many rows they cost their ends; us on 8 / 100 / 301 / 1,000 / 2,048 rows, weights in the L2: 2,048 x 8,192 in one 91 / 89 / 95 / 205 / 372, in four 34 / 38 /
// 66 / 195 / 415; 2,048 x 4,096 50 / 50 / 52 / 104 / 184 and 17 / 24 / 40 / 102 / 195; 4,096 x 4,096 55 / 52 / 60 / 177 / 368, in two 30 / 38 / 61 / 178 / 366
// (in four 22 / 39 / 68 / 190 / 400); 3,072 x 4,096 55 / 52 / 54 / 152 / 290 and 33 / 33 / 54 / 150 / 288; 2,048 x 2,048 32 / 32 / 32 / 59 / 94 and 20 / 22 /
// 27 / 58 / 95; 3,072 x 2,048 32 / 31 / 33 / 84 / 152 and 21 / 26 / 34 / 83 / 150; 8,192 x 2,048 33 / 35 / 65 / 182 / 380 and 23 / 36 / 68 / 183 / 380.
static int ft_parts(int N, int K) {
  const int f_tiles = ceil_div(N, kFtM), k_steps = K / kFtK;
  return f_tiles <= 16 && k_steps >= 64 ? 4 : f_tiles <= 64 && k_steps >= 32 ? 2 : 1;
}

// Rows of a tile, and whether the parts go to blocks of their own: whole rounds of work over the SMs times its steps' cost (0.65 us with 16
// rows, 0.76 with 48, 0.95 with 80: in units of 1 / 210 us), and for parts of their own the launch that adds them (3 us, and their way through the L2).
struct FtPlan { int rows; bool apart; };
static FtPlan ft_plan(int rows, int N, int K, bool may_part) {
  const int parts = ft_parts(N, K), k_steps = K / kFtK;
  FtPlan plan = {kFtRows, false};
  double least = 1e30;
  for (int tiles = ceil_div(rows, kFtRows); tiles <= ceil_div(rows, 16); ++tiles) {
    const int r = ceil_div(ceil_div(rows, tiles), 16) * 16;
    const int64_t n = (int64_t)ceil_div(rows, r) * ceil_div(N, kFtM);
    const double step = 120 + r, whole = (double)ceil_div64(n, 148) * k_steps * step;
    const double bytes = 8.0 * parts * rows * N;
    const double apart = parts > 1 && may_part && bytes <= 128e6 ? (double)ceil_div64(n * parts, 148) * ceil_div(k_steps, parts) * step + 210 * (3 + bytes / 4e6) : 1e30;
    if (whole < least) {
      least = whole;
      plan = {r, false};
    }
    if (apart < least) {
      least = apart;
      plan = {r, true};
    }
  }
  return plan;
}

// Rows of 32-bit weights in boxes of 128 x 32.
static int ft_weight_map(CUtensorMap* map, const float* w, int N, int K, int64_t ldw) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return TIB_E_ARG;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, strides[1] = {(cuuint64_t)ldw * 4};
  const cuuint32_t box[2] = {32u, (cuuint32_t)kFtM}, elem[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? TIB_OK : TIB_E_ARG;
}

}  // namespace tib

using namespace tib;

// Whether a weight's product runs here.  By the weight's sizes and the alignment alone, not by the number of rows: a request's
// numbers do not depend on what else is in the step.  On the device terms are faster from a million weights on, whatever the rows (1,024 x 1,024,
// us on 8 / 40 / 300 rows: 19 / 19 / 43 by multiply-adds and 16 / 17 / 19 here; 2,048 x 2,048 37 / 50 / 110 and 26 / 27 / 31).  But a product issued
// call by call costs the host some 8 us more (two launches and the scratch), and a block of such weights on few tokens waits for the host.
// Blocks call by call (8 / 4 heads of 128), us on 8 / 40 / 100 / 300 tokens, by multiply-adds alone, with the line at 2^22 weights and at 2^20:
//     1,024 wide, 1,024 inside   119 / 123 / 155 / 277   118 / 123 / 155 / 277   143 / 144 / 145 / 145
//     1,024 wide, 2,112 inside   127 / 146 / 196 / 354   127 / 132 / 169 / 285   149 / 149 / 150 / 150
//     1,536 wide, 3,200 inside   173 / 214 / 299 / 528   137 / 139 / 173 / 281   149 / 150 / 150 / 191
//     1,536 wide, 6,400 inside   242 / 292 / 448 / 798   138 / 147 / 197 / 331   150 / 151 / 153 / 238
// So no line is best for all: 2^20 would cost few tokens 10 to 20 % and gain prompts of a hundred tokens and more 6 to 48 %.
// (Weights whose rows overlap or are one and the same are none of a tensor map's.)
TIB_API int tib_gemm_f32_tcgen05_takes(const void* x, const void* w, int N, int K, int64_t ldx, int64_t ldw) {
  return N >= 512 && K >= 512 && (int64_t)N * K >= (1 << 22) && K % kFtK == 0 && ldx % 4 == 0 && ldw % 4 == 0 && ldw >= K &&
         (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
}

// Rows of N numbers that a product of M rows, made scratch_rows at a time, takes for its parts' sums (0: none).
TIB_API int tib_gemm_f32_tcgen05_partial(int M, int N, int K, int scratch_rows) {
  if (M < 1 || N < 1 || K < kFtK || scratch_rows < 1) return 0;
  int most = 0;
  for (int rows : {M < scratch_rows ? M : scratch_rows, M % scratch_rows})
    if (rows > 0 && ft_plan(rows, N, K, true).apart && ft_parts(N, K) * rows > most) most = ft_parts(N, K) * rows;
  return most;
}

// x: [M, K] (row stride ldx), w: [N, K] (row stride ldw), out: [M, N] (row stride ldo), all fp32.  scratch: bf16, 3 K numbers for each
// of scratch_rows rows, on a 16-byte boundary; the product is made for that many rows at a time.  partial: partial_rows rows of N numbers, as many as
// tib_gemm_f32_tcgen05_partial says (fewer, or none: the same bits, a block taking all parts of a tile).  launches: takes the number of kernels launched.
TIB_API int tib_gemm_f32_tcgen05(const float* x, const float* w, float* out, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo,
                                 void* scratch, int scratch_rows, float* partial, int partial_rows, int* error_word, int* launches, cudaStream_t stream) {
  *launches = 0;
  if (M == 0) return TIB_OK;
  if (!x || !w || !out || !scratch || M < 0 || scratch_rows < 1 || ((uintptr_t)scratch & 15)) return TIB_E_ARG;
  if (!tib_gemm_f32_tcgen05_takes(x, w, N, K, ldx, ldw) || (int64_t)scratch_rows * 3 > 0x7fffffff - 256) return TIB_E_SIZE;
  const int parts = ft_parts(N, K);
  for (int first = 0; first < M; first += scratch_rows) {
    const int rows = M - first < scratch_rows ? M - first : scratch_rows;
    const FtPlan plan = ft_plan(rows, N, K, partial && (int64_t)parts * rows <= partial_rows);
    const int best = plan.rows;
    FtArgs a;
    a.x = x + (size_t)first * ldx; a.w = w; a.out = out + (size_t)first * ldo;
    a.ldx = ldx; a.ldw = ldw; a.ldo = ldo; a.M = rows; a.N = N; a.K = K; a.rows = best; a.error_word = error_word;
    a.parts = parts; a.partial = plan.apart ? partial : nullptr;
    const int x_stage = 3 * best * kFtK * 2;
    a.x_stages = best > 48 ? 4 : 6;
    a.w_stages = (220 * 1024 - a.x_stages * x_stage) / (int)kFtW < 6 ? (220 * 1024 - a.x_stages * x_stage) / (int)kFtW : 6;
    const int smem = 1024 + a.w_stages * (int)kFtW + a.x_stages * x_stage + 512;
    CUtensorMap map_w, map;
    int rc = ft_weight_map(&map_w, w, N, K, ldw);
    if (rc == TIB_OK) rc = make_map(&map, scratch, 3 * rows, K, K, best);
    if (rc != TIB_OK) return rc;
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
    if (e != cudaSuccess) return (int)e;
    const int64_t blocks = ceil_div64((int64_t)rows * K / 4, 256);
    TIB_LAUNCH_DEPENDENT(split_rows_kernel, (int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream, a.x, ldx, rows, K, (__nv_bfloat16*)scratch);
    const int64_t tiles = (int64_t)ceil_div(rows, best) * ceil_div(N, kFtM) * (plan.apart ? parts : 1);
    TIB_LAUNCH_DEPENDENT(gemm_f32_tcgen05_kernel, (int)(tiles < 148 ? tiles : 148), kFtThreads, smem, stream, map_w, map, a);
    *launches += 2;
    if (plan.apart) {
      TIB_LAUNCH_DEPENDENT(add_parts_kernel, (unsigned)ceil_div64((int64_t)rows * N, 1024), 256, 0, stream, a);
      ++*launches;
    }
  }
  return TIB_OK;
}

// The calls the Python parts make (common.cuh).
TIB_PACKED(tib_gemm_f32_tcgen05)
TIB_PACKED(tib_gemm_f32_tcgen05_partial)
TIB_PACKED(tib_gemm_f32_tcgen05_takes)
