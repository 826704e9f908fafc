// The experts' products over the sorted (token, choice) rows on the 5th-generation tensor cores (bf16 operands, fp32 sums):
//     y[s] = act(x[source of s] . W_e^T)    for the rows s of expert e, W: [experts, N, K]
//
// The weights are the 128-row operand of the MMA and the sorted rows its N dimension: a tile is 128 features x up to NT rows of
// one expert, rounded up to 16 only, so an expert's last few rows cost what they are, and the accumulator is the transposed
// output (TMEM lane = feature, column = row).  An expert's rows are cut into equal tiles (170 rows are two tiles of 96 and
// 74, not 160 and 10).  Which tiles there are is known on the device only: every block sums the experts' tiles once and walks
// the tiles t = blockIdx.x, + gridDim.x, ...; feature tiles run fastest, so blocks that run together read the same rows of x.
//   warp 0             TMA producer of the weights: 128 x 64 slices, 128-byte swizzle
//   warp 1             issues tcgen05.mma (M 128, N = the tile's rows, K 16); owns the TMEM allocation
//   the next 4 or 8    epilogue: tcgen05.ld, activation, stores; two accumulators alternate, so it runs under the next tile.  Eight
//                      warps for tiles of 96 rows and more, four for each half of the columns
//   the last 4 or 8    producers of the rows where these are gathered (GATHER): cp.async, 16 bytes each, by source row straight
//                      into the swizzled stage; a stage is announced kLag stages later, when its copies have landed.
//                      Rows that lie sorted in memory are copied by warp 0 as well, in TMA boxes of half a tile (32 rows in small ones)
// Producer and issuer walk their loops as whole warps and one elected lane issues: a lone lane took 520 cycles to wait for a stage and
// issue its four products (N 128 takes the tensor core 256), and 590 to issue a sorted stage's copies.
// (Sorting the rows of the first product in a pass of its own, so that TMA could copy them too, gained 12 us in the product and
// cost 12 in the pass.)
//
// What bounds it: a prompt reads every expert's weights once (134 MB a product at 32 experts of 1024 on rows of 2048: 21 us) and
// then brings 32 KB of weights and rows to an SM for every 128 x 128 x 64 product (256 cycles of the tensor core): 2,048 tokens x 4
// choices, 2048 -> 1024, gathered: 57 us warm (69 with a lone lane's loops and the unrolled epilogue).  A decode step streams the chosen
// experts' weights with 144 KB of them on their way per SM (180 with the token rows): eight tokens x 4, gate and up of 1024 on 2048:
// 36 us for 176 MB (42 before), down 19 (24).
// Every wait is bounded and reports in error_word, as in gemm_tcgen05.cu.
#include "moe.cuh"
#include "mma.cuh"
#include "cluster.cuh"

namespace tib {

constexpr int kMpM = 128, kMpK = 64;
constexpr int kMpMaxExperts = 1024;
constexpr uint32_t kMpWBytes = kMpM * kMpK * 2;
template <int NT> struct MpShape {
  static constexpr uint32_t kXBytes = NT * kMpK * 2;
  static constexpr uint32_t kStage = kMpWBytes + kXBytes;
  static constexpr int kStages = 200 * 1024 / kStage < 9 ? 200 * 1024 / kStage : 9;
  static constexpr int kLag = NT >= 96 ? 3 : 2;      // stages after which a gathered one is announced
  static constexpr int kStorers = NT >= 96 ? 8 : 4, kThreads = 64 + 32 * kStorers;      // warps of the epilogue; threads without the gather's
  static constexpr int kGather = NT >= 96 ? 256 : 128, kGatherRows = kGather / 8;       // threads of the gather, rows they copy at a time
  static constexpr int kBox = NT >= 96 ? NT / 2 : 32;       // rows of one TMA copy of x
  static constexpr uint32_t kTmemCols = NT <= 32 ? 64 : NT <= 64 ? 128 : NT <= 128 ? 256 : 512;      // two accumulators of NT columns
  static constexpr uint32_t kSmem = 1024 + kStages * kStage + 256 + (kMpMaxExperts + 1) * 4;
};

// (what this thread's cp.async copies left in shared memory becomes visible to the tensor cores)
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

struct MpTile { int expert, first, rows, feature; };

// One warp's 32 features of the tile's columns c0 .. c1 - 1 (c0 a multiple of eight), from tensor memory through the activation to y.
// A loop of eight columns: unrolled over 32, the code was fetched anew for every tile (3,000 cycles for 32 columns; rolled 1,250).
template <int ACT, typename TO>
__device__ __forceinline__ void mp_store(uint32_t tmem, TO* __restrict__ y, int64_t ldy, const MpTile& t, int c0, int c1, int feature, int N, int lane,
                                         const int* __restrict__ order, const MoeEpilogue& ep) {
  constexpr bool kGated = moe_act_gated(ACT);
  // (gated: a lane pair holds (gate, up) of one output for every column; of two columns the even lane finishes the first, the odd lane
  // the second)
  const bool odd = lane & 1;
  const bool in = kGated ? (feature | 1) < N : feature < N;
  TO* dst = y + (size_t)(t.first + c0 + (kGated && odd)) * ldy + (kGated ? feature >> 1 : feature);
  float scale = 1.f;
#pragma unroll 1
  for (int c = c0; c < c1; c += 8) {
    if (ep.row_scale && ((c - c0) & 31) == 0) scale = c + lane < c1 ? ep.row_scale[order[t.first + c + lane]] : 1.f;
    uint32_t raw[8];
    tmem_ld8(tmem + c, raw);
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(raw[j]);
    if (ep.row_scale) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= __shfl_sync(0xffffffffu, scale, ((c - c0) & 31) + j);
    }
    if constexpr (kGated) {
#pragma unroll
      for (int j = 0; j < 8; j += 2, dst += 2 * ldy) {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
        const float g = odd ? got : v[j], u = odd ? v[j + 1] : got;
        if (in && c + j + odd < c1) *dst = from_f32<TO>(moe_gated(g, u, ACT, ep.limit, ep.alpha));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j, dst += ldy)
        if (in && c + j < c1) *dst = from_f32<TO>(moe_act(v[j], ACT));
    }
  }
}

template <int NT, bool GATHER, typename TO>
__global__ void __launch_bounds__(MpShape<NT>::kThreads + (GATHER ? MpShape<NT>::kGather : 0), 1)
moe_product_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                           const __nv_bfloat16* __restrict__ x, int64_t ldx, TO* __restrict__ y, int64_t ldy,
                           const int* __restrict__ offsets, const int* __restrict__ order, int experts, int top, int x_by_pair, int N,
                           int K, MoeEpilogue ep, int* __restrict__ error_word) {
  using S = MpShape<NT>;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* smem_gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + S::kStages * S::kStage;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (S::kStages + s); };
  auto acc_full_bar = [&](int b) { return bars + 8u * (2 * S::kStages + b); };
  auto acc_empty_bar = [&](int b) { return bars + 8u * (2 * S::kStages + 2 + b); };
  const uint32_t tmem_slot = bars + 8u * (2 * S::kStages + 4);
  static_assert(8 * (2 * S::kStages + 4) + 4 <= 256, "the barriers' share of shared memory");
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - base));
  int* tiles_before = reinterpret_cast<int*>(smem_gen + (bars - base) + 256);      // [experts + 1]

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      mbar_init(full_bar(s), GATHER ? 1 + S::kGather / 32 : 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full_bar(b), 1);
      mbar_init(acc_empty_bar(b), S::kStorers);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tmem_slot), "r"(S::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  pdl_wait();
  pdl_trigger();
  if (warp == 0) {      // the experts' row tiles, summed
    int before = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
      const int e = e0 + lane;
      int sum = e < experts ? (offsets[e + 1] - offsets[e] + NT - 1) / NT : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += up;
      }
      if (e < experts) tiles_before[e + 1] = before + sum;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) tiles_before[0] = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem_base = *tmem_slot_ptr;

  const int k_blocks = (K + kMpK - 1) / kMpK, f_tiles = (N + kMpM - 1) / kMpM;
  const int num_tiles = tiles_before[experts] * f_tiles;
  auto tile_of = [&](int t) {
    const int row_tile = t / f_tiles;
    int lo = 0, hi = experts;                    // tiles_before[lo] <= row_tile < tiles_before[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tiles_before[mid] <= row_tile) lo = mid; else hi = mid;
    }
    const int first = offsets[lo], n = offsets[lo + 1] - first;
    const int tiles = tiles_before[lo + 1] - tiles_before[lo];
    const int per = ((n + tiles - 1) / tiles + 15) & ~15;      // (at most NT, and the last tile is not empty)
    const int j = row_tile - tiles_before[lo];
    MpTile m;
    m.expert = lo;
    m.first = first + j * per;
    m.rows = min(per, n - j * per);
    m.feature = (t - row_tile * f_tiles) * kMpM;
    return m;
  };

  if (warp == 0) {
    const uint32_t leader = umma_leader();
    uint32_t s = 0, phase = 1;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const MpTile m = tile_of(t);
      const int row = m.expert * N + m.feature;      // (a tile may reach into the next expert's features: such lanes are never stored)
      const int boxes = GATHER ? 0 : (m.rows + S::kBox - 1) / S::kBox;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_warp(empty_bar(s), phase)) {
          if (error_word && leader) atomicExch(error_word, 0x7C0061);
          ok = false;
          break;
        }
        if (leader) {
          const uint32_t stage = base + s * S::kStage;
          mbar_expect_tx(full_bar(s), kMpWBytes + boxes * S::kBox * kMpK * 2);
          tma_load_2d(stage, &map_w, kb * kMpK, row, full_bar(s));
#pragma unroll
          for (int i = 0; i < NT / S::kBox; ++i)      // (likewise a last box into the next tile's rows, or past the matrix)
            if (i < boxes) tma_load_2d(stage + kMpWBytes + i * S::kBox * kMpK * 2, &map_x, kb * kMpK, m.first + i * S::kBox, full_bar(s));
        }
        if (++s == S::kStages) { s = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = umma_leader();
    uint32_t s = 0, phase = 0;
    bool ok = true;
    int j = 0;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++j) {
      const MpTile m = tile_of(t);
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((m.rows + 15) >> 4) << 18) | ((uint32_t)(kMpM >> 4) << 24);
      const int b = j & 1;
      if (!mbar_wait_warp(acc_empty_bar(b), ((j >> 1) & 1) ^ 1)) {
        if (error_word && leader) atomicExch(error_word, 0x7C0064);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_warp(full_bar(s), phase)) {
          if (error_word && leader) atomicExch(error_word, 0x7C0062);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t w_src = umma_low_k128(base + s * S::kStage), x_src = w_src + (kMpWBytes >> 4);
#pragma unroll
        for (int k = 0; k < kMpK / 16; ++k) umma_warp(leader, tmem_base + b * NT, w_src + k * 2, x_src + k * 2, idesc, (kb | k) != 0);
        if (leader) umma_commit(empty_bar(s));
        if (++s == S::kStages) { s = 0; phase ^= 1; }
      }
      if (leader) umma_commit(acc_full_bar(b));      // (also on failure, so that the epilogue does not wait in vain)
    }
  } else if (warp < 2 + S::kStorers) {
    // (with eight warps, four take the tile's first columns and four the others)
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    int j = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++j) {
      const MpTile m = tile_of(t);
      const int b = j & 1, feature = m.feature + quarter * 32 + lane;
      const int middle = S::kStorers == 8 ? ((m.rows >> 1) + 7) & ~7 : m.rows;
      const int c0 = half ? middle : 0, c1 = half ? m.rows : min(middle, m.rows);
      if (!mbar_wait_warp(acc_full_bar(b), (j >> 1) & 1)) {
        if (error_word && lane == 0) atomicExch(error_word, 0x7C0063);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + b * NT;
      if (c0 < c1) {
        switch (ep.act) {
          case MOE_ACT_NONE: mp_store<MOE_ACT_NONE>(acc, y, ldy, m, c0, c1, feature, N, lane, order, ep); break;
          case MOE_ACT_RELU2: mp_store<MOE_ACT_RELU2>(acc, y, ldy, m, c0, c1, feature, N, lane, order, ep); break;
          case MOE_ACT_SILU: mp_store<MOE_ACT_SILU>(acc, y, ldy, m, c0, c1, feature, N, lane, order, ep); break;
          case MOE_ACT_GELU: mp_store<MOE_ACT_GELU>(acc, y, ldy, m, c0, c1, feature, N, lane, order, ep); break;
          case MOE_ACT_GLU_CLAMP: mp_store<MOE_ACT_GLU_CLAMP>(acc, y, ldy, m, c0, c1, feature, N, lane, order, ep); break;
          default: mp_store<MOE_ACT_SWIGLU>(acc, y, ldy, m, c0, c1, feature, N, lane, order, ep); break;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty_bar(b));
    }
  } else if constexpr (GATHER) {
    // row r = r0 + kGatherRows i of the tile, 16-byte piece c of its 128 bytes; the swizzle of a row depends on r % 8 = r0 % 8
    const int g = threadIdx.x - S::kThreads, r0 = g >> 3, c = g & 7;
    const uint32_t dst0 = kMpWBytes + r0 * 128 + ((c ^ (r0 & 7)) << 4);
    uint32_t it = 0, s = 0, phase = 1, ready = 0;      // (ready: the next stage to announce)
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const MpTile m = tile_of(t);
      const __nv_bfloat16* src[NT / S::kGatherRows];
#pragma unroll
      for (int i = 0; i < NT / S::kGatherRows; ++i) {
        const int r = m.first + min(r0 + S::kGatherRows * i, m.rows - 1);
        src[i] = x + (size_t)(x_by_pair ? order[r] / top : r) * ldx + c * 8;
      }
      for (int kb = 0; kb < k_blocks; ++kb, ++it) {
        if (!mbar_wait_warp(empty_bar(s), phase)) {
          if (error_word) atomicExch(error_word, 0x7C0065);
          ok = false;
          break;
        }
        const bool in = kb * kMpK + c * 8 < K;      // (k beyond the rows: zeros, as the weights' copies have there)
        unsigned char* dst = smem_gen + s * S::kStage + dst0;
#pragma unroll
        for (int i = 0; i < NT / S::kGatherRows; ++i)
          if (r0 + S::kGatherRows * i < m.rows) cp_async16(dst + i * S::kGatherRows * 128, in ? src[i] + kb * kMpK : x, in);      // (columns behind the rows are never stored)
        cp_async_commit();
        if (++s == S::kStages) { s = 0; phase ^= 1; }
        if (it >= S::kLag) {
          cp_async_wait<S::kLag>();
          fence_async_shared();
          __syncwarp();
          if (lane == 0) mbar_arrive(full_bar(ready));
          if (++ready == S::kStages) ready = 0;
        }
      }
    }
    cp_async_wait<0>();
    fence_async_shared();
    __syncwarp();
    for (uint32_t late = it >= S::kLag ? it - S::kLag : 0; late < it; ++late) {
      if (lane == 0) mbar_arrive(full_bar(ready));
      if (++ready == S::kStages) ready = 0;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(S::kTmemCols) : "memory");
  }
}

struct MpArgs {
  CUtensorMap map_w, map_x;
  const __nv_bfloat16* x;
  int64_t ldx;
  void* y;
  int64_t ldy;
  const int* offsets;
  const int* order;
  int pairs, experts, top, x_by_pair, N, K;
  MoeEpilogue ep;
  int* error_word;
};

template <int NT, bool GATHER, typename TO>
static int launch_moe_product(MpArgs& a, cudaStream_t stream) {
  auto kern = moe_product_tcgen05_kernel<NT, GATHER, TO>;
  a.map_x = a.map_w;      // (unused when gathered)
  if (!GATHER) {
    const int rc = make_map(&a.map_x, a.x, a.pairs, a.K, a.ldx, MpShape<NT>::kBox);
    if (rc != TIB_OK) return rc;
  }
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MpShape<NT>::kSmem);
  if (e != cudaSuccess) return (int)e;
  const int64_t most = ((int64_t)a.pairs / NT + (a.pairs < a.experts ? a.pairs : a.experts)) * ceil_div(a.N, kMpM);
  TIB_LAUNCH_DEPENDENT(kern, (int)(most < 148 ? most : 148), MpShape<NT>::kThreads + (GATHER ? MpShape<NT>::kGather : 0), MpShape<NT>::kSmem, stream, a.map_w, a.map_x,
                       a.x, a.ldx, (TO*)a.y, a.ldy, a.offsets, a.order, a.experts, a.top, a.x_by_pair, a.N, a.K, a.ep, a.error_word);
  return TIB_OK;
}

bool moe_product_tcgen05_takes(const void* x, int64_t ldx, const void* w, int experts, int N, int K) {
  return K % 8 == 0 && ldx % 8 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 && experts <= kMpMaxExperts &&
         (int64_t)experts * N < 0x7fffffff - kMpM;
}

int moe_product_tcgen05(const void* x, int64_t ldx, const void* w, void* y, int y_dtype, int64_t ldy, const int* offsets, const int* order,
                        int pairs, int experts, int top, int x_by_pair, int N, int K, const MoeEpilogue& ep, int* error_word,
                        cudaStream_t stream) {
  MpArgs a;
  int rc = make_map(&a.map_w, w, experts * N, K, K, kMpM);
  if (rc != TIB_OK) return rc;
  a.x = (const __nv_bfloat16*)x; a.ldx = ldx; a.y = y; a.ldy = ldy; a.offsets = offsets; a.order = order; a.pairs = pairs;
  a.experts = experts; a.top = top; a.x_by_pair = x_by_pair; a.N = N; a.K = K; a.ep = ep; a.error_word = error_word;
  // Rows of an expert on average: the smallest tile that mostly holds them all, up to 160 rows.  (The whole layer on 2,048
  // tokens, 256 rows an expert, with tiles of 32 / 64 / 96 / 128 / 160 / 192 / 256 rows: 414 / 294 / 264 / 255 / 250 / 250 / 261 us;
  // on eight tokens, a row or two an expert: 98 / 97 / 99 / 99 / 101 / 103 / 110.)
  const int average = ceil_div(pairs, experts);
#define TIB_MP_GO(NT)                                                                                                          \
  (y_dtype == TIB_BF16 ? (x_by_pair ? launch_moe_product<NT, true, __nv_bfloat16>(a, stream) : launch_moe_product<NT, false, __nv_bfloat16>(a, stream)) \
                       : (x_by_pair ? launch_moe_product<NT, true, float>(a, stream) : launch_moe_product<NT, false, float>(a, stream)))
  if (average <= 24) return TIB_MP_GO(32);
  if (average <= 48) return TIB_MP_GO(64);
  if (average <= 80) return TIB_MP_GO(96);
  return TIB_MP_GO(160);
#undef TIB_MP_GO
}

}  // namespace tib
