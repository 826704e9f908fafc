// The experts' products over the sorted (token, choice) rows on the 5th-generation tensor cores (bf16 operands, fp32 sums):
//     y[s] = act(x[source of s] . W_e^T)    for the rows s of expert e, W: [experts, N, K]
//
// The weights are the 128-row operand of the MMA and the sorted rows its N dimension: a tile is 128 features x up to NT rows of
// one expert, rounded up to 16 only, so an expert's last few rows cost what they are, and the accumulator is the transposed
// output (TMEM lane = feature, column = row).  An expert's rows are cut into equal tiles (170 rows are two tiles of 96 and
// 74, not 160 and 10).  Which tiles there are is known on the device only: every block sums the experts' tiles once and walks
// the tiles t = blockIdx.x, + gridDim.x, ...; feature tiles run fastest, so blocks that run together read the same rows of x.
//   warp 0, one lane   TMA producer of the weights: 128 x 64 slices, 128-byte swizzle
//   warp 1, one lane   issues tcgen05.mma (M 128, N = the tile's rows, K 16); owns the TMEM allocation
//   warps 2..5         epilogue: tcgen05.ld, activation, stores; two accumulators alternate, so it runs under the next tile
//   warps 6..9         producers of the rows where these are gathered (GATHER): cp.async, 16 bytes each, by source row straight
//                      into the swizzled stage; a stage is announced two stages later, when its copies have landed.
//                      Rows that lie sorted in memory are copied by warp 0 as well, in TMA boxes of 32 rows
// (Sorting the rows of the first product in a pass of its own, so that TMA could copy them too, gained 12 us in the product and
// cost 12 in the pass.)
//
// What bounds it: a prompt reads every expert's weights once (134 MB a product at 32 experts of 1024 on rows of 2048: 21 us) and
// multiplies at the rate shared memory feeds 128 x 128 x 16 products; 2,048 tokens x 4 choices take 68 us gathered and 62 sorted where
// the mma.sync kernel before took 199 and 207 (cold).  A decode step streams the chosen experts' weights with 144 KB of them on their
// way per SM (180 with the token rows): eight tokens x 4, gate and up of 1024 on 2048: 42 us for 176 MB (68 before), down 24 (38).
// Every wait is bounded and reports in error_word, as in gemm_tcgen05.cu.
#include "moe.cuh"
#include "mma.cuh"
#include "cluster.cuh"

namespace tib {

constexpr int kMpM = 128, kMpK = 64, kMpThreads = 192, kMpGather = 128, kMpLag = 2, kMpBox = 32;
constexpr int kMpMaxExperts = 1024;
constexpr uint32_t kMpWBytes = kMpM * kMpK * 2;
template <int NT> struct MpShape {
  static constexpr uint32_t kXBytes = NT * kMpK * 2;
  static constexpr uint32_t kStage = kMpWBytes + kXBytes;
  static constexpr int kStages = 200 * 1024 / kStage < 9 ? 200 * 1024 / kStage : 9;
  static constexpr uint32_t kTmemCols = NT <= 32 ? 64 : NT <= 64 ? 128 : NT <= 128 ? 256 : 512;      // two accumulators of NT columns
  static constexpr uint32_t kSmem = 1024 + kStages * kStage + 256 + (kMpMaxExperts + 1) * 4;
};

// (what this thread's cp.async copies left in shared memory becomes visible to the tensor cores)
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

struct MpTile { int expert, first, rows, feature; };

// Stores columns c0 .. c0 + 31 (rows of the tile) of one warp's 32 features.
template <int ACT, typename TO>
__device__ __forceinline__ void mp_store(const uint32_t (&v)[32], TO* __restrict__ y, int64_t ldy, const MpTile& t, int c0, int feature, int N,
                                         int lane, float scale_lane, const MoeEpilogue& ep) {
  if constexpr (moe_act_gated(ACT)) {
    // a lane pair holds (gate, up) of one output for every column: of two columns the even lane finishes the first, the odd
    // lane the second
    const bool odd = lane & 1;
    const bool in = (feature | 1) < N;
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float send = __uint_as_float(odd ? v[j] : v[j + 1]);
      const float got = __shfl_xor_sync(0xffffffffu, send, 1);
      const float rs = __shfl_sync(0xffffffffu, scale_lane, j + (odd ? 1 : 0));
      const float g = odd ? got : __uint_as_float(v[j]), u = odd ? __uint_as_float(v[j + 1]) : got;
      const int col = c0 + j + (odd ? 1 : 0);
      if (in && col < t.rows)
        y[(size_t)(t.first + col) * ldy + (feature >> 1)] = from_f32<TO>(moe_gated(g * rs, u * rs, ACT, ep.limit, ep.alpha));
    }
  } else {
    const bool in = feature < N;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float rs = __shfl_sync(0xffffffffu, scale_lane, j);
      if (in && c0 + j < t.rows) y[(size_t)(t.first + c0 + j) * ldy + feature] = from_f32<TO>(moe_act(__uint_as_float(v[j]) * rs, ACT));
    }
  }
}

template <int NT, bool GATHER, typename TO>
__global__ void __launch_bounds__(kMpThreads + (GATHER ? kMpGather : 0), 1)
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

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      mbar_init(full_bar(s), GATHER ? 1 + kMpGather : 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full_bar(b), 1);
      mbar_init(acc_empty_bar(b), 4);
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
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        const MpTile m = tile_of(t);
        const int row = m.expert * N + m.feature;      // (a tile may reach into the next expert's features: such lanes are never stored)
        const int boxes = GATHER ? 0 : (m.rows + kMpBox - 1) / kMpBox;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % S::kStages;
          if (!mbar_wait(empty_bar(s), ((it / S::kStages) & 1) ^ 1)) {
            if (error_word) atomicExch(error_word, 0x7C0061);
            ok = false;
            break;
          }
          mbar_expect_tx(full_bar(s), kMpWBytes + boxes * kMpBox * kMpK * 2);
          tma_load_2d(base + s * S::kStage, &map_w, kb * kMpK, row, full_bar(s));
          for (int i = 0; i < boxes; ++i)      // (likewise a last box into the next tile's rows, or past the matrix)
            tma_load_2d(base + s * S::kStage + kMpWBytes + i * kMpBox * kMpK * 2, &map_x, kb * kMpK, m.first + i * kMpBox, full_bar(s));
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      int j = 0;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++j) {
        const MpTile m = tile_of(t);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((m.rows + 15) >> 4) << 18) | ((uint32_t)(kMpM >> 4) << 24);
        const int b = j & 1;
        if (!mbar_wait(acc_empty_bar(b), ((j >> 1) & 1) ^ 1)) {
          if (error_word) atomicExch(error_word, 0x7C0064);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % S::kStages;
          if (!mbar_wait(full_bar(s), (it / S::kStages) & 1)) {
            if (error_word) atomicExch(error_word, 0x7C0062);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint32_t w_src = base + s * S::kStage, x_src = w_src + kMpWBytes;
#pragma unroll
          for (int k = 0; k < kMpK / 16; ++k)
            umma_f16_idesc(tmem_base + b * NT, umma_desc_k128(w_src + k * 32), umma_desc_k128(x_src + k * 32), idesc, (kb | k) != 0);
          umma_commit(empty_bar(s));
        }
        umma_commit(acc_full_bar(b));      // (also on failure, so that the epilogue does not wait in vain)
      }
    }
  } else if (warp < 6) {
    const int quarter = warp & 3;
    int j = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++j) {
      const MpTile m = tile_of(t);
      const int b = j & 1, feature = m.feature + quarter * 32 + lane;
      if (!mbar_wait(acc_full_bar(b), (j >> 1) & 1)) {
        if (error_word && lane == 0) atomicExch(error_word, 0x7C0063);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
      for (int c0 = 0; c0 < m.rows; c0 += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + b * NT + c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        const float scale = ep.row_scale && c0 + lane < m.rows ? ep.row_scale[order[m.first + c0 + lane]] : 1.f;
        switch (ep.act) {
          case MOE_ACT_NONE: mp_store<MOE_ACT_NONE>(v, y, ldy, m, c0, feature, N, lane, scale, ep); break;
          case MOE_ACT_RELU2: mp_store<MOE_ACT_RELU2>(v, y, ldy, m, c0, feature, N, lane, scale, ep); break;
          case MOE_ACT_SILU: mp_store<MOE_ACT_SILU>(v, y, ldy, m, c0, feature, N, lane, scale, ep); break;
          case MOE_ACT_GELU: mp_store<MOE_ACT_GELU>(v, y, ldy, m, c0, feature, N, lane, scale, ep); break;
          case MOE_ACT_GLU_CLAMP: mp_store<MOE_ACT_GLU_CLAMP>(v, y, ldy, m, c0, feature, N, lane, scale, ep); break;
          default: mp_store<MOE_ACT_SWIGLU>(v, y, ldy, m, c0, feature, N, lane, scale, ep); break;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty_bar(b));
    }
  } else if constexpr (GATHER) {
    // row r = r0 + 16 i of the tile, 16-byte piece c of its 128 bytes; the swizzle of a row depends on r % 8 = r0 % 8
    const int g = threadIdx.x - kMpThreads, r0 = g >> 3, c = g & 7;
    const uint32_t dst0 = kMpWBytes + r0 * 128 + ((c ^ (r0 & 7)) << 4);
    uint32_t it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const MpTile m = tile_of(t);
      const __nv_bfloat16* src[NT / 16];
#pragma unroll
      for (int i = 0; i < NT / 16; ++i) {
        const int s = m.first + min(r0 + 16 * i, m.rows - 1);
        src[i] = x + (size_t)(x_by_pair ? order[s] / top : s) * ldx + c * 8;
      }
      for (int kb = 0; kb < k_blocks; ++kb, ++it) {
        const int s = it % S::kStages;
        if (!mbar_wait(empty_bar(s), ((it / S::kStages) & 1) ^ 1)) {
          if (error_word) atomicExch(error_word, 0x7C0065);
          ok = false;
          break;
        }
        const bool in = kb * kMpK + c * 8 < K;      // (k beyond the rows: zeros, as the weights' copies have there)
        unsigned char* dst = smem_gen + s * S::kStage + dst0;
#pragma unroll
        for (int i = 0; i < NT / 16; ++i)
          if (r0 + 16 * i < m.rows) cp_async16(dst + i * 2048, in ? src[i] + kb * kMpK : x, in);      // (columns behind the rows are never stored)
        cp_async_commit();
        if (it >= kMpLag) {
          cp_async_wait<kMpLag>();
          fence_async_shared();
          mbar_arrive(full_bar((it - kMpLag) % S::kStages));
        }
      }
    }
    cp_async_wait<0>();
    fence_async_shared();
    for (uint32_t late = it >= kMpLag ? it - kMpLag : 0; late < it; ++late) mbar_arrive(full_bar(late % S::kStages));
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
static int launch_moe_product(const MpArgs& a, cudaStream_t stream) {
  auto kern = moe_product_tcgen05_kernel<NT, GATHER, TO>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MpShape<NT>::kSmem);
  if (e != cudaSuccess) return (int)e;
  const int64_t most = ((int64_t)a.pairs / NT + (a.pairs < a.experts ? a.pairs : a.experts)) * ceil_div(a.N, kMpM);
  TIB_LAUNCH_DEPENDENT(kern, (int)(most < 148 ? most : 148), kMpThreads + (GATHER ? kMpGather : 0), MpShape<NT>::kSmem, stream, a.map_w, a.map_x,
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
  if (rc == TIB_OK) rc = x_by_pair ? make_map(&a.map_x, w, experts * N, K, K, kMpBox) : make_map(&a.map_x, x, pairs, K, ldx, kMpBox);      // (unused when gathered)
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
