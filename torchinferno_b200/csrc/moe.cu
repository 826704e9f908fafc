// Routed feed-forward (mixture of experts): routing, grouping of (token, choice) pairs by expert, the experts'
// two products over the grouped rows, and the weighted sum back per token.  Nothing here returns to the host:
// every count and offset stays on the device and grids are sized for the worst case, so a step can be captured.
//
//   moe_route    from fp32 router logits [tokens, ld]: softmax over the experts (or sigmoid), the `top` largest
//                scores (lowest index first among equals), their weights = score / (sum of the chosen + norm_eps)
//                (or the bare scores), all fp32; optionally a correction per expert that counts for the choice only, and
//                groups of neighbouring experts of which only the best few may be chosen from
//   moe_group    counting sort of the tokens * top pairs by expert: offsets [experts + 1], order[sorted] = pair,
//                place[pair] = sorted index.  The order inside an expert may differ from run to run; every row
//                of a product is computed by itself, so no value depends on it
//   moe_expert_product   y[s] = act(x[src(s)] . W_e^T) for the sorted rows s of expert e; W: [experts, n, k];
//                act: none, relu^2, silu, gelu (the erf form), or a clamped gated unit over (gate, up) row pairs of W (row 2i = gate i,
//                row 2i + 1 = up i): g = min(g, limit), u = clamp(u, -limit, limit), y_i = g * sigmoid(alpha * g) * (u + 1),
//                or the plain gated unit y_i = silu(g) * u over the same pairs; either leaves n / 2 columns.  `row_scale` (per pair, may be null) multiplies the fp32 sums before the
//                activation: a router weight that belongs on the expert's input.  bf16 operands whose rows are 16-byte aligned run on the tensor cores
//                (moe_tcgen05.cu, fp32 accumulation); everything else, and the 32-bit path, on fp32 FMAs in fixed k order
//   moe_combine  out[t] = sum_k weight[t, k] * y[place[t * top + k]]  (+ sigmoid(gate[t]) * shared[t]); weights may be null (1);
//                a choice whose id is `identity_from` or above has no expert: it adds weight * x[t], the input itself
#include "moe.cuh"
#include <math_constants.h>

namespace tib {

// ----------------------------------------------------------- router logits
// out[t, e] = x[t] . w[e] (+ bias[e]) in fp32 for a handful of rows w (the router, perhaps a gate row behind it): one warp per
// row and group of tokens, lanes stride over k (eight at a time where rows are 16-byte aligned), then a butterfly sum per
// token: the order of every sum is fixed by k and the alignment alone, so a token's logits do not depend on what else is
// in the step.  (The general fp32 product gives a product
// this narrow to a single block.)
// A block takes four tokens, so that a row of w read from the L2 serves several of them.  With 16-byte aligned
// rows (VEC) a lane takes eight consecutive k at a time: 16 bytes of a bf16 token row, 32 bytes of w.
constexpr int kRouterTokens = 4;

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const float2 a = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  const float2 c = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&raw.z)), d = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&raw.w));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}

// DENSE: fewer registers (bf16 rows 64 for 74, four blocks an SM for three; fp32 rows 50 for 60), by one clamp of an index, which has the compiler keep fewer
// addresses and loads.  With one block an SM the more loads are ahead; beyond that it goes by how the blocks fall into rounds.  16 rows of 4,096, bf16, us,
// dense and not, by blocks on the fullest SM: one 6.0 and 5.5 (200 tokens), two 6.6 and 8.5 (500), three 10.7 and 8.6 (600), four 10.9 and 15.9 (1,180); fp32
// rows of 2,048, 16 of them: one 6.0 and 4.7, two 7.7 and 7.3, 24 of them 7.7 and 8.4, 12 of them 6.5 and 7.8, four 12.7 and 12.8.
template <typename TX, bool VEC, bool DENSE>
__global__ void __launch_bounds__(256)
router_logits_kernel(const TX* __restrict__ x, int64_t ldx, const float* __restrict__ w, const float* __restrict__ bias,
                     float* __restrict__ out, int64_t ldo, int tokens, int rows, int K) {
  pdl_wait();
  pdl_trigger();
  constexpr int TOK = kRouterTokens;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int t0 = blockIdx.x * TOK;
  const int nt = min(TOK, tokens - t0);
  const int K8 = VEC ? (K / 8) * 8 : 0;
  const auto work = [&](int e, int row) {
    float acc[TOK];
#pragma unroll
    for (int i = 0; i < TOK; ++i) acc[i] = 0.f;
    if (VEC) {
      // (small steps wait for loads: 12 us for eight tokens of 2,048 with one round's in flight, 7.4 with four rounds')
#pragma unroll 4
      for (int k = lane * 8; k < K8; k += 256) {
        float wv[8];
        load8(w + (size_t)row * K + k, wv);
#pragma unroll
        for (int i = 0; i < TOK; ++i) {
          float xv[8];
          load8(x + (size_t)(t0 + min(i, nt - 1)) * ldx + k, xv);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i] = fmaf(xv[j], wv[j], acc[i]);
        }
      }
    }
    for (int k = K8 + lane; k < K; k += 32) {
      const float wv = w[(size_t)e * K + k];
#pragma unroll
      for (int i = 0; i < TOK; ++i)
        if (i < nt) acc[i] = fmaf(to_f32(x[(size_t)(t0 + i) * ldx + k]), wv, acc[i]);
    }
#pragma unroll
    for (int i = 0; i < TOK; ++i) {
      const float v = warp_sum(acc[i]);
      if (lane == 0 && i < nt) out[(size_t)(t0 + i) * ldo + e] = bias ? v + bias[e] : v;
    }
  };
  if constexpr (DENSE) {
    const int stride = nwarps * gridDim.y;
    for (int e = warp + blockIdx.y * nwarps; e < rows; e += stride) work(e, min(e, rows - 1));
  } else {
    for (int e = warp + blockIdx.y * nwarps; e < rows; e += nwarps * gridDim.y) work(e, e);
  }
}

// The same sums for large steps with 16-byte aligned rows: a warp works six rows of w on eight tokens, two tokens an instruction (packed fp32), so a
// piece of w serves eight tokens and an element is widened for six rows; what it loads and widens is a third of its instructions.  (A lane's sums
// run over k in the kernel above's order, and the sum over lanes is its butterfly, whose two halves of a pair add the same two numbers.)  What bounds
// it: the loads of a step wait for one another's registers (two blocks of six warps an SM), then the fp32 pipe.  2,048 tokens of 2,048, one call after another,
// everything in the L2: 17 rows 8.6 us, 33 12.4; 1,300 tokens, 129 rows 27, 513 88 (33 rows in a running layer, behind the kernel that wrote the tokens, 20);
// five rows of whole warps of eight and scalar products 13.6, 19.8, 72 and 246 (24 in the layer); rows and tokens through shared memory 27 to 50 in the layer.
constexpr int kRouterRows = 6, kRouterMany = 8, kRouterWarps = 6;

__device__ __forceinline__ void load8_pairs(const float* a, const float* b, f32x2 (&v)[8]) {
  float x[8], y[8];
  load8(a, x);
  load8(b, y);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = f2_pack(x[j], y[j]);
}
__device__ __forceinline__ void load8_pairs(const __nv_bfloat16* a, const __nv_bfloat16* b, f32x2 (&v)[8]) {
  const uint4 p = *reinterpret_cast<const uint4*>(a), q = *reinterpret_cast<const uint4*>(b);
  const uint32_t x[4] = {p.x, p.y, p.z, p.w}, y[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = f2_pack(__uint_as_float(x[i] << 16), __uint_as_float(y[i] << 16));
    v[2 * i + 1] = f2_pack(__uint_as_float(x[i] & 0xffff0000u), __uint_as_float(y[i] & 0xffff0000u));
  }
}

// grid (runs of kRouterMany tokens, runs of rows: kRouterRows a warp)
template <typename TX>
__global__ void __launch_bounds__(kRouterWarps * 32)
router_logits_many_kernel(const TX* __restrict__ x, int64_t ldx, const float* __restrict__ w, const float* __restrict__ bias,
                          float* __restrict__ out, int64_t ldo, int tokens, int rows, int K) {
  constexpr int TOK = kRouterMany, R = kRouterRows;
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, e0 = (blockIdx.y * warps + (threadIdx.x >> 5)) * R;
  const int t0 = blockIdx.x * TOK, nt = min(TOK, tokens - t0), K8 = K / 8 * 8;
  if (e0 >= rows) return;
  const float* row[R];
  const TX* token[TOK];
#pragma unroll
  for (int r = 0; r < R; ++r) row[r] = w + (size_t)min(e0 + r, rows - 1) * K;      // (a row or token too many is not stored)
#pragma unroll
  for (int i = 0; i < TOK; ++i) token[i] = x + (size_t)(t0 + min(i, nt - 1)) * ldx;
  f32x2 acc[R][TOK / 2];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < TOK / 2; ++i) acc[r][i] = f2_pack(0.f, 0.f);
#pragma unroll 1
  for (int k = lane * 8; k < K8; k += 256) {
    float wv[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r) load8(row[r] + k, wv[r]);
#pragma unroll
    for (int i = 0; i < TOK / 2; ++i) {
      f32x2 xv[8];
      load8_pairs(token[2 * i] + k, token[2 * i + 1] + k, xv);
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r][i] = f2_fma(xv[j], f2_pack(wv[r][j], wv[r][j]), acc[r][i]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int e = e0 + r;
    if (e >= rows) break;
    float own[TOK];
#pragma unroll
    for (int i = 0; i < TOK / 2; ++i) f2_unpack(acc[r][i], own[2 * i], own[2 * i + 1]);
    for (int k = K8 + lane; k < K; k += 32) {
      const float wv = w[(size_t)e * K + k];
#pragma unroll
      for (int i = 0; i < TOK; ++i)
        if (i < nt) own[i] = fmaf(to_f32(x[(size_t)(t0 + i) * ldx + k]), wv, own[i]);
    }
    // the sums over the lanes: at each of three steps a lane hands on the half of its tokens that its partner keeps
#pragma unroll
    for (int half = TOK / 2; half > 0; half /= 2) {
      const bool upper = lane & (4 * half);
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float give = upper ? own[i] : own[i + half], keep = upper ? own[i + half] : own[i];
        own[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * half);
      }
    }
    float v = own[0];
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    const int i = lane >> 2;
    if ((lane & 3) == 0 && i < nt) out[(size_t)(t0 + i) * ldo + e] = bias ? v + bias[e] : v;
  }
}

// ------------------------------------------------------------------- route
// One warp per token.  score(e) = softmax(z)[e] or sigmoid(z[e]); the choice looks at score + correction[e] (when a
// correction is given) and, with `groups` > 1, only at the experts of the `keep` runs of adjacent experts whose best
// corrected score ranks highest (an expert of another run is not eligible, whatever its score); the weights are made from the
// scores without the correction.  Lowest index first among equals, for groups and for experts.
constexpr int kRouteMaxGroups = 64;      // (two groups a lane)

struct MoeRouteArgs {
  const float* logits; int64_t ld;
  int experts, top, sigmoid_scores, normalize;
  float norm_eps;
  const float* correction;
  int groups, keep;
  int* ids; float* weights;
  int tokens;
};

// One token, by a whole warp; kept: this warp's place for the kept groups.
__device__ __forceinline__ void moe_route_token(const MoeRouteArgs& r, int t, unsigned char* kept) {
  const float* __restrict__ logits = r.logits;
  const float* __restrict__ correction = r.correction;
  const int64_t ld = r.ld;
  const int experts = r.experts, top = r.top, sigmoid_scores = r.sigmoid_scores, normalize = r.normalize, groups = r.groups, keep = r.keep;
  const float norm_eps = r.norm_eps;
  int* __restrict__ ids = r.ids;
  float* __restrict__ weights = r.weights;
  const int lane = threadIdx.x & 31;
  const float* z = logits + (size_t)t * ld;
  float mx = -CUDART_INF_F;
  for (int e = lane; e < experts; e += 32) mx = fmaxf(mx, z[e]);
  mx = warp_max(mx);
  float sum = 0.f;
  for (int e = lane; e < experts; e += 32) sum += expf(z[e] - mx);
  sum = warp_sum(sum);
  auto score = [&](int e) { return sigmoid_scores ? 1.f / (1.f + expf(-z[e])) : expf(z[e] - mx) / sum; };
  const bool grouped = groups > 1 && keep < groups;
  const int per_group = grouped ? experts / groups : experts;
  if (grouped) {
    float gscore[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int g = lane + 32 * i;
      gscore[i] = -CUDART_INF_F;
      if (g < groups) {
        kept[g] = 0;
        for (int e = g * per_group; e < (g + 1) * per_group; ++e)
          gscore[i] = fmaxf(gscore[i], score(e) + (correction ? correction[e] : 0.f));
      }
    }
    __syncwarp();
    unsigned taken = 0u;
    for (int k = 0; k < keep; ++k) {
      float best = -CUDART_INF_F;
      int best_g = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int g = lane + 32 * i;
        if (g < groups && !((taken >> i) & 1u) && (gscore[i] > best || best_g == 0x7fffffff)) { best = gscore[i]; best_g = g; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int og = __shfl_xor_sync(0xffffffffu, best_g, o);
        if (og != 0x7fffffff && (best_g == 0x7fffffff || ob > best || (ob == best && og < best_g))) { best = ob; best_g = og; }
      }
      if (best_g < groups) {
        if ((best_g & 31) == lane) { taken |= 1u << (best_g >> 5); kept[best_g] = 1; }
      }
    }
    __syncwarp();
  }
  float chosen_sum = 0.f;
  unsigned long long taken_lo = 0ull;    // lane-local mask over this lane's experts (e = lane + 32 * i, i < 64)
  for (int k = 0; k < top; ++k) {
    float best = -CUDART_INF_F, best_s = 0.f;
    int best_e = 0x7fffffff;
    for (int e = lane, i = 0; e < experts; e += 32, ++i) {
      if ((taken_lo >> i) & 1ull) continue;
      if (grouped && !kept[e / per_group]) continue;
      const float s = score(e);
      const float c = s + (correction ? correction[e] : 0.f);
      if (c > best || best_e == 0x7fffffff) { best = c; best_s = s; best_e = e; }     // (rising e: the lowest index wins among equals)
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const float os = __shfl_xor_sync(0xffffffffu, best_s, o);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
      if (oe != 0x7fffffff && (best_e == 0x7fffffff || ob > best || (ob == best && oe < best_e))) { best = ob; best_s = os; best_e = oe; }
    }
    if ((best_e & 31) == lane && best_e < experts) taken_lo |= 1ull << (best_e >> 5);
    chosen_sum += best_s;
    if (lane == 0) { ids[(size_t)t * top + k] = best_e < experts ? best_e : -1; weights[(size_t)t * top + k] = best_e < experts ? best_s : 0.f; }
  }
  __syncwarp();
  if (normalize && lane < top) weights[(size_t)t * top + lane] /= (chosen_sum + norm_eps);
  if (normalize) for (int k = lane + 32; k < top; k += 32) weights[(size_t)t * top + k] /= (chosen_sum + norm_eps);
}

// The same choices and weights, to the bit, of at most 32 S experts without groups and at most 32 choices: a lane works its S scores out once and
// keeps them, and lane k the k-th choice, so that nothing is read back from memory.  2,048 tokens, 4 of 32: 6.8 us behind the logits, 12.2 in the form above.
template <int S>
__device__ __forceinline__ void moe_route_token_few(const MoeRouteArgs& r, int t) {
  const int lane = threadIdx.x & 31;
  const float* z = r.logits + (size_t)t * r.ld;
  float logit[S], score[S], rank[S];
  float mx = -CUDART_INF_F;
#pragma unroll
  for (int i = 0; i < S; ++i) {
    const int e = lane + 32 * i;
    logit[i] = e < r.experts ? z[e] : -CUDART_INF_F;
    if (e < r.experts) mx = fmaxf(mx, logit[i]);
  }
  if (!r.sigmoid_scores) {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < S; ++i) {
      score[i] = expf(logit[i] - mx);
      if (lane + 32 * i < r.experts) sum += score[i];
    }
    sum = warp_sum(sum);
#pragma unroll
    for (int i = 0; i < S; ++i) score[i] = score[i] / sum;
  } else {
#pragma unroll
    for (int i = 0; i < S; ++i) score[i] = 1.f / (1.f + expf(-logit[i]));
  }
#pragma unroll
  for (int i = 0; i < S; ++i) rank[i] = score[i] + (r.correction && lane + 32 * i < r.experts ? r.correction[lane + 32 * i] : 0.f);
  unsigned left = 0u;      // of the lane's experts
#pragma unroll
  for (int i = 0; i < S; ++i) left |= lane + 32 * i < r.experts ? 1u << i : 0u;
  float chosen_sum = 0.f, weight = 0.f;
  int id = -1;
  for (int k = 0; k < r.top; ++k) {
    float best = -CUDART_INF_F, best_s = 0.f;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < S; ++i)
      if ((left >> i & 1u) && (rank[i] > best || best_e == 0x7fffffff)) { best = rank[i]; best_s = score[i]; best_e = lane + 32 * i; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const float os = __shfl_xor_sync(0xffffffffu, best_s, o);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
      if (oe != 0x7fffffff && (best_e == 0x7fffffff || ob > best || (ob == best && oe < best_e))) { best = ob; best_s = os; best_e = oe; }
    }
    if ((best_e & 31) == lane && best_e < r.experts) left &= ~(1u << (best_e >> 5));
    chosen_sum += best_s;
    if (lane == k && best_e < r.experts) { id = best_e; weight = best_s; }
  }
  if (lane < r.top) {
    r.ids[(size_t)t * r.top + lane] = id;
    r.weights[(size_t)t * r.top + lane] = r.normalize ? weight / (chosen_sum + r.norm_eps) : weight;
  }
}

// S: scores a lane keeps, 0: the general form.
static int route_scores_a_lane(const MoeRouteArgs& r) {
  if ((r.groups > 1 && r.keep < r.groups) || r.top > 32) return 0;
  return r.experts <= 32 ? 1 : r.experts <= 64 ? 2 : r.experts <= 256 ? 8 : 0;
}
template <int S> __device__ __forceinline__ void moe_route_one(const MoeRouteArgs& r, int t, unsigned char* kept) {
  if constexpr (S > 0) moe_route_token_few<S>(r, t);
  else moe_route_token(r, t, kept);
}
#define TIB_ROUTE_PICK(S_OF, kernel, ...)                                                        \
  do {                                                                                           \
    switch (S_OF) {                                                                              \
      case 1: TIB_LAUNCH_DEPENDENT(kernel<1>, __VA_ARGS__); break;                               \
      case 2: TIB_LAUNCH_DEPENDENT(kernel<2>, __VA_ARGS__); break;                               \
      case 8: TIB_LAUNCH_DEPENDENT(kernel<8>, __VA_ARGS__); break;                               \
      default: TIB_LAUNCH_DEPENDENT(kernel<0>, __VA_ARGS__);                                     \
    }                                                                                            \
  } while (0)

template <int S>
__global__ void __launch_bounds__(128) moe_route_kernel(MoeRouteArgs r) {
  pdl_wait();
  pdl_trigger();
  __shared__ unsigned char kept_s[4][kRouteMaxGroups];
  const int warp = threadIdx.x >> 5, t = blockIdx.x * (blockDim.x >> 5) + warp;
  if (t < r.tokens) moe_route_one<S>(r, t, kept_s[warp]);
}

// ------------------------------------------------------------------- group
// One block.  counts in shared memory (experts <= 1024), exclusive scan by one warp, then placement with atomics.
__device__ __forceinline__ void moe_group_pairs(const int* ids, int pairs, int experts, int* __restrict__ offsets, int* __restrict__ order,
                                               int* __restrict__ place) {
  __shared__ int count[1024];
  __shared__ int cursor[1024];
  for (int e = threadIdx.x; e < experts; e += blockDim.x) count[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    const int e = ids[p];
    if (e >= 0 && e < experts) atomicAdd(&count[e], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {      // a warp's running sums, 32 experts at a time
    int run = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
      const int e = e0 + (int)threadIdx.x, own = e < experts ? count[e] : 0;
      int upto = own;
#pragma unroll
      for (int step = 1; step < 32; step *= 2) {
        const int below = __shfl_up_sync(0xffffffffu, upto, step);
        if ((int)threadIdx.x >= step) upto += below;
      }
      if (e < experts) { offsets[e] = run + upto - own; cursor[e] = run + upto - own; }
      run += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (threadIdx.x == 0) offsets[experts] = run;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    const int e = ids[p];
    if (e >= 0 && e < experts) {
      const int s = atomicAdd(&cursor[e], 1);
      order[s] = p;
      place[p] = s;
    } else {
      place[p] = -1;
    }
  }
}

// Up to kGroupPairs pairs a thread and kGroupExperts experts: every warp counts its own pairs, whose place among the warp's stays in a register, so
// that ids are read once and no two warps meet in an atomic, at the price of 32 counts an expert to add up.  A kernel of its own, since twice the registers
// make a small call longer; us, one set of counts / a set a warp: 64 pairs over 32 experts 1.7 / 2.6, 4,096 over 32 4.1 / 4.6, 8,192 over 24, 32 and 64
// 6.2 / 6.3, 6.5 / 6.5 (behind the choices 7.8 / 6.5) and 7.5 / 7.3, 16,384 over 16, 32 and 256 8.7 / 9.4, 11.4 / 10.8 and 15.3 / 13.9.
constexpr int kGroupPairs = 16, kGroupExperts = 256;
static bool group_by_warps(int pairs, int experts) { return pairs >= 8192 && pairs <= kGroupPairs * 1024 && experts >= 32 && experts <= kGroupExperts; }

__global__ void __launch_bounds__(1024)
moe_group_warps_kernel(const int* __restrict__ ids, int pairs, int experts, int* __restrict__ offsets, int* __restrict__ order, int* __restrict__ place) {
  pdl_wait();
  pdl_trigger();
  __shared__ int count[32][kGroupExperts];      // of a warp's pairs, then where the warp's begin
  __shared__ int total[kGroupExperts];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int id[kGroupPairs], at[kGroupPairs];
#pragma unroll
  for (int j = 0; j < kGroupPairs; ++j) {
    const int p = tid + j * 1024;
    id[j] = p < pairs ? ids[p] : -1;
  }
  for (int e = lane; e < experts; e += 32) count[warp][e] = 0;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < kGroupPairs; ++j)
    if (id[j] >= 0 && id[j] < experts) at[j] = atomicAdd(&count[warp][id[j]], 1);
  __syncthreads();
  if (tid < experts) {
    int sum = 0;
#pragma unroll
    for (int w = 0; w < 32; ++w) {
      const int own = count[w][tid];
      count[w][tid] = sum;
      sum += own;
    }
    total[tid] = sum;
  }
  __syncthreads();
  if (tid < 32) {      // a warp's running sums, 32 experts at a time
    int run = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {
      const int e = e0 + tid, own = e < experts ? total[e] : 0;
      int upto = own;
#pragma unroll
      for (int step = 1; step < 32; step *= 2) {
        const int below = __shfl_up_sync(0xffffffffu, upto, step);
        if (tid >= step) upto += below;
      }
      if (e < experts) { offsets[e] = run + upto - own; total[e] = run + upto - own; }
      run += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (tid == 0) offsets[experts] = run;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kGroupPairs; ++j) {
    const int p = tid + j * 1024;
    if (p >= pairs) break;
    int s = -1;
    if (id[j] >= 0 && id[j] < experts) {
      s = total[id[j]] + count[warp][id[j]] + at[j];
      order[s] = p;
    }
    place[p] = s;
  }
}

__global__ void __launch_bounds__(1024)
moe_group_kernel(const int* __restrict__ ids, int pairs, int experts, int* __restrict__ offsets, int* __restrict__ order,
                 int* __restrict__ place) {
  pdl_wait();
  pdl_trigger();
  moe_group_pairs(ids, pairs, experts, offsets, order, place);
}

// Both for a step of few tokens, in one launch: a warp per token makes its choices, then the block sorts the pairs.  (Eight tokens x 4
// of 32: 7.4 us cold, where the two kernels took 5.0 and 3.5 and the second's launch; beyond 64 tokens, two rounds of the block's
// warps, one block's arithmetic is slower than the grid's.)
constexpr int kRouteGroupTokens = 64;
template <int S>
__global__ void __launch_bounds__(1024)
moe_route_group_kernel(MoeRouteArgs r, int kept_experts, int* __restrict__ offsets, int* __restrict__ order, int* __restrict__ place) {
  pdl_wait();
  pdl_trigger();
  __shared__ unsigned char kept_s[32][kRouteMaxGroups];
  const int warp = threadIdx.x >> 5;
  for (int t = warp; t < r.tokens; t += 32) moe_route_one<S>(r, t, kept_s[warp]);
  __syncthreads();
  moe_group_pairs(r.ids, r.tokens * r.top, kept_experts, offsets, order, place);
}

// ---------------------------------------------------------------- products
constexpr int GM = 64, GN = 64, GK = 16;

// Row tile `blockIdx.y` counts tiles of GM sorted rows expert by expert; it finds its expert by walking offsets.
// x_by_pair: source row of sorted row s is order[s] / top (the token), else s itself (rows already sorted).
template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(256)
moe_expert_product_kernel(const TX* __restrict__ x, int64_t ldx, const TW* __restrict__ w, TO* __restrict__ y, int64_t ldy,
                          const int* __restrict__ offsets, const int* __restrict__ order, int experts, int top,
                          int x_by_pair, int N, int K, MoeEpilogue ep) {
  pdl_wait();
  pdl_trigger();
  __shared__ float xs[GK][GM + 4];
  __shared__ float ws[GK][GN + 4];
  __shared__ int src_row[GM];
  __shared__ int tile_info[3];     // expert, first sorted row, rows
  if (threadIdx.x == 0) {
    int tile = blockIdx.y, e = 0, found = -1, first = 0, rows = 0;
    for (; e < experts; ++e) {
      const int lo = offsets[e], n = offsets[e + 1] - lo;
      const int tiles = (n + GM - 1) / GM;
      if (tile < tiles) { found = e; first = lo + tile * GM; rows = min(GM, n - tile * GM); break; }
      tile -= tiles;
    }
    tile_info[0] = found; tile_info[1] = first; tile_info[2] = rows;
  }
  __syncthreads();
  const int expert = tile_info[0], first = tile_info[1], rows = tile_info[2];
  if (expert < 0) return;
  const int tid = threadIdx.x;
  if (tid < GM) src_row[tid] = tid < rows ? (x_by_pair ? order[first + tid] / top : first + tid) : -1;
  __syncthreads();
  const TW* we = w + (size_t)expert * N * K;
  const int tx = tid & 15, ty = tid >> 4;
  const int n0 = blockIdx.x * GN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += GK) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int e = tid + it * 256;
      const int r = e >> 4, c = e & 15;
      const int gk = k0 + c, gn = n0 + r;
      const int sr = src_row[r];
      xs[c][r] = (sr >= 0 && gk < K) ? to_f32(x[(size_t)sr * ldx + gk]) : 0.f;
      ws[c][r] = (gn < N && gk < K) ? to_f32(we[(size_t)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (r >= rows) continue;
    const float rs = ep.row_scale ? ep.row_scale[order[first + r]] : 1.f;
    if (moe_act_gated(ep.act)) {
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const int gn = n0 + tx * 4 + j;
        if (gn + 1 >= N) continue;
        y[(size_t)(first + r) * ldy + (gn >> 1)] = from_f32<TO>(moe_gated(acc[i][j] * rs, acc[i][j + 1] * rs, ep.act, ep.limit, ep.alpha));
      }
      continue;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      y[(size_t)(first + r) * ldy + gn] = from_f32<TO>(moe_act(acc[i][j] * rs, ep.act));
    }
  }
}

// ----------------------------------------------------------------- combine
template <typename TS, typename TO>
__global__ void moe_combine_kernel(const float* __restrict__ y, const int* __restrict__ place, const float* __restrict__ weights,
                                   int top, const TS* __restrict__ shared, const float* __restrict__ gate, int64_t ld_gate,
                                   TO* __restrict__ out, int width, const int* __restrict__ ids, int identity_from,
                                   const TO* __restrict__ x, int64_t ldx) {
  pdl_wait();
  pdl_trigger();
  const size_t t = blockIdx.x;
  const float g = (shared && gate) ? 1.f / (1.f + expf(-gate[t * ld_gate])) : 1.f;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < width; c += gridDim.y * blockDim.x) {
    float v = 0.f;
    for (int k = 0; k < top; ++k) {
      const int s = place[t * top + k];
      if (s >= 0) v = fmaf(weights ? weights[t * top + k] : 1.f, y[(size_t)s * width + c], v);
      else if (ids && ids[t * top + k] >= identity_from) v = fmaf(weights ? weights[t * top + k] : 1.f, to_f32(x[t * ldx + c]), v);
    }
    if (shared) v = fmaf(g, to_f32(shared[t * width + c]), v);
    out[t * width + c] = from_f32<TO>(v);
  }
}

// The same with rows on 16-byte boundaries: a thread takes eight neighbouring columns, and all choices' rows are asked for before the
// first is used (four at a time).  Same sums in the same order.  What bounds it is reading top x 4 bytes a column: 2,048 tokens x
// 2,048 columns with four choices and a shared expert 19 us cold, 46 element by element.
template <typename TS, typename TO>
__global__ void __launch_bounds__(256)
moe_combine_vec_kernel(const float* __restrict__ y, const int* __restrict__ place, const float* __restrict__ weights,
                       int top, const TS* __restrict__ shared, const float* __restrict__ gate, int64_t ld_gate,
                       TO* __restrict__ out, int width, const int* __restrict__ ids, int identity_from,
                       const TO* __restrict__ x, int64_t ldx) {
  pdl_wait();
  pdl_trigger();
  const size_t t = blockIdx.x;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= width) return;
  float own[8], v[8];
  if (shared) load8(shared + t * width + c, own);
  const float g = (shared && gate) ? 1.f / (1.f + expf(-gate[t * ld_gate])) : 1.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0.f;
  for (int k0 = 0; k0 < top; k0 += 4) {
    float row[4][8], f[4];
    bool add[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      add[u] = false;
      if (k0 + u >= top) continue;
      const int s = place[t * top + k0 + u];
      f[u] = weights ? weights[t * top + k0 + u] : 1.f;
      if (s >= 0) { load8(y + (size_t)s * width + c, row[u]); add[u] = true; }
      else if (ids && ids[t * top + k0 + u] >= identity_from) { load8(x + t * ldx + c, row[u]); add[u] = true; }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (add[u]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = fmaf(f[u], row[u][j], v[j]);
      }
  }
  if (shared) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = fmaf(g, own[j], v[j]);
  }
  if constexpr (sizeof(TO) == 2) {
    uint4 packed;
    uint32_t* p = reinterpret_cast<uint32_t*>(&packed);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      p[j] = *reinterpret_cast<const uint32_t*>(&pair);
    }
    *reinterpret_cast<uint4*>(out + t * width + c) = packed;
  } else {
    reinterpret_cast<float4*>(out + t * width + c)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(out + t * width + c)[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

}  // namespace tib

using namespace tib;

// x: [tokens, K] (row stride ldx) float or bf16; w: [rows, K] fp32; bias: [rows] fp32 or null; out: [tokens, rows] fp32 (row
// stride ldo)
TIB_API int tib_router_logits(const void* x, int x_dtype, int64_t ldx, const float* w, const float* bias, float* out, int64_t ldo, int tokens,
                              int rows, int K, cudaStream_t stream) {
  if (tokens == 0 || rows == 0) return TIB_OK;
  if (!x || !w || !out || tokens < 0 || rows < 0 || K < 1) return TIB_E_ARG;
  if (tokens > 0x7fffffff / 2) return TIB_E_SIZE;
  const int64_t xbytes = x_dtype == TIB_F32 ? 4 : 2;
  const bool vec = K % 4 == 0 && (ldx * xbytes) % 16 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  // The kernel of large steps from 20,000 logits on: below, a warp a row and four tokens fill the GPU better (33 rows: 400 tokens 8.7 us against 11.5,
  // 800 13.9 against 12.3; 61: 400 tokens 9.9 and 10.3; 129: 100 8.8 and 11.6, 200 13.8 and 12.3).
  // fp32 tokens in their thousands from 10,400 on (2,048 wide, 12 rows, 1,300 tokens 11.1 against 18.5; 4 rows, 3,000 10.6 and 12.4; 6 rows, 1,300 10.6 and 9.8).
  const int passes = ceil_div(rows, kRouterWarps * kRouterRows);      // (of a grid's second dimension)
  if (vec && (int64_t)tokens * rows >= (x_dtype == TIB_F32 && tokens >= 1184 ? 10400 : 20000) && passes <= 65535) {
    const int warps = ceil_div(rows, kRouterRows * passes);
    const dim3 grid(ceil_div(tokens, kRouterMany), passes);
    if (x_dtype == TIB_F32)
      TIB_LAUNCH_DEPENDENT(router_logits_many_kernel<float>, grid, warps * 32, 0, stream, (const float*)x, ldx, w, bias, out, ldo, tokens, rows, K);
    else if (x_dtype == TIB_BF16)
      TIB_LAUNCH_DEPENDENT(router_logits_many_kernel<__nv_bfloat16>, grid, warps * 32, 0, stream, (const __nv_bfloat16*)x, ldx, w, bias, out, ldo, tokens,
                           rows, K);
    else
      return TIB_E_DTYPE;
    return TIB_OK;
  }
  int slices = 1;      // few tokens: the rows of w are spread over several blocks a token
  const int groups = ceil_div(tokens, kRouterTokens);
  while (groups * slices < 2 * 148 && slices * 8 < rows) slices *= 2;
  const dim3 grid(groups, slices);
  // Blocks an SM, of which a slice's last one may be half empty: which form is ahead depends on how they fall into rounds (see DENSE).
  const int first_rows = rows < 8 * slices ? rows : 8 * slices;
  const int most = ceil_div64((int64_t)groups * ceil_div(first_rows, 8), 148), least = ceil_div64((int64_t)groups * ceil_div(first_rows, 4), 2 * 148);
  const bool dense = vec && (x_dtype == TIB_F32 ? most > 1 : most % 2 == 0 || least % 2 == 0);
#define TIB_ROUTER_D(TX, VEC, DENSE) \
  TIB_LAUNCH_DEPENDENT((router_logits_kernel<TX, VEC, DENSE>), grid, 256, 0, stream, (const TX*)x, ldx, w, bias, out, ldo, tokens, rows, K)
#define TIB_ROUTER_GO(TX, VEC) do { if (VEC && dense) TIB_ROUTER_D(TX, VEC, VEC); else TIB_ROUTER_D(TX, VEC, false); } while (0)
  if (x_dtype == TIB_F32) { if (vec) TIB_ROUTER_GO(float, true); else TIB_ROUTER_GO(float, false); }
  else if (x_dtype == TIB_BF16) { if (vec) TIB_ROUTER_GO(__nv_bfloat16, true); else TIB_ROUTER_GO(__nv_bfloat16, false); }
#undef TIB_ROUTER_GO
#undef TIB_ROUTER_D
  else
    return TIB_E_DTYPE;
  return TIB_OK;
}

// correction: [experts] fp32 added to the scores for the choice only, or null; groups > 1 with keep < groups: the experts
// are cut into `groups` equal runs of adjacent ones and only members of the best `keep` runs are eligible.
// offsets, order, place (or null): with at most 64 tokens the pairs are sorted by expert in the same launch, as
// tib_moe_group does for `sorted_experts` experts.
TIB_API int tib_moe_route(const float* logits, int64_t ld, int tokens, int experts, int top, int sigmoid_scores, int normalize,
                          float norm_eps, const float* correction, int groups, int keep, int* ids, float* weights,
                          int sorted_experts, int* offsets, int* order, int* place, cudaStream_t stream) {
  if (tokens == 0) return TIB_OK;
  if (!logits || !ids || !weights) return TIB_E_ARG;
  if (experts < 1 || experts > 2048 || top < 1 || top > experts) return TIB_E_SIZE;
  if (groups < 1 || keep < 1 || keep > groups || groups > kRouteMaxGroups || experts % groups) return TIB_E_SIZE;
  if (groups > 1 && keep < groups && top > keep * (experts / groups)) return TIB_E_SIZE;
  MoeRouteArgs r;
  r.logits = logits; r.ld = ld; r.experts = experts; r.top = top; r.sigmoid_scores = sigmoid_scores; r.normalize = normalize; r.norm_eps = norm_eps;
  r.correction = correction; r.groups = groups; r.keep = keep; r.ids = ids; r.weights = weights; r.tokens = tokens;
  if (offsets) {      // choices and sorting in one launch
    if (!order || !place) return TIB_E_ARG;
    if (tokens > kRouteGroupTokens || sorted_experts < 1 || sorted_experts > 1024) return TIB_E_SIZE;
    TIB_ROUTE_PICK(route_scores_a_lane(r), moe_route_group_kernel, 1, 1024, 0, stream, r, sorted_experts, offsets, order, place);
    return TIB_OK;
  }
  TIB_ROUTE_PICK(route_scores_a_lane(r), moe_route_kernel, ceil_div(tokens, 4), 128, 0, stream, r);
  return TIB_OK;
}

TIB_API int tib_moe_group(const int* ids, int pairs, int experts, int* offsets, int* order, int* place, cudaStream_t stream) {
  if (!ids || !offsets || !order || !place) return TIB_E_ARG;
  if (experts < 1 || experts > 1024 || pairs < 0) return TIB_E_SIZE;
  if (group_by_warps(pairs, experts)) TIB_LAUNCH_DEPENDENT(moe_group_warps_kernel, 1, 1024, 0, stream, ids, pairs, experts, offsets, order, place);
  else TIB_LAUNCH_DEPENDENT(moe_group_kernel, 1, 1024, 0, stream, ids, pairs, experts, offsets, order, place);
  return TIB_OK;
}

// x: rows of K (row stride ldx) in x_dtype; w: [experts, N, K] in w_dtype; y: [pairs, N] (row stride ldy) in y_dtype
// ([pairs, N / 2] for the clamped gated unit, whose N is even); row_scale: [pairs] fp32 or null; error_word: where a bounded
// wait that ran out is reported, or null.
TIB_API int tib_moe_expert_product(const void* x, int x_dtype, int64_t ldx, const void* w, int w_dtype, void* y, int y_dtype,
                                   int64_t ldy, const int* offsets, const int* order, int pairs, int experts, int top,
                                   int x_by_pair, int N, int K, int act, float limit, float alpha, const float* row_scale,
                                   int* error_word, cudaStream_t stream) {
  if (pairs == 0 || N == 0) return TIB_OK;
  if (!x || !w || !y || !offsets || !order || pairs < 0 || N < 0 || K < 1 || top < 1) return TIB_E_ARG;
  if (act < MOE_ACT_NONE || act > MOE_ACT_GELU || (moe_act_gated(act) && N % 2)) return TIB_E_SIZE;
  MoeEpilogue ep;
  ep.act = act; ep.limit = limit; ep.alpha = alpha; ep.row_scale = row_scale;
  const int row_tiles = ceil_div(pairs, GM) + experts;      // at most this many tiles hold a row
  if (row_tiles > 65535) return TIB_E_SIZE;
  dim3 grid(ceil_div(N, GN), row_tiles);
  if (x_dtype == TIB_BF16 && w_dtype == TIB_BF16 && moe_product_tcgen05_takes(x, ldx, w, experts, N, K)) {
    if (y_dtype != TIB_BF16 && y_dtype != TIB_F32) return TIB_E_DTYPE;
    return moe_product_tcgen05(x, ldx, w, y, y_dtype, ldy, offsets, order, pairs, experts, top, x_by_pair, N, K, ep, error_word, stream);
  }
#define TIB_MOE_GO(TX, TW, TO)                                                                                             \
  TIB_LAUNCH_DEPENDENT((moe_expert_product_kernel<TX, TW, TO>), grid, 256, 0, stream, (const TX*)x, ldx, (const TW*)w, (TO*)y, \
                       ldy, offsets, order, experts, top, x_by_pair, N, K, ep)
  if (x_dtype == TIB_F32 && w_dtype == TIB_F32 && y_dtype == TIB_F32) TIB_MOE_GO(float, float, float);
  else if (x_dtype == TIB_BF16 && w_dtype == TIB_BF16 && y_dtype == TIB_BF16) TIB_MOE_GO(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
  else if (x_dtype == TIB_BF16 && w_dtype == TIB_BF16 && y_dtype == TIB_F32) TIB_MOE_GO(__nv_bfloat16, __nv_bfloat16, float);
  else return TIB_E_DTYPE;
#undef TIB_MOE_GO
  return TIB_OK;
}

// y: [pairs, width] fp32; shared: [tokens, width] in shared_dtype or null; gate: fp32 logit per token (stride ld_gate) or
// null (the shared rows are added as they are); out: [tokens, width] in out_dtype.  ids [tokens * top] with identity_from
// and x (the experts' input rows, in out_dtype, ldx elements apart): choices of id >= identity_from add weight * x[t].
TIB_API int tib_moe_combine(const float* y, const int* place, const float* weights, int top, const void* shared,
                            int shared_dtype, const float* gate, int64_t ld_gate, void* out, int out_dtype, int tokens,
                            int width, const int* ids, int identity_from, const void* x, int64_t ldx, cudaStream_t stream) {
  if (tokens == 0 || width == 0) return TIB_OK;
  if (!y || !place || !out || top < 1 || (ids && !x)) return TIB_E_ARG;
  const int threads = width >= 1024 ? 256 : 128;
  // (few tokens: a row's columns are spread over several blocks)
  const dim3 grid(tokens, tokens < 2 * 148 ? ceil_div(width, threads) : 1);
  const int64_t xsize = out_dtype == TIB_F32 ? 4 : 2;
  const bool vec = width % 8 == 0 && (((uintptr_t)y | (uintptr_t)shared | (uintptr_t)out) & 15) == 0 &&
                   (!ids || (((uintptr_t)x & 15) == 0 && (ldx * xsize) % 16 == 0));
  const int vec_threads = tokens < 2 * 148 ? 64 : 256;
  const dim3 vec_grid(tokens, ceil_div(width / 8, vec_threads));
#define TIB_COMBINE_GO(TS, TO)                                                                                       \
  do {                                                                                                               \
    if (vec)                                                                                                         \
      TIB_LAUNCH_DEPENDENT((moe_combine_vec_kernel<TS, TO>), vec_grid, vec_threads, 0, stream, y, place, weights, top, (const TS*)shared, \
                           gate, ld_gate, (TO*)out, width, ids, identity_from, (const TO*)x, ldx);                    \
    else                                                                                                             \
      TIB_LAUNCH_DEPENDENT((moe_combine_kernel<TS, TO>), grid, threads, 0, stream, y, place, weights, top, (const TS*)shared, gate, \
                           ld_gate, (TO*)out, width, ids, identity_from, (const TO*)x, ldx);                         \
  } while (0)
  const int sd = shared ? shared_dtype : out_dtype;
  if (sd == TIB_F32 && out_dtype == TIB_F32) TIB_COMBINE_GO(float, float);
  else if (sd == TIB_BF16 && out_dtype == TIB_BF16) TIB_COMBINE_GO(__nv_bfloat16, __nv_bfloat16);
  else if (sd == TIB_BF16 && out_dtype == TIB_F32) TIB_COMBINE_GO(__nv_bfloat16, float);
  else if (sd == TIB_F32 && out_dtype == TIB_BF16) TIB_COMBINE_GO(float, __nv_bfloat16);
  else return TIB_E_DTYPE;
#undef TIB_COMBINE_GO
  return TIB_OK;
}

// The calls the Python parts make (common.cuh).
TIB_PACKED(tib_moe_combine)
TIB_PACKED(tib_moe_expert_product)
TIB_PACKED(tib_moe_group)
TIB_PACKED(tib_moe_route)
TIB_PACKED(tib_router_logits)
