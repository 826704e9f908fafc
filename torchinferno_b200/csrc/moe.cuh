// What the kernels of a routed feed-forward share: the experts' activations and what is done to a product's sums.
#pragma once

#include "common.cuh"

namespace tib {

enum MoeAct : int { MOE_ACT_NONE = 0, MOE_ACT_RELU2 = 1, MOE_ACT_SILU = 2, MOE_ACT_GLU_CLAMP = 3, MOE_ACT_SWIGLU = 4, MOE_ACT_GELU = 5 };
__host__ __device__ constexpr bool moe_act_gated(int act) { return act == MOE_ACT_GLU_CLAMP || act == MOE_ACT_SWIGLU; }

struct MoeEpilogue {
  int act;
  float limit, alpha;          // of the clamped gated unit
  const float* row_scale;      // [pairs] or null: sorted row s is multiplied by row_scale[order[s]] before the activation
};

__device__ __forceinline__ float moe_act(float v, int act) {
  if (act == MOE_ACT_RELU2) { v = fmaxf(v, 0.f); return v * v; }
  if (act == MOE_ACT_SILU) return v / (1.f + expf(-v));
  if (act == MOE_ACT_GELU) return gelu_erf(v);
  return v;
}
// the gated units over (gate, up) row pairs: clamped, g = min(g, limit), u = clamp(u, -limit, limit), g * sigmoid(alpha * g) * (u + 1);
// or silu(g) * u
__device__ __forceinline__ float moe_gated(float g, float u, int act, float limit, float alpha) {
  if (act == MOE_ACT_SWIGLU) return g / (1.f + expf(-g)) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.f + expf(-alpha * g)) * (u + 1.f);
}

// The products of bf16 operands on the 5th-generation tensor cores (moe_tcgen05.cu), where moe_product_tcgen05_takes them;
// y_dtype TIB_F32 or TIB_BF16; the other arguments as tib_moe_expert_product.
bool moe_product_tcgen05_takes(const void* x, int64_t ldx, const void* w, int experts, int N, int K);
int moe_product_tcgen05(const void* x, int64_t ldx, const void* w, void* y, int y_dtype, int64_t ldy, const int* offsets,
                        const int* order, int pairs, int experts, int top, int x_by_pair, int N, int K, const MoeEpilogue& ep,
                        int* error_word, cudaStream_t stream);

}  // namespace tib
