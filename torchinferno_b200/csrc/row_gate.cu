// See row_gate.cuh.  A block owns a run of `part` columns of one row; a thread holds up to four pieces of eight neighbouring columns in
// registers between the sum of squares and the result, so x and z are read once, all of a thread's loads in flight together.
// What bounds it is memory: 2,048 rows of 4,096 (fp32 in, bf16 gate and out) take 18 us cold,
// and took 50 element by element in two passes.
#include "row_gate.cuh"

namespace tib {

__device__ __forceinline__ void rg_load8(const float* p, float (&v)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void rg_load8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = bf16x2_floats(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

template <typename TX, int MODE, int NV>
__global__ void __launch_bounds__(256) row_gate_kernel(RowGateArgs a) {
  pdl_wait();
  pdl_trigger();
  __shared__ float scratch[33];
  const size_t row = blockIdx.x;
  const int first = blockIdx.y * a.part;
  const TX* x = reinterpret_cast<const TX*>(a.x) + row * a.ldx + first;
  const __nv_bfloat16* z = reinterpret_cast<const __nv_bfloat16*>(a.z) + row * a.ldz;
  float v[NV][8], g[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (i * blockDim.x + threadIdx.x) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i][j] = g[i][j] = 0.f;
    if (c < a.part) {
      rg_load8(x + c, v[i]);
      if (MODE != ROW_GATE_ONLY || a.group == 1) rg_load8(z + first + c, g[i]);
      else {
        const float one = __bfloat162float(z[(first + c) / a.group]);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[i][j] = one;
      }
    }
  }
  float inv = 1.f;
  if (MODE != ROW_GATE_ONLY) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (MODE == ROW_GATE_FIRST) v[i][j] *= g[i][j] / (1.f + expf(-g[i][j]));
        ss = fmaf(v[i][j], v[i][j], ss);
      }
    inv = 1.f / sqrtf(block_sum(ss, scratch) / (float)a.part + a.eps);
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (i * blockDim.x + threadIdx.x) * 8;
    if (c >= a.part) continue;
    float w[8];
    if (MODE != ROW_GATE_ONLY) rg_load8(a.weight + first + c, w);
    uint4 packed;
    __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&packed);
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o[j] = v[i][j];
      if (MODE != ROW_GATE_ONLY) o[j] = o[j] * inv * w[j];
      if (MODE != ROW_GATE_FIRST) o[j] *= 1.f / (1.f + expf(-g[i][j]));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) p2[j] = __floats2bfloat162_rn(o[2 * j], o[2 * j + 1]);
    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + row * a.width + first + c) = packed;
  }
}

bool row_gate_takes(const RowGateArgs& a, int mode) {
  const int64_t xsize = a.x_dtype == TIB_F32 ? 4 : 2;
  if (a.z_dtype != TIB_BF16 || a.out_dtype != TIB_BF16 || a.part % 8 || a.part < 8 || a.part > 8192) return false;
  if ((a.ldx * xsize) % 16 || (((uintptr_t)a.x | (uintptr_t)a.out | (uintptr_t)a.weight) & 15)) return false;
  if (mode == ROW_GATE_ONLY && a.group > 1) return a.group % 8 == 0;
  return a.group == 1 && a.ldz % 8 == 0 && ((uintptr_t)a.z & 15) == 0;
}

int row_gate(const RowGateArgs& a, int mode, cudaStream_t stream) {
  const int pieces = a.part / 8, nv = pieces <= 256 ? 1 : pieces <= 512 ? 2 : 4;
  const int threads = (ceil_div(pieces, nv) + 31) / 32 * 32;
  const dim3 grid(a.rows, a.width / a.part);
#define TIB_RG_NV(TX, MODE)                                                                    \
  do {                                                                                         \
    if (nv == 1) TIB_LAUNCH_DEPENDENT((row_gate_kernel<TX, MODE, 1>), grid, threads, 0, stream, a);      \
    else if (nv == 2) TIB_LAUNCH_DEPENDENT((row_gate_kernel<TX, MODE, 2>), grid, threads, 0, stream, a); \
    else TIB_LAUNCH_DEPENDENT((row_gate_kernel<TX, MODE, 4>), grid, threads, 0, stream, a);              \
  } while (0)
#define TIB_RG_GO(TX)                                        \
  do {                                                       \
    if (mode == ROW_GATE_ONLY) TIB_RG_NV(TX, ROW_GATE_ONLY); \
    else if (mode == ROW_GATE_LAST) TIB_RG_NV(TX, ROW_GATE_LAST); \
    else TIB_RG_NV(TX, ROW_GATE_FIRST);                      \
  } while (0)
  if (a.x_dtype == TIB_F32) TIB_RG_GO(float);
  else TIB_RG_GO(__nv_bfloat16);
#undef TIB_RG_GO
#undef TIB_RG_NV
  return TIB_OK;
}

}  // namespace tib
