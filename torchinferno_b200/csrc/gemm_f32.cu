// True 32-bit matrix product on CUDA cores: out[M, N] = x[M, K] . w[N, K]^T.
//
// No tensor cores and no reduced-precision mode: every product and sum is an
// fp32 fused multiply-add.  Each output element is accumulated by one thread
// over k = 0 .. K-1 in rising order, so a row's result does not depend on how
// many other rows are in the call (the projections of the reference are plain
// `F.linear` calls: src/torchinferno/models/llama3/pipeline.py:206-208,245,248-250,400).
// Optionally w and/or x may be bf16 in memory; they are widened on load.
//
// Weights that gemm_f32_tcgen05.cu takes (by their sizes) run there; this file has the products of small, odd or bf16 weights.
//
// Two kernels with the same sums, bit for bit.  32-bit operands whose rows are 16-byte aligned run through a ring of four
// shared-memory stages (cp.async, 16 k each) with up to 8 x 8 outputs a thread; everything else (bf16 in memory, odd
// strides) runs the plain kernel.
#include "mma.cuh"

namespace tib {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TX, typename TW>
__global__ void __launch_bounds__(256)
gemm_f32_kernel(const TX* __restrict__ x, const TW* __restrict__ w, float* __restrict__ out, int M,
                int N, int K, int64_t ldx, int64_t ldw, int64_t ldo) {
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, each 4 x 4 outputs
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 x 16 elements per tile, 256 threads: 4 elements each.
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int e = tid + it * 256;
      const int r = e >> 4, c = e & 15;
      const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
      xs[c][r] = (gm < M && gk < K) ? to_f32(x[(size_t)gm * ldx + gk]) : 0.f;
      ws[c][r] = (gn < N && gk < K) ? to_f32(w[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
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
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn < N) out[(size_t)gm * ldo + gn] = acc[i][j];
    }
  }
}

// ------------------------------------------------------------------------------------------ aligned 32-bit operands
// A thread owns rows ty + 8 i and columns tx + 16 j of a tile of TM * 8 x TN * 16.  Both operands stay as they lie in memory, rows
// of 16 k on a stride of 20 floats: a thread reads four k of a row in one 16-byte load, and the eight rows of a quarter of a warp
// start in eight different groups of four banks.  Per four k that is TM + TN loads for 4 TM TN multiply-adds, so the fp32
// pipe, not shared memory, bounds it, and the copies of the next three stages run under the arithmetic.
// (The plain kernel fetches element by element, with nothing in flight under its arithmetic: 301 x 16,384 x 2,048
// took 1,006 us there and takes 541 here, 2,048 cubed 783 and 432: 40 TFLOP/s, 58 % of the fp32 pipe; what is left is the
// dispatch of three-operand instructions.)
constexpr int kFgK = 16, kFgStride = kFgK + 4, kFgStages = 4;

template <int TM, int TN>
__global__ void __launch_bounds__(128)
gemm_f32_ring_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int M, int N, int K,
                     int64_t ldx, int64_t ldw, int64_t ldo) {
  constexpr int TBM = TM * 8, TBN = TN * 16, ROWS = TBM + TBN;
  extern __shared__ __align__(16) float ring[];      // [stages][ROWS][kFgStride]: rows of x, then rows of w
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
  // (rows beyond the matrix and k beyond K are filled with zeros, which add nothing)
  auto fetch = [&](int stage, int k0) {
    float* dst = ring + stage * ROWS * kFgStride;
#pragma unroll
    for (int it = 0; it < (ROWS * 4 + 127) / 128; ++it) {
      const int p = tid + it * 128, r = p >> 2, c = (p & 3) * 4;
      if (ROWS * 4 % 128 != 0 && r >= ROWS) break;
      const bool first = r < TBM;
      const int row = first ? m0 + r : n0 + r - TBM;
      const bool in = (first ? row < M : row < N) && k0 + c < K;
      const float* src = first ? x + (size_t)(in ? row : 0) * ldx : w + (size_t)(in ? row : 0) * ldw;
      cp_async16(dst + r * kFgStride + c, src + (in ? k0 + c : 0), in);
    }
    cp_async_commit();
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  const int steps = (K + kFgK - 1) / kFgK;
#pragma unroll
  for (int s = 0; s < kFgStages - 1; ++s) {
    if (s < steps) fetch(s, s * kFgK);
    else cp_async_commit();
  }
  for (int ks = 0; ks < steps; ++ks) {
    cp_async_wait<kFgStages - 2>();
    __syncthreads();                 // the stage has landed for everyone, and the one before it is free
    if (ks + kFgStages - 1 < steps) fetch((ks + kFgStages - 1) % kFgStages, (ks + kFgStages - 1) * kFgK);
    else cp_async_commit();
    const float* xs = ring + (ks % kFgStages) * ROWS * kFgStride + ty * kFgStride;
    const float* ws = ring + (ks % kFgStages) * ROWS * kFgStride + (TBM + tx) * kFgStride;
#pragma unroll
    for (int kk = 0; kk < kFgK; kk += 4) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * 8 * kFgStride + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 b = *reinterpret_cast<const float4*>(ws + j * 16 * kFgStride + kk);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty + 8 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx + 16 * j;
      if (gn < N) out[(size_t)gm * ldo + gn] = acc[i][j];
    }
  }
}

template <int TM, int TN>
static int launch_gemm_f32_ring(const float* x, const float* w, float* out, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo,
                                cudaStream_t stream) {
  constexpr int smem = kFgStages * (TM * 8 + TN * 16) * kFgStride * 4;
  cudaError_t e = cudaFuncSetAttribute(gemm_f32_ring_kernel<TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  gemm_f32_ring_kernel<TM, TN><<<dim3(ceil_div(N, TN * 16), ceil_div(M, TM * 8)), 128, smem, stream>>>(x, w, out, M, N, K, ldx, ldw, ldo);
  TIB_LAUNCH_CHECK();
  return TIB_OK;
}

}  // namespace tib

using namespace tib;

// x: [M, K] (row stride ldx), w: [N, K] (row stride ldw), out: [M, N] fp32 (row stride ldo).
TIB_API int tib_gemm_f32(const void* x, const void* w, float* out, int M, int N, int K, int64_t ldx,
                         int64_t ldw, int64_t ldo, int x_dtype, int w_dtype, cudaStream_t stream) {
  if (M == 0 || N == 0) return TIB_OK;
  if (!x || !w || !out || M < 0 || N < 0 || K < 1) return TIB_E_ARG;
  dim3 grid(ceil_div(N, BN), ceil_div(M, BM));
  if (grid.y > 65535) return TIB_E_SIZE;
  if (x_dtype == TIB_F32 && w_dtype == TIB_F32 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0) {
    // The tile with the least work for the busiest SM: whole rounds of tiles over the SMs times a tile's area, the area of the
    // smaller tiles counted up for what they lose to shared-memory reads (us: 301 x 2,048 x 2,048 plain kernel
    // 238, 32 x 64 tiles 117; 8 x 2,048 x 8,192 plain 821, 16 x 32 tiles 154).
    const auto cost = [&](int bm, int bn, double weight) {
      const int64_t tiles = (int64_t)ceil_div(M, bm) * ceil_div(N, bn);
      return (double)ceil_div64(tiles, 148) * bm * bn * weight;
    };
    const double big = cost(64, 128, 1.0), middle = cost(64, 64, 1.1), small = cost(32, 64, 1.25), least = cost(16, 32, 2.0);
    const float* xf = (const float*)x;
    const float* wf = (const float*)w;
    if (ceil_div(M, 16) <= 65535) {
      if (least < small && least < middle && least < big) return launch_gemm_f32_ring<2, 2>(xf, wf, out, M, N, K, ldx, ldw, ldo, stream);
      if (small < middle && small < big) return launch_gemm_f32_ring<4, 4>(xf, wf, out, M, N, K, ldx, ldw, ldo, stream);
      if (middle < big) return launch_gemm_f32_ring<8, 4>(xf, wf, out, M, N, K, ldx, ldw, ldo, stream);
      return launch_gemm_f32_ring<8, 8>(xf, wf, out, M, N, K, ldx, ldw, ldo, stream);
    }
  }
  if (x_dtype == TIB_F32 && w_dtype == TIB_F32)
    gemm_f32_kernel<float, float><<<grid, 256, 0, stream>>>((const float*)x, (const float*)w, out, M, N, K, ldx, ldw, ldo);
  else if (x_dtype == TIB_F32 && w_dtype == TIB_BF16)
    gemm_f32_kernel<float, __nv_bfloat16><<<grid, 256, 0, stream>>>((const float*)x, (const __nv_bfloat16*)w, out, M, N, K, ldx, ldw, ldo);
  else if (x_dtype == TIB_BF16 && w_dtype == TIB_F32)
    gemm_f32_kernel<__nv_bfloat16, float><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, (const float*)w, out, M, N, K, ldx, ldw, ldo);
  else if (x_dtype == TIB_BF16 && w_dtype == TIB_BF16)
    gemm_f32_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w, out, M, N, K, ldx, ldw, ldo);
  else
    return TIB_E_DTYPE;
  TIB_LAUNCH_CHECK();
  return TIB_OK;
}

// The calls the Python parts make (common.cuh).
TIB_PACKED(tib_gemm_f32)
