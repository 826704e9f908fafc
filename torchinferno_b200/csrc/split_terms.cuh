// Pieces shared by the kernels that make 32-bit products on the tensor cores: a float as the sum of three bf16 numbers, operands' places, and what a
// block begins and ends with.
#pragma once

#include "tcgen05.cuh"
#include "mma.cuh"

namespace tib {

__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The three terms of two floats, packed.
__device__ __forceinline__ void ft_split2(float a, float b, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
  t0 = pack_bf16(a, b);
  f2_unpack(f2_sub(f2_pack(a, b), f2_pack(__uint_as_float(t0 << 16), __uint_as_float(t0 & 0xffff0000u))), a, b);
  t1 = pack_bf16(a, b);
  f2_unpack(f2_sub(f2_pack(a, b), f2_pack(__uint_as_float(t1 << 16), __uint_as_float(t1 & 0xffff0000u))), a, b);
  t2 = pack_bf16(a, b);
}

// The same, but what the first term cannot hold (an infinity; anything above
// 3.39e38) is an infinity there, with nothing left for the others.
__device__ __forceinline__ void ft_split2_finite(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const float2 hf = bf16x2_floats(h);
  float ra = a - hf.x, rb = b - hf.y;
  ra = isfinite(hf.x) ? ra : 0.f;
  rb = isfinite(hf.y) ? rb : 0.f;
  const __nv_bfloat162 m = __floats2bfloat162_rn(ra, rb);
  const float2 mf = bf16x2_floats(m);
  const __nv_bfloat162 l = __floats2bfloat162_rn(ra - mf.x, rb - mf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  mid = *reinterpret_cast<const uint32_t*>(&m);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// The bits of a packed pair that belong to finite numbers.
__device__ __forceinline__ uint32_t ft_finite2(uint32_t v) {
  return ((v & 0x7f80u) == 0x7f80u ? 0u : 0xffffu) | ((v & 0x7f800000u) == 0x7f800000u ? 0u : 0xffff0000u);
}

__device__ __forceinline__ void ft_tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// The place, in a tile of [width / 64][rows][64] bf16 with 128-byte swizzle, of eight elements of row r from column 8 c8.
__device__ __forceinline__ uint32_t ft_place(int r, int c8, int rows) { return (uint32_t)((c8 >> 3) * rows * 128 + r * 128 + (((c8 & 7) ^ (r & 7)) << 4)); }

__device__ __forceinline__ void ft_store8(float* dst, const float (&v)[8]) {      // (on a 16-byte boundary)
  if ((uintptr_t)dst & 16) {
    reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
    return;
  }
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
               ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// Barriers that one commit completes, and `columns` columns of tensor memory; called by the whole block, with a barrier of the block behind it.
// pdl_trigger() comes after it: a block of the next kernel that is placed before this one has its columns could take them, and wait for this
// kernel's end with them.
__device__ __forceinline__ uint32_t ft_setup(uint32_t bar0, int bars, uint32_t slot, volatile uint32_t* slot_ptr, int warp, uint32_t columns) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < bars; ++i) mbar_init(bar0 + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return *slot_ptr;
}
// What the threads left in shared and tensor memory becomes the tensor cores' (called by the whole block).
__device__ __forceinline__ void ft_hand_over() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void ft_wait(uint32_t bar, uint32_t parity, int* error_word, int code) {
  if (!mbar_wait(bar, parity) && error_word && (threadIdx.x & 31) == 0) atomicExch(error_word, code);
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void ft_release(int warp, uint32_t tmem, uint32_t columns) {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(columns) : "memory");
  }
}

}  // namespace tib
