// Pieces shared by the kernels that make 32-bit products on the tensor cores: a float as the sum of three bf16 numbers, and MMAs issued by a
// whole warp.
#pragma once

#include "tcgen05.cuh"
#include "mma.cuh"

namespace tib {

__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
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

// One lane of the warp.  A warp that walks its loop together and lets one lane issue keeps the instructions' operands in uniform registers: 8 cycles
// an instruction, where a lane on its own takes 45 (measured with 128 x 16 x 16 products, which take the tensor core 10).
__device__ __forceinline__ uint32_t ft_elect() {
  uint32_t one;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
  return one;
}
// The product with the weights in tensor memory, issued by the leader of a warp that is together.
__device__ __forceinline__ void ft_mma(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %5, 0;\n"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}

// The same with both operands in shared memory.
__device__ __forceinline__ void ft_mma_shared(uint32_t leader, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %5, 0;\n"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
__device__ __forceinline__ void ft_tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void ft_tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}

}  // namespace tib
