// What the tensor-core kernels of float32 sums share (lattice_conv_tc.cu, factored_tc.cu): warp products of 16 x 8 x 16, float32 as
// three bfloat16, and additions of two float32 at a time.
#pragma once
#include <cuda_bf16.h>

namespace gmb {

// d += a b, a 16 x 16 by rows, b 16 x 8 by columns
__device__ __forceinline__ void mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// d = a b.  zero: four zeros that the compiler does not see through (it would clear four registers for every product)
__device__ __forceinline__ void mma_first(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1, const float (&zero)[4]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(zero[0]), "f"(zero[1]), "f"(zero[2]), "f"(zero[3]));
}
// (x, y) as the sum of three pairs of bfloat16, largest first: exact from 2^-110 on, below with an error of up to 2^-134; NaN from
// 3.396e38 on, which rounds to infinity
__device__ __forceinline__ void split3(float x, float y, unsigned (&w)[3]) {
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    w[s] = *reinterpret_cast<const unsigned*>(&h);
    x -= __uint_as_float(w[s] << 16);
    y -= __uint_as_float(w[s] & 0xffff0000u);
  }
}

// Two float32 sums in one 64-bit register pair
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
__device__ __forceinline__ void add2(f32x2& d, f32x2 v) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(v)); }
__device__ __forceinline__ void add2(f32x2& d, float x, float y) { add2(d, pack2(x, y)); }
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

}  // namespace gmb
