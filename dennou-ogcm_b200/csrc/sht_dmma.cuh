// sht_dmma.cuh -- the FP64 mma.sync fragment products of the Legendre kernels.
#pragma once

namespace sht {
namespace dmma {

// d (8x8 FP64 tile, two values per lane) += a (8x4, one per lane) * b (4x8, one per lane)
__device__ __forceinline__ void mma884(double (&d)[2], double a, double b)
{
  // no side effects beyond d: left non-volatile so that the compiler may
  // schedule fragment loads across the products
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// two row tiles and two steps at once: the m8n8k4 products d0 += a0 b0, then
// a2 b1, and d1 += a1 b0, then a3 b1 (rows 0-7 and 8-15 of a 16x8 tile) as one
// instruction.  The kernels count on its rounding like the two m8n8k4 steps: a
// field-level has the same bits whichever of the two its batch's kernel issues
// (measured on B200, tested on every form the kernels have).
__device__ __forceinline__ void mma1688(double (&d0)[2], double (&d1)[2], double a0, double a1, double a2, double a3,
                                        double b0, double b1)
{
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d0[0]), "+d"(d0[1]), "+d"(d1[0]), "+d"(d1[1])
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

}  // namespace dmma
}  // namespace sht
