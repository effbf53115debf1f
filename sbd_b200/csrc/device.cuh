// Device functions shared by the kernels on the FP64 tensor pipe.
#pragma once

#include <cuda_runtime.h>

namespace sbdgpu {

// D (16 x 8) += A (16 x 4) B (4 x 8), FP64
__device__ __forceinline__ void mma16(double (&d)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5},{%6},{%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b));
}

// index of the off-diagonal pair of orbitals a != b
__device__ __forceinline__ int od_pair(int a, int b) {
  const int hi = max(a, b), lo = min(a, b);
  return hi * (hi - 1) / 2 + lo;
}

// the larger orbital hi of off-diagonal pair o: hi (hi - 1) / 2 <= o < hi (hi + 1) / 2
__device__ __forceinline__ int od_larger(int o) {
  int hi = (int)((1.0f + sqrtf(8.0f * (float)o + 1.0f)) * 0.5f);
  hi += hi * (hi + 1) / 2 <= o;
  hi -= hi * (hi - 1) / 2 > o;
  return hi;
}

}  // namespace sbdgpu
