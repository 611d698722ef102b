// FP64 tensor-core tiles (mma.sync m8n8k4) for the contractions that stay in
// FP64: the tcgen05 units have no FP64 form, and the FP64 mma path of sm_100a
// runs at 37 TFLOP/s (measured with 8 or more warps per SM, register operands)
// against 33 for scalar FP64 FMAs, with a sixteenth of the instructions and
// no operand broadcast through the register file.
//
// A warp holds a 32 x 32 tile: acc[i][j] is the 8 x 8 block at rows 8 i, columns
// 8 j, thread (g = lane / 4, t = lane % 4) its row g and columns 2 t, 2 t + 1.
// The order of the K index inside a group of 8 is free as long as A and B agree:
// the first mma takes k = 2 t, the second k = 2 t + 1, so that an operand stored
// with K contiguous is read as one 16-byte word per thread.
#pragma once
#include "tc_sm100.cuh"

namespace dm {

constexpr int LDK = 40;   // row stride (doubles) of a [row][32 k] operand: 64 mod 128 bytes, so
                          // the 16-byte reads of a quarter warp (2 rows x 4 t) hit all banks
constexpr int LDN = 130;  // row stride of a [k][128 n] operand: rows 2 t are 4 words of 8 bytes
                          // apart mod 16, so the 8-byte reads of a half warp hit all banks

__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ void zero(double (&acc)[4][4][2]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
}

// acc += A B^T over 32 k: A at the warp's first row of [m][LDK], B at its first
// column of [n][LDK]
__device__ __forceinline__ void chunk_nk(double (&acc)[4][4][2], const double* A, const double* B,
                                         int lane) {
  const int g = lane >> 2, t = lane & 3;
  const double* a0 = A + g * LDK + 2 * t;
  const double* b0 = B + g * LDK + 2 * t;
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    double2 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = *reinterpret_cast<const double2*>(a0 + i * 8 * LDK + kk * 8);
      b[i] = *reinterpret_cast<const double2*>(b0 + i * 8 * LDK + kk * 8);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) mma884(acc[i][j], a[i].x, b[j].x);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) mma884(acc[i][j], a[i].y, b[j].y);
  }
}

// the same with B [k][LDN] (n contiguous), B at the warp's first column
__device__ __forceinline__ void chunk_kn(double (&acc)[4][4][2], const double* A, const double* B,
                                         int lane) {
  const int g = lane >> 2, t = lane & 3;
  const double* a0 = A + g * LDK + 2 * t;
  const double* b0 = B + 2 * t * LDN + g;
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    double2 a[4];
    double b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = *reinterpret_cast<const double2*>(a0 + i * 8 * LDK + kk * 8);
      b[i] = b0[kk * 8 * LDN + i * 8];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) mma884(acc[i][j], a[i].x, b[j]);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = b0[(kk * 8 + 1) * LDN + i * 8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) mma884(acc[i][j], a[i].y, b[j]);
  }
}

}  // namespace dm
