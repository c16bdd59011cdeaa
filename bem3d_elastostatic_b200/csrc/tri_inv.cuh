// Inverse of a 128 x 128 unit upper triangle in shared memory, FP64, in place.
#pragma once

namespace bem {

constexpr int kTriPitch = 130;    // column pitch: even, so that four rows of a column load as two 16 B words
constexpr int kTriThreads = 512;  // threads of a CTA that inverts
// shared memory of unit_upper_inverse: the triangle and a 96 x 32 product
constexpr int kTriDoubles = 128 * kTriPitch + 96 * 32;

// U (column-major, pitch kTriPitch, 16-byte aligned; its strict upper part given, zero below
// the diagonal, the diagonal itself ignored) := (I + strict upper part)^{-1}; all kTriThreads
// threads take part, with a barrier before and after.
//
// Blocked by 32 as LAPACK's dtrtri: four warps invert the diagonal blocks (a lane per column
// in registers, column by column of U so that a step's updates are independent of each
// other), then block column j follows from the inverse of the leading part,
//   V_{<j,j} = -V_{<j,<j} (U_{<j,j} V_jj),
// two products per block column, four rows and one column per thread and step, everything
// in shared memory.  (Kept in global memory and taken block by block, 18 barriers and an L2
// round trip per product, the same inverse took 97 us; a 128-block now takes 20 us.)
__device__ __forceinline__ void unit_upper_inverse(double* U, double* T) {
  constexpr int B = 32, P = kTriPitch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kTriThreads / 32;
  __syncthreads();
  if (warp < 4) {
    double* D = U + warp * B * (P + 1);
    double x[B];
#pragma unroll
    for (int i = 0; i < B; ++i) x[i] = (i == lane) ? 1.0 : 0.0;
#pragma unroll
    for (int k = B - 1; k > 0; --k)
#pragma unroll
      for (int i = 0; i < k; ++i) x[i] = fma(-D[i + k * P], x[k], x[i]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < B; ++i)
      if (i <= lane) D[i + lane * P] = x[i];
  }
  __syncthreads();
  for (int j = 1; j < 4; ++j) {
    const int R = B * j;
    // T (R x 32, [k][row pairs] as T[row + 96 c]) = U_{<j,j} V_jj
    for (int g = warp; g < R / 4; g += nw) {
      double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll 8
      for (int k = 0; k < B; ++k) {
        const double2* a = reinterpret_cast<const double2*>(U + 4 * g + (R + k) * P);
        const double2 a0 = a[0], a1 = a[1];
        const double b = U[R + k + (R + lane) * P];  // zero below V_jj's diagonal
        s0 = fma(a0.x, b, s0);
        s1 = fma(a0.y, b, s1);
        s2 = fma(a1.x, b, s2);
        s3 = fma(a1.y, b, s3);
      }
      T[(4 * g + 0) * B + lane] = s0;
      T[(4 * g + 1) * B + lane] = s1;
      T[(4 * g + 2) * B + lane] = s2;
      T[(4 * g + 3) * B + lane] = s3;
    }
    __syncthreads();
    for (int g = warp; g < R / 4; g += nw) {
      double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll 4
      for (int k = 4 * g; k < R; ++k) {
        const double2* a = reinterpret_cast<const double2*>(U + 4 * g + k * P);
        const double2 a0 = a[0], a1 = a[1];
        const double b = T[k * B + lane];
        s0 = fma(a0.x, b, s0);
        s1 = fma(a0.y, b, s1);
        s2 = fma(a1.x, b, s2);
        s3 = fma(a1.y, b, s3);
      }
      double* o = U + 4 * g + (R + lane) * P;  // the columns of block j are not read here
      o[0] = -s0;
      o[1] = -s1;
      o[2] = -s2;
      o[3] = -s3;
    }
    __syncthreads();
  }
}

}  // namespace bem
