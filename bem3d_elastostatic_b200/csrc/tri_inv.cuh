// Inverse of a 128 x 128 unit upper triangle in shared memory, in place.
#pragma once

namespace bem {

// column pitch: four rows of a column load as 16-byte words
template <typename T>
constexpr int kTriPitch = sizeof(T) == 8 ? 130 : 132;
constexpr int kTriThreads = 512;  // threads of a CTA that only inverts
// shared memory of unit_upper_inverse: the triangle and a 96 x 32 product
template <typename T>
constexpr int kTriElems = 128 * kTriPitch<T> + 96 * 32;

__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = a.z;
  v[3] = a.w;
}

// U (column-major, pitch kTriPitch, 16-byte aligned; its strict upper part given, zero below
// the diagonal, the diagonal itself ignored) := (I + strict upper part)^{-1}; all NT threads
// of the CTA take part, with a barrier before and after.
//
// Blocked by 32 as LAPACK's dtrtri: four warps invert the diagonal blocks (a lane per column
// in registers, column by column of U so that a step's updates are independent of each
// other), then block column j follows from the inverse of the leading part,
//   V_{<j,j} = -V_{<j,<j} (U_{<j,j} V_jj),
// two products per block column, four rows and one column per thread and step, everything
// in shared memory.  (Kept in global memory and taken block by block, 18 barriers and an L2
// round trip per product, the FP64 inverse took 97 us; a 128-block now takes 20 us.)
template <typename T, int NT>
__device__ __forceinline__ void unit_upper_inverse(T* U, T* W) {
  constexpr int B = 32, P = kTriPitch<T>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = NT / 32;
  __syncthreads();
  if (warp < 4) {
    T* D = U + warp * B * (P + 1);
    T x[B];
#pragma unroll
    for (int i = 0; i < B; ++i) x[i] = (i == lane) ? T(1) : T(0);
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
    // W (R x 32, row by row) = U_{<j,j} V_jj
    for (int g = warp; g < R / 4; g += nw) {
      T s[4] = {};
#pragma unroll 8
      for (int k = 0; k < B; ++k) {
        T a[4];
        load4(U + 4 * g + (R + k) * P, a);
        const T b = U[R + k + (R + lane) * P];  // zero below V_jj's diagonal
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = fma(a[i], b, s[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) W[(4 * g + i) * B + lane] = s[i];
    }
    __syncthreads();
    for (int g = warp; g < R / 4; g += nw) {
      T s[4] = {};
#pragma unroll 4
      for (int k = 4 * g; k < R; ++k) {
        T a[4];
        load4(U + 4 * g + k * P, a);
        const T b = W[k * B + lane];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = fma(a[i], b, s[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) U[4 * g + i + (R + lane) * P] = -s[i];  // not read by this product
    }
    __syncthreads();
  }
}

}  // namespace bem
