// The two triangle inverses of a window-pivoted FP32 panel's diagonal block (lu.cu), which turn
// its block TRSMs into one product each.
//
// One cooperative launch, the same code for both triangles: the lower one W is taken as the
// transpose of the upper one W^T, by strides.  With U upper and X its inverse,
//   X_bb (128 x 128) in shared memory, one CTA per block and triangle, then block column by
//   block column X_{<b,b} = -(X_{<b,<b} U_{<b,b}) X_bb:
// strips of eight rows are independent, so a CTA forms its strip of X_{<b,<b} U_{<b,b} (8 x 128,
// the k range split over its sixteen warps, 8 x 4 entries per thread), keeps it in shared memory
// and multiplies it by X_bb; a grid barrier ends the block column.  FP32 products and sums.
// Measured at jb = 1,024 by itself: 134 us, the 128-blocks 19, the strips 100 (a chunk of 64 k
// takes 1 us, of which the FMAs are a quarter: its barrier, copies and shared-memory reads bound
// it), the grid barriers 14.  As a chain of 14 small tensor products per triangle with their
// operand splits, copies and two streams the same took 0.7 ms a panel.
#include "grid_sync.cuh"
#include "lu.cuh"
#include "tri_inv.cuh"

namespace bem {
namespace {

constexpr int kNT = 512, kWarps = kNT / 32;
constexpr int kRows = 8;    // rows of a strip
constexpr int kKc = 64;     // k of a staged chunk, four per warp
constexpr int kStages = 3;  // chunks staged
constexpr int kOut = kRows * 128 / kNT;  // entries of a strip per thread
constexpr int kPK = kKc + 4, kPB = 128 + 4;  // pitches: [column or row][k], [k][column]

struct Strip {
  // a chunk of the right factor as it lies in memory: [column][k] (upper) or [k][column]; and
  // of the left one: [k][row] (upper) or [row][k]
  float b[kStages][128 * kPK];
  float a[kStages][kRows * kPK];
  float red[kWarps][kRows * kPB];  // the warps' sums
  float t[128][kRows];             // the first product, [column][row]
};
static_assert(kKc * kPB <= 128 * kPK, "either layout fits");
constexpr size_t kSmem = sizeof(Strip) > kTriElems<float> * sizeof(float) ? sizeof(Strip)
                                                                           : kTriElems<float> * sizeof(float);

__device__ __forceinline__ void cp_async16(float* smem, const float* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem)
               : "memory");
}

// Column of a thread's entry u: the lanes take every 32nd column where four k of a column are one
// 16-byte word, else four neighbouring ones, so that a warp's reads meet every bank.
template <bool UPPER>
__device__ __forceinline__ int col_of(int lane, int u) {
  return UPPER ? lane + 32 * u : 4 * lane + u;
}

// acc (8 rows x 4 columns) += A(row, k) B(k, column) over this warp's four k of a chunk; A is
// [k][row] with K_A, else [row][k]
template <bool UPPER, bool K_A>
__device__ __forceinline__ void chunk_product(const float* a, const float* b, float (&acc)[kRows][4]) {
  const int lane = threadIdx.x & 31, k0 = (threadIdx.x >> 5) * (kKc / kWarps);
  static_assert(kKc / kWarps == 4, "a 16-byte word per column and row");
  float av[kRows][4], bv[4][4];  // [row][k], [column][k] or [k][column]
#pragma unroll
  for (int u = 0; u < 4; ++u) load4(UPPER ? b + col_of<true>(lane, u) * kPK + k0 : b + (k0 + u) * kPB + 4 * lane, bv[u]);
  if (K_A) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float v[4];
        load4(a + (k0 + k) * kRows + 4 * h, v);
#pragma unroll
        for (int r = 0; r < 4; ++r) av[4 * h + r][k] = v[r];
      }
  } else {
#pragma unroll
    for (int r = 0; r < kRows; ++r) load4(a + r * kPK + k0, av[r]);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(av[r][k], UPPER ? bv[c][k] : bv[k][c], acc[r][c]);
}

// the totals of the warps' sums: each thread's entries, row tid % 8 of columns tid / 8 + kNT / 8 u
template <bool UPPER>
__device__ __forceinline__ void reduce(Strip& sm, float (&acc)[kRows][4], float (&out)[kOut]) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
#pragma unroll
  for (int r = 0; r < kRows; ++r)
    if (UPPER) {
#pragma unroll
      for (int u = 0; u < 4; ++u) sm.red[w][r * kPB + lane + 32 * u] = acc[r][u];
    } else {
      *reinterpret_cast<float4*>(&sm.red[w][r * kPB + 4 * lane]) =
          make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kOut; ++u) {
    const int at = (tid % 8) * kPB + tid / 8 + kNT / 8 * u;
    float s = 0.f;
#pragma unroll
    for (int v = 0; v < kWarps; ++v) s += sm.red[v][at];
    out[u] = s;
  }
}

// strip s of block column b: rows [8 s, 8 s + 8)
template <bool UPPER>
__device__ __forceinline__ void strip(Strip& sm, const float* D, int64_t lda, int jb, float* X, int b, int s) {
  const int tid = threadIdx.x, r0 = kRows * s, c0 = 128 * b;
  const int kbeg = r0 / kKc * kKc, n1 = (c0 - kbeg) / kKc, n = n1 + 128 / kKc;  // X(r, k) is zero for k < r
  const float* Xb = X + c0 + (int64_t)c0 * jb;                                   // X_bb
  // chunk i: of X_{<b,<b} and U_{<b,b} for i < n1, then of X_bb.  X(r, k) at X[r + k jb], U(k, c)
  // at D[k + c lda], transposed for the lower triangle
  constexpr int kQ = kKc / 4;  // 16-byte words of a column's k
  auto load = [&](int i) {
    if (i < n) {
      const int st = i % kStages;
      const bool first = i < n1;
      const int k = first ? kbeg + i * kKc : (i - n1) * kKc;
      const int64_t ld = first ? lda : jb;
      const float* B = first ? (UPPER ? D + k + (int64_t)c0 * lda : D + c0 + (int64_t)k * lda)
                             : (UPPER ? Xb + k : Xb + (int64_t)k * jb);
#pragma unroll
      for (int u = 0; u < kKc * 128 / 4 / kNT; ++u) {
        const int q = tid + kNT * u;
        if (UPPER) cp_async16(&sm.b[st][(q / kQ) * kPK + 4 * (q % kQ)], B + 4 * (q % kQ) + (q / kQ) * ld);
        else cp_async16(&sm.b[st][(q / 32) * kPB + 4 * (q % 32)], B + 4 * (q % 32) + (q / 32) * ld);
      }
      if (first && tid < kRows * kKc / 4) {
        if (UPPER) cp_async16(&sm.a[st][4 * tid], X + r0 + 4 * (tid % 2) + (int64_t)(k + tid / 2) * jb);
        else cp_async16(&sm.a[st][(tid / kQ) * kPK + 4 * (tid % kQ)], X + k + 4 * (tid % kQ) + (int64_t)(r0 + tid / kQ) * jb);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[kRows][4] = {}, o[kOut];
  __syncthreads();  // the buffers are free
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) load(i);
  for (int i = 0; i < n; ++i) {
    if (i == n1) {
      reduce<UPPER>(sm, acc, o);
#pragma unroll
      for (int u = 0; u < kOut; ++u) sm.t[tid / 8 + kNT / 8 * u][tid % 8] = o[u];
#pragma unroll
      for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // chunk i (and t) is in, chunk i - 1 is done with
    load(i + kStages - 1);
    if (i < n1) chunk_product<UPPER, UPPER>(sm.a[i % kStages], sm.b[i % kStages], acc);
    else chunk_product<UPPER, true>(&sm.t[(i - n1) * kKc][0], sm.b[i % kStages], acc);
  }
  reduce<UPPER>(sm, acc, o);
#pragma unroll
  for (int u = 0; u < kOut; ++u) {
    const int r = r0 + tid % 8, c = c0 + tid / 8 + kNT / 8 * u;
    X[UPPER ? r + (int64_t)c * jb : c + (int64_t)r * jb] = -o[u];
  }
}

__global__ void __launch_bounds__(kNT, 1)
    panel_inverses_kernel(const float* __restrict__ D, int64_t lda, int jb, float* XU, float* XL, unsigned* barrier,
                          unsigned bar_base, int* status, unsigned long long wait_ns) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_abort;
  __shared__ float s_d[128];
  const int G = gridDim.x, g = blockIdx.x, tid = threadIdx.x, nblk = jb / 128;
  // the diagonal blocks, and zeros in the blocks outside the triangles
  for (int item = g; item < 2 * nblk; item += G) {
    constexpr int P = kTriPitch<float>;
    float* U = reinterpret_cast<float*>(smem_raw);
    const bool lower = item & 1;
    const int o = 128 * (item / 2);
    const float* B = D + o + (int64_t)o * lda;
    __syncthreads();
    if (tid < 128) s_d[tid] = lower ? B[tid + (int64_t)tid * lda] : 1.f;
    __syncthreads();
    // U(a, c), a < c: B(a, c), or for the lower triangle W = N diag(d) the transpose of N,
    // W(c, a) / d(a); then X = U^{-1}, or X(i, j) = U^{-1}(j, i) / d(i)
    for (int base = tid; base < 128 * 128; base += 16 * kNT) {
      float v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int i = (base + u * kNT) % 128, j = (base + u * kNT) / 128;
        v[u] = (lower ? j < i : i < j) ? B[i + (int64_t)j * lda] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int i = (base + u * kNT) % 128, j = (base + u * kNT) / 128;
        if (lower) U[j + i * P] = v[u] / s_d[j];
        else U[i + j * P] = v[u];
      }
    }
    unit_upper_inverse<float, kNT>(U, U + 128 * P);
    float* X = (lower ? XL : XU) + o + (int64_t)o * jb;
    for (int idx = tid; idx < 128 * 128; idx += kNT) {
      const int i = idx % 128, j = idx / 128;
      X[i + (int64_t)j * jb] = lower ? (j <= i ? U[j + i * P] / s_d[i] : 0.f) : U[i + j * P];
    }
  }
  const int free0 = min(2 * nblk, G - 1);  // CTAs past the inverting ones clear
  if (g >= free0)
    for (int64_t q = (int64_t)(g - free0) * kNT + tid; q < (int64_t)jb * jb / 4; q += (int64_t)(G - free0) * kNT) {
      const int64_t at = 4 * q;
      const int i = (int)(at % jb), j = (int)(at / jb);
      if (i / 128 > j / 128) *reinterpret_cast<float4*>(XU + at) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i / 128 < j / 128) *reinterpret_cast<float4*>(XL + at) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  Strip& sm = *reinterpret_cast<Strip*>(smem_raw);
  unsigned target = bar_base;
  for (int b = 1; b < nblk; ++b) {
    target += (unsigned)G;
    if (!coop_barrier(barrier, target, status, wait_ns, &s_abort)) return;
    // the longest strips (the first rows) first
    for (int q = g; q < 2 * (128 / kRows) * b; q += G) {
      if (q & 1) strip<false>(sm, D, lda, jb, XL, b, q / 2);
      else strip<true>(sm, D, lda, jb, XU, b, q / 2);
    }
  }
}

}  // namespace

int panel_inverses_launch(bem_ctx* c, const float* D, int64_t lda, int jb, float* XU, float* XL, unsigned* barrier,
                          unsigned& bar_base, int* status) {
  if (lda % 4 != 0 || (reinterpret_cast<uintptr_t>(D) & 15) != 0 || jb % 128 != 0)
    return bem_fail(c, BEM_ERR_ARG, "panel inverses: the block is not aligned");
  static DeviceOnce attr;
  if (attr.pending()) {
    BEM_CUDA(c, cudaFuncSetAttribute(panel_inverses_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    attr.mark();
  }
  const int G = c->sm_count;
  unsigned bb = bar_base;
  unsigned long long wns = c->wait_ns;
  void* args[] = {&D, &lda, &jb, &XU, &XL, &barrier, &bb, &status, &wns};
  BEM_CUDA(c, cudaLaunchCooperativeKernel((void*)panel_inverses_kernel, dim3(G), dim3(kNT), args, kSmem,
                                          c->stream));
  ++c->launches;
  bar_base += (unsigned)(jb / 128 - 1) * (unsigned)G;
  return BEM_OK;
}

}  // namespace bem
