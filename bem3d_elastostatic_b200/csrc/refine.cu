// Mixed-precision solve (FP32 factors + FP64 iterative refinement against the FP64
// A) and reorganize_solution (io_mod.f90:148-183).
#include <cmath>
#include <limits>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <vector>

#include "lu.cuh"

namespace bem {

// panel width of the FP32 factorisation: at 512 the tcgen05 trailing update has as much
// tensor work per tile as C traffic (measured at 73,734 DOF: 1.79 s per bench step at 256,
// 1.61 s at 384, 1.58 s at 512)
constexpr int kNbMixed = 512;   // panel width of the FP32 factors of BEM_PREC_FP32_IR
constexpr int kNbBf16 = 1024;   // and of BEM_PREC_BF16_IR
constexpr int kNbFp64IR = 512;  // panel width of the FP64 factors of BEM_PREC_FP64_IR

__global__ void to_fp32_kernel(const double* A, int64_t lda, int n, float* A32) {
  const int64_t total = (int64_t)lda * n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
    A32[i] = (float)A[i];
}

// Equilibration of the BF16 mode: power-of-two row scales r_i (row maxima of |A| in
// [1, 2)), then column scales c_j of the row-scaled matrix, so that the factored copy
// r_i A_ij c_j holds entries of magnitude < 2 whatever the units of the unknowns; the
// scales are exact, and the preconditioner of the refinement is c (LU)^-1 r.
__device__ __forceinline__ double pow2_scale(double mx) {
  if (!(mx > 0.0) || !(mx < INFINITY)) return 1.0;
  return exp2(-floor(log2(mx)));
}

// Row maxima of |A| by column chunks: a thread per row and a CTA column range of
// kRowChunk columns, 16 loads in flight per thread; the chunks' maxima meet in rmax
// (the bits of a non-negative double order like the double).  NaNs are skipped by fmax.
constexpr int kRowChunk = 1024;
__global__ void row_max_kernel(const double* __restrict__ A, int64_t lda, int n, unsigned long long* rmax) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int j0 = blockIdx.y * kRowChunk, j1 = min(n, j0 + kRowChunk);
  double mx = 0.0;
  int j = j0;
  for (; j + 16 <= j1; j += 16) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = fabs(A[i + (int64_t)(j + u) * lda]);
#pragma unroll
    for (int u = 0; u < 16; ++u) mx = fmax(mx, v[u]);
  }
  for (; j < j1; ++j) mx = fmax(mx, fabs(A[i + (int64_t)j * lda]));
  atomicMax(rmax + i, (unsigned long long)__double_as_longlong(mx));
}

__global__ void row_scale_kernel(int n, const unsigned long long* __restrict__ rmax, double* __restrict__ rs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) rs[i] = pow2_scale(__longlong_as_double((long long)rmax[i]));
}

// Column scales of the row-scaled matrix and the scaled FP32 copy in one pass per
// column: a CTA reads column j, reduces its maximum, then converts the column again while
// it is still in L2, and walks its columns in turn.  What bounds it is the 64 bytes
// a cycle an SM reads from L2, so the row scales, powers of two, stay in shared memory as
// their exponents (SMEM; orders whose exponents do not fit read them with the column, which
// doubles those bytes), and eight 16-byte loads a thread are in flight throughout, the
// remainder of a column included.  The FP32 copy's padding rows are zero.
// An SM holds 1,024 of its threads, as four CTAs, two or one: with more CTAs one's loads cover
// another's reduction, and short columns leave fewer lanes idle, as long as the columns in
// flight fill no more than half the L2 (kColL2).  Measured (ms at 4,614, 10,374, 18,438,
// 28,806, 41,478 and 56,454 columns): 256 threads 0.063, 0.232, 0.89, 2.42, 6.5 and 14.3; 512
// threads 0.072, 0.294, 0.80, 1.93, 5.5 and 11.3; 1,024 threads 0.136, 0.357, 1.08, 1.93, 4.0
// and 7.7.  A grid of more CTAs than the SMs hold is no faster and at 41,478 takes 5.6.
constexpr int kColThreads = 1024;  // per SM
constexpr int kColLoads = 8;  // double2 per thread and turn
constexpr size_t kColL2 = 64ull << 20;
constexpr int kColSmem = 220 * 1024;
// a power of two from its exponent field; the one subnormal among the scales is 2^-1023
__device__ __forceinline__ double pow2_of_field(unsigned f) {
  return __hiloint2double(f == 0 ? 0x00080000 : (int)(f << 20), 0);
}
template <bool SMEM, int NT>
__global__ void __launch_bounds__(NT) col_scale_convert_kernel(const double* __restrict__ A, int64_t lda, int n,
                                                               const double* __restrict__ rs,
                                                               double* __restrict__ cs, float* A32) {
  extern __shared__ __align__(16) unsigned short s_exp[];  // [n rounded up to even]
  __shared__ double red[NT / 32];
  __shared__ double s_c;
  const int t = threadIdx.x;
  if (SMEM) {
    for (int i = t; i < (n + 1) / 2 * 2; i += NT)
      s_exp[i] = i < n ? (unsigned short)((__double2hiint(rs[i]) >> 20) & 0x7ff) : 1023;
    __syncthreads();
  }
  constexpr int STEP = 2 * NT;
  // rows i and i + 1 of a column, row-scaled; zeros past the matrix
  auto load = [&](const double* a, int i0, double2 (&v)[kColLoads]) {
#pragma unroll
    for (int u = 0; u < kColLoads; ++u) {
      const int i = i0 + u * STEP;
      v[u] = i < n ? *reinterpret_cast<const double2*>(a + i) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < kColLoads; ++u) {
      const int i = i0 + u * STEP;
      if (i < n) {
        if (SMEM) {
          const ushort2 e = *reinterpret_cast<const ushort2*>(s_exp + i);
          v[u].x *= pow2_of_field(e.x);
          v[u].y = i + 1 < n ? v[u].y * pow2_of_field(e.y) : 0.0;
        } else {
          v[u].x *= rs[i];
          v[u].y = i + 1 < n ? v[u].y * rs[i + 1] : 0.0;
        }
      }
    }
  };
  for (int64_t j = blockIdx.x; j < n; j += gridDim.x) {
    const double* a = A + j * lda;
    double mx = 0.0;
    for (int i0 = 2 * t; i0 < n; i0 += kColLoads * STEP) {
      double2 v[kColLoads];
      load(a, i0, v);
#pragma unroll
      for (int u = 0; u < kColLoads; ++u) mx = fmax(mx, fmax(fabs(v[u].x), fabs(v[u].y)));
    }
    for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if ((t & 31) == 0) red[t >> 5] = mx;
    __syncthreads();
    if (t == 0) {
      double m = red[0];
      for (int w = 1; w < NT / 32; ++w) m = fmax(m, red[w]);
      s_c = pow2_scale(m);
      cs[j] = s_c;
    }
    __syncthreads();
    const double c = s_c;
    float* o = A32 + j * lda;
    for (int i0 = 2 * t; i0 < lda; i0 += kColLoads * STEP) {  // lda is even
      double2 v[kColLoads];
      load(a, i0, v);
#pragma unroll
      for (int u = 0; u < kColLoads; ++u) {
        const int i = i0 + u * STEP;
        if (i < lda) *reinterpret_cast<float2*>(o + i) = make_float2((float)(v[u].x * c), (float)(v[u].y * c));
      }
    }
    __syncthreads();  // red and s_c are reused by the next column
  }
}

template <int NT>
int col_scale_convert_as(bem_ctx* c, int n, int64_t lda) {
  const int ctas = std::min(n, kColThreads / NT * c->sm_count);
  const size_t exps = ((size_t)n + 1) / 2 * 2 * sizeof(unsigned short);
  if constexpr (NT == kColThreads)
    if (exps > kColSmem) {
      col_scale_convert_kernel<false, NT>
          <<<ctas, NT, 0, c->stream>>>(c->A.p, lda, n, c->rowscale.p, c->colscale.p, c->A32.p);
      return BEM_OK;
    }
  static DeviceOnce attr;
  if (attr.pending()) {
    BEM_CUDA(c, cudaFuncSetAttribute(col_scale_convert_kernel<true, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kColSmem));
    attr.mark();
  }
  col_scale_convert_kernel<true, NT>
      <<<ctas, NT, exps, c->stream>>>(c->A.p, lda, n, c->rowscale.p, c->colscale.p, c->A32.p);
  return BEM_OK;
}

// colscale and A32 from A and rowscale, by the most CTAs per SM whose columns fit kColL2 (one, if
// none do)
int col_scale_convert(bem_ctx* c, int n, int64_t lda) {
  const size_t columns = kColL2 / ((size_t)lda * sizeof(double));
  if (columns >= (size_t)4 * c->sm_count) return col_scale_convert_as<kColThreads / 4>(c, n, lda);
  if (columns >= (size_t)2 * c->sm_count) return col_scale_convert_as<kColThreads / 2>(c, n, lda);
  return col_scale_convert_as<kColThreads>(c, n, lda);
}

__global__ void mul_kernel(int n, const double* s, double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] *= s[i];
}

__global__ void axpy_kernel(int n, const double* d, double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += d[i];
}

// x += d and dmax = max |d| (non-negative doubles order like their bit patterns)
__global__ void axpy_max_kernel(int n, const double* d, double* x, double* dmax) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (i < n) {
    x[i] += d[i];
    v = fabs(d[i]);
  }
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0 && v > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(dmax), (unsigned long long)__double_as_longlong(v));
}

// ---------------------------------------------------------------------------------
// GMRES-IR building blocks: FP64 vectors, deterministic reductions
// ---------------------------------------------------------------------------------
constexpr int kGmresM = 30;       // restart length
constexpr int kDotBlocks = 296;   // 2 CTAs per SM for the multi-dot partials

// part[b][i] = sum over block b's slice of V[i] . w, i < k
__global__ void __launch_bounds__(256) multidot_kernel(int n, int k, const double* V, int64_t ldv, const double* w,
                                                       double* part) {
  __shared__ double red[8][kGmresM + 1];
  double acc[kGmresM + 1];
#pragma unroll
  for (int i = 0; i <= kGmresM; ++i) acc[i] = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const double we = w[e];
#pragma unroll
    for (int i = 0; i <= kGmresM; ++i)
      if (i < k) acc[i] = fma(V[e + i * ldv], we, acc[i]);
  }
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i <= kGmresM; ++i) {
    double v = acc[i];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) red[wp][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < k) {
    double sacc = 0.0;
    for (int q = 0; q < 8; ++q) sacc += red[q][threadIdx.x];
    part[(int64_t)blockIdx.x * (kGmresM + 1) + threadIdx.x] = sacc;
  }
}

__global__ void reduce_parts_kernel(int nb, int k, const double* part, double* out) {
  const int i = threadIdx.x;
  if (i >= k) return;
  double sacc = 0.0;
  for (int b = 0; b < nb; ++b) sacc += part[(int64_t)b * (kGmresM + 1) + i];
  out[i] = sacc;
}

// w += sign * sum_{i<k} V[i] h[i]
__global__ void vcomb_kernel(int n, int k, const double* V, int64_t ldv, const double* h, double sign, double* w) {
  __shared__ double hs[kGmresM + 1];
  if (threadIdx.x < k) hs[threadIdx.x] = h[threadIdx.x];
  __syncthreads();
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  double sacc = 0.0;
  for (int i = 0; i < k; ++i) sacc = fma(V[e + i * ldv], hs[i], sacc);
  w[e] = fma(sign, sacc, w[e]);
}

__global__ void scale_kernel(int n, double a, const double* x, double* y) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) y[e] = a * x[e];
}

int solve_mixed(bem_ctx* c, int precision, double rel_tol, int max_iter, bem_solve_info* st, int* info) {
  const int n = (int)c->nsys;
  const int64_t lda = c->lda;
  *info = 0;
  if (c->factored_fp64) return bem_fail(c, BEM_ERR_STATE, "A was overwritten by an FP64 factorisation");
  // BEM_IR_PROFILE: host time stamps of the solve's stages (stderr)
  const bool host_prof = getenv("BEM_IR_PROFILE") != nullptr;
  const auto h0 = std::chrono::steady_clock::now();
  auto stamp = [&](const char* what) {
    if (host_prof)
      fprintf(stderr, "[solve host] %-14s %9.3f ms\n", what,
              std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - h0).count());
  };
  // BEM_PREC_FP64_IR factors an FP64 copy of A (partial pivoting) and refines against A
  const bool dbl = (precision == BEM_PREC_FP64_IR);
  if (dbl) {
    if (c->A64f.count != (size_t)(lda * n)) {
      c->A64f.release();
      if (c->A64f.alloc((size_t)(lda * n)) != cudaSuccess)
        return bem_fail(c, BEM_ERR_OOM, "allocating the FP64 factor copy");
    }
  } else if (c->A32.count != (size_t)(lda * n)) {
    c->A32.release();
    cudaError_t e = c->A32.alloc((size_t)(lda * n));
    if (e != cudaSuccess) return bem_fail(c, BEM_ERR_OOM, "allocating the FP32 factor copy");
  }
  // residuals in double-double (the default) or in FP64
  const bool ext = c->ext_residual;
  BEM_CUDA(c, c->piv.alloc(n));
  BEM_CUDA(c, c->perm.alloc(n));
  DBuf<double>& r = c->ir_r;
  DBuf<double>& d = c->ir_d;
  if (r.count != (size_t)n) BEM_CUDA(c, r.alloc(n));
  if (d.count != (size_t)n) BEM_CUDA(c, d.alloc(n));
  {
    // one workspace for the triangular solves and the residual, sized once
    const size_t nchunk = ((size_t)n + 511) / 512;
    const size_t need = std::max(((size_t)n + 127) / 128 * 256 + 256, nchunk * n * 3 + 8);
    if (c->work.count < need) {
      c->work.release();
      BEM_CUDA(c, c->work.alloc(need));
    }
  }
  for (auto& e : c->solve_ev)
    if (!e) BEM_CUDA(c, cudaEventCreate(&e));
  cudaEvent_t e0 = c->solve_ev[0], e1 = c->solve_ev[1], e2 = c->solve_ev[2];
  // Window pivoting first (pivot search within each 32-wide sub-panel's diagonal
  // block: no grid-wide exchange per pivot); if that factorisation meets a zero pivot or
  // its refinement does not converge, the solve is repeated with partial pivoting.
  bool window = c->pivot_pref != BEM_PIVOT_PARTIAL && !dbl;
  int fallbacks = 0;
  double berr = 1.0;
  int it = 0, restarts = 0;
  const bool use_gmres = (precision == BEM_PREC_BF16_IR);
  int rc = BEM_OK;
  for (;;) {
  BEM_CUDA(c, cudaEventRecord(e0, c->stream));
  const bool scaled = (precision == BEM_PREC_BF16_IR);
  if (scaled) {
    BEM_CUDA(c, c->rowscale.alloc(n));
    BEM_CUDA(c, c->colscale.alloc(n));
    // the column scales' buffer holds the row maxima until the column pass
    unsigned long long* rmax = reinterpret_cast<unsigned long long*>(c->colscale.p);
    BEM_CUDA(c, cudaMemsetAsync(rmax, 0, (size_t)n * sizeof(unsigned long long), c->stream));
    row_max_kernel<<<dim3((n + 255) / 256, (n + kRowChunk - 1) / kRowChunk), 256, 0, c->stream>>>(c->A.p, lda, n,
                                                                                                  rmax);
    BEM_LAUNCH_CHECK(c);
    row_scale_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(n, rmax, c->rowscale.p);
    BEM_LAUNCH_CHECK(c);
    if ((rc = col_scale_convert(c, n, lda))) return rc;
  } else if (dbl) {
    BEM_CUDA(c, cudaMemcpyAsync(c->A64f.p, c->A.p, (size_t)lda * n * sizeof(double), cudaMemcpyDeviceToDevice,
                                c->stream));
  } else {
    to_fp32_kernel<<<c->sm_count * 8, 256, 0, c->stream>>>(c->A.p, lda, n, c->A32.p);
  }
  BEM_LAUNCH_CHECK(c);
  // v := M^{-1} v with M the factored copy: c (LU)^{-1} r in the scaled mode
  auto psolve = [&](double* v) -> int {
    if (scaled) {
      mul_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(n, c->rowscale.p, v);
      BEM_LAUNCH_CHECK(c);
    }
    int prc = dbl ? lu_solve<double>(c, c->A64f.p, lda, n, c->perm.p, v)
                  : lu_solve<float>(c, c->A32.p, lda, n, c->perm.p, v);
    if (prc) return prc;
    if (scaled) {
      mul_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(n, c->colscale.p, v);
      BEM_LAUNCH_CHECK(c);
    }
    return BEM_OK;
  };
  const int saved = c->f32_gemm;
  if (c->f32_gemm_override >= 0)
    c->f32_gemm = c->f32_gemm_override;
  else
    c->f32_gemm = (precision == BEM_PREC_BF16_IR) ? 2 : 4;
  // the one-product update is HBM-bound (the FP32 trailing matrix is read and written
  // once per panel): the wider panel halves that traffic; the three-product update is
  // tensor-bound
  const int nb = c->panel_width > 0 ? c->panel_width : (precision == BEM_PREC_BF16_IR ? kNbBf16 : kNbMixed);
  stamp("enqueued");
  c->lu_window = window;
  rc = dbl ? lu_factor<double>(c, c->A64f.p, lda, n, c->piv.p, c->perm.p, kNbFp64IR, info)
           : lu_factor<float>(c, c->A32.p, lda, n, c->piv.p, c->perm.p, nb, info);
  c->lu_window = false;
  c->f32_gemm = saved;
  if (rc) return rc;
  stamp("factored");
  BEM_CUDA(c, cudaEventRecord(e1, c->stream));
  if (*info != 0) {
    if (window) {  // a zero pivot inside a window: partial pivoting may still succeed
      window = false;
      ++fallbacks;
      *info = 0;
      continue;
    }
    return BEM_OK;
  }
  // x0 = LU^{-1} b, then x += LU^{-1} (b - A x)   (plain refinement), or
  // x += GMRES(M^{-1} A, M^{-1} r) with M = the low-precision LU (GMRES-IR)
  BEM_CUDA(c, cudaMemsetAsync(c->X.p, 0, n * sizeof(double), c->stream));
  BEM_CUDA(c, cudaMemcpyAsync(r.p, c->FI.p, n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  double norms[4] = {0, 0, 0, 0};
  double anorm = -1.0, prev = 1e300, prev_d = 1e300;
  if (c->ir_dmax.count < 1) BEM_CUDA(c, c->ir_dmax.alloc(1));
  berr = 1.0;
  it = 0;
  restarts = 0;
  const bool ir_prof = getenv("BEM_IR_PROFILE") != nullptr;
  if (!use_gmres) {
    cudaEvent_t q0, q1, q2;
    if (ir_prof) {
      cudaEventCreate(&q0);
      cudaEventCreate(&q1);
      cudaEventCreate(&q2);
    }
    for (it = 1; it <= max_iter; ++it) {
      if (ir_prof) cudaEventRecord(q0, c->stream);
      BEM_CUDA(c, cudaMemcpyAsync(d.p, r.p, n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
      if ((rc = psolve(d.p))) return rc;
      BEM_CUDA(c, cudaMemsetAsync(c->ir_dmax.p, 0, sizeof(double), c->stream));
      axpy_max_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(n, d.p, c->X.p, c->ir_dmax.p);
      BEM_LAUNCH_CHECK(c);
      if (ir_prof) cudaEventRecord(q1, c->stream);
      double dmax = 0.0;
      BEM_CUDA(c, cudaMemcpyAsync(&dmax, c->ir_dmax.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
      if ((rc = residual_fp64(c, c->A.p, lda, n, c->X.p, c->FI.p, r.p, norms, anorm < 0, ext))) return rc;
      if (ir_prof) {
        cudaEventRecord(q2, c->stream);
        cudaEventSynchronize(q2);
        float a = 0.f, b2 = 0.f;
        cudaEventElapsedTime(&a, q0, q1);
        cudaEventElapsedTime(&b2, q1, q2);
        fprintf(stderr, "[ir it=%d] lu-solve %.2f ms residual %.2f ms\n", it, a, b2);
      }
      if (anorm < 0) anorm = norms[3];
      berr = norms[0] / (anorm * norms[1] + norms[2]);
      if (!(berr == berr)) break;  // NaN: diverged
      if (!ext) {
        if (berr <= rel_tol) break;
        if (berr > 0.5 * prev && it > 3) break;  // stagnation
      } else {
        // with exact residuals the iterates approach the solution of the stored system
        // itself: stop once the backward error meets the tolerance and the last
        // correction is below it relative to x (at the default tolerances: below 4 units
        // of roundoff of x), or the corrections stop shrinking (they then only carry
        // x's rounding)
        const double u = 1.1102230246251565e-16;
        if (berr <= rel_tol && dmax <= std::max(4.0 * u, rel_tol) * norms[1]) break;
        if (it > 3 && dmax > 0.5 * prev_d && berr > 0.5 * prev) break;
        prev_d = dmax;
      }
      prev = berr;
    }
  } else {
    // GMRES-IR: Krylov basis V (kGmresM + 1 vectors), FP64; Hessenberg least squares
    // by Givens rotations on the host
    const int64_t ldv = ((int64_t)n + 31) / 32 * 32;
    // the Krylov basis and the reduction buffers are kept in the context (allocation
    // and release next to a 10^10-byte system stall the host)
    DBuf<double>& Vb = c->gm_V;
    DBuf<double>& hd = c->gm_h;
    DBuf<double>& part = c->gm_part;
    DBuf<double>& zero = c->gm_zero;
    if (Vb.count != (size_t)ldv * (kGmresM + 1)) BEM_CUDA(c, Vb.alloc((size_t)ldv * (kGmresM + 1)));
    if (hd.count != 2 * (size_t)(kGmresM + 1)) BEM_CUDA(c, hd.alloc(2 * (kGmresM + 1)));
    if (part.count != (size_t)kDotBlocks * (kGmresM + 1)) BEM_CUDA(c, part.alloc((size_t)kDotBlocks * (kGmresM + 1)));
    if (zero.count != (size_t)n) BEM_CUDA(c, zero.alloc(n));
    BEM_CUDA(c, cudaMemsetAsync(zero.p, 0, n * sizeof(double), c->stream));
    double* V = Vb.p;
    const int vb = (n + 255) / 256;
    auto dots = [&](int k, const double* w, double* out_host) -> int {
      multidot_kernel<<<kDotBlocks, 256, 0, c->stream>>>(n, k, V, ldv, w, part.p);
      BEM_LAUNCH_CHECK(c);
      reduce_parts_kernel<<<1, 32, 0, c->stream>>>(kDotBlocks, k, part.p, hd.p);
      BEM_LAUNCH_CHECK(c);
      BEM_CUDA(c, cudaMemcpyAsync(out_host, hd.p, k * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
      BEM_CUDA(c, cudaStreamSynchronize(c->stream));
      return BEM_OK;
    };
    auto norm2 = [&](const double* w, double* out) -> int {
      // ||w||_2 through the multi-dot with V[0] temporarily replaced is awkward; use a
      // dedicated pass over w . w
      multidot_kernel<<<kDotBlocks, 256, 0, c->stream>>>(n, 1, w, ldv, w, part.p);
      BEM_LAUNCH_CHECK(c);
      reduce_parts_kernel<<<1, 32, 0, c->stream>>>(kDotBlocks, 1, part.p, hd.p);
      BEM_LAUNCH_CHECK(c);
      double v2 = 0.0;
      BEM_CUDA(c, cudaMemcpyAsync(&v2, hd.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
      BEM_CUDA(c, cudaStreamSynchronize(c->stream));
      *out = std::sqrt(v2);
      return BEM_OK;
    };
    const double inner_tol = 1e-6;
    for (restarts = 0; restarts < max_iter; ++restarts) {
      if (restarts == 0) {
        // x = 0: the residual is b itself (r holds a copy) and the backward error
        // |r| / (|A| |x| + |b|) is 1, or undefined for b = 0, without a pass over A;
        // the matrix norm comes with the next residual
        double bn = 0.0;
        if ((rc = norm2(r.p, &bn))) return rc;
        berr = bn > 0.0 ? 1.0 : std::numeric_limits<double>::quiet_NaN();
      } else {
        if ((rc = residual_fp64(c, c->A.p, lda, n, c->X.p, c->FI.p, r.p, norms, anorm < 0, ext))) return rc;
        if (anorm < 0) anorm = norms[3];
        berr = norms[0] / (anorm * norms[1] + norms[2]);
      }
      if (!(berr == berr) || berr <= rel_tol) break;
      if (berr > 0.5 * prev && restarts > 3) break;  // stagnation
      prev = berr;
      // v0 = M^{-1} r / beta
      BEM_CUDA(c, cudaMemcpyAsync(V, r.p, n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
      if ((rc = psolve(V))) return rc;
      double beta = 0.0;
      if ((rc = norm2(V, &beta))) return rc;
      if (!(beta > 0.0)) break;
      scale_kernel<<<vb, 256, 0, c->stream>>>(n, 1.0 / beta, V, V);
      BEM_LAUNCH_CHECK(c);
      double H[kGmresM + 1][kGmresM] = {}, cs[kGmresM] = {}, sn[kGmresM] = {}, g[kGmresM + 1] = {};
      g[0] = beta;
      int kdim = 0;
      for (int j = 0; j < kGmresM; ++j) {
        double* w = V + (int64_t)(j + 1) * ldv;
        // w = M^{-1} A v_j  (residual_fp64 with b = 0 gives -A v_j)
        if ((rc = residual_fp64(c, c->A.p, lda, n, V + (int64_t)j * ldv, zero.p, w, norms, false))) return rc;
        if ((rc = psolve(w))) return rc;
        scale_kernel<<<vb, 256, 0, c->stream>>>(n, -1.0, w, w);
        BEM_LAUNCH_CHECK(c);
        // classical Gram-Schmidt, twice
        double h1[kGmresM + 1], h2[kGmresM + 1];
        if ((rc = dots(j + 1, w, h1))) return rc;
        BEM_CUDA(c, cudaMemcpyAsync(hd.p, h1, (j + 1) * sizeof(double), cudaMemcpyHostToDevice, c->stream));
        vcomb_kernel<<<vb, 256, 0, c->stream>>>(n, j + 1, V, ldv, hd.p, -1.0, w);
        BEM_LAUNCH_CHECK(c);
        if ((rc = dots(j + 1, w, h2))) return rc;
        BEM_CUDA(c, cudaMemcpyAsync(hd.p, h2, (j + 1) * sizeof(double), cudaMemcpyHostToDevice, c->stream));
        vcomb_kernel<<<vb, 256, 0, c->stream>>>(n, j + 1, V, ldv, hd.p, -1.0, w);
        BEM_LAUNCH_CHECK(c);
        for (int i = 0; i <= j; ++i) H[i][j] = h1[i] + h2[i];
        double hn = 0.0;
        if ((rc = norm2(w, &hn))) return rc;
        H[j + 1][j] = hn;
        if (hn > 0.0) {
          scale_kernel<<<vb, 256, 0, c->stream>>>(n, 1.0 / hn, w, w);
          BEM_LAUNCH_CHECK(c);
        }
        // apply the previous rotations, then a new one for (H[j][j], H[j+1][j])
        for (int i = 0; i < j; ++i) {
          const double a = H[i][j], b2 = H[i + 1][j];
          H[i][j] = cs[i] * a + sn[i] * b2;
          H[i + 1][j] = -sn[i] * a + cs[i] * b2;
        }
        const double a = H[j][j], b2 = H[j + 1][j];
        const double rr = std::hypot(a, b2);
        cs[j] = rr > 0 ? a / rr : 1.0;
        sn[j] = rr > 0 ? b2 / rr : 0.0;
        H[j][j] = rr;
        H[j + 1][j] = 0.0;
        g[j + 1] = -sn[j] * g[j];
        g[j] = cs[j] * g[j];
        ++it;
        kdim = j + 1;
        if (std::fabs(g[j + 1]) <= inner_tol * beta || hn == 0.0) break;
      }
      // y = H^{-1} g, x += V y
      double y[kGmresM] = {};
      for (int i = kdim - 1; i >= 0; --i) {
        double sacc = g[i];
        for (int q = i + 1; q < kdim; ++q) sacc -= H[i][q] * y[q];
        y[i] = sacc / H[i][i];
      }
      BEM_CUDA(c, cudaMemcpyAsync(hd.p, y, kdim * sizeof(double), cudaMemcpyHostToDevice, c->stream));
      vcomb_kernel<<<vb, 256, 0, c->stream>>>(n, kdim, V, ldv, hd.p, 1.0, c->X.p);
      BEM_LAUNCH_CHECK(c);
      BEM_CUDA(c, cudaStreamSynchronize(c->stream));
    }
  }
  stamp("refined");
  BEM_CUDA(c, cudaEventRecord(e2, c->stream));
  BEM_CUDA(c, cudaEventSynchronize(e2));
  stamp("synchronised");
  if (window && !(berr <= std::max(rel_tol, 1e-14))) {  // no convergence: partial pivoting
    window = false;
    ++fallbacks;
    continue;
  }
  break;
  }  // attempts
  float f_ms = 0.f, r_ms = 0.f;
  cudaEventElapsedTime(&f_ms, e0, e1);
  cudaEventElapsedTime(&r_ms, e1, e2);
  if (st) {
    st->iterations = use_gmres ? it : std::min(it, max_iter);
    st->restarts = restarts;
    st->rel_residual = berr;
    st->factor_seconds = f_ms * 1e-3;
    st->refine_seconds = r_ms * 1e-3;
    st->gflops = f_ms > 0 ? (2.0 / 3.0) * (double)n * n * n / (f_ms * 1e-3) * 1e-9 : 0.0;
    st->pivoting = window ? BEM_PIVOT_WINDOW : BEM_PIVOT_PARTIAL;
    st->fallbacks = fallbacks;
  }
  // Stagnation at the FP64 working-precision floor counts as converged: a requested
  // tolerance below ~1e-14 is met "to working precision".
  if (!(berr <= std::max(rel_tol, 1e-14)))
    return bem_fail(c, BEM_ERR_NOCONV, "refinement did not reach the tolerance");
  return BEM_OK;
}

// reorganize_solution: DFI(3k+ld, e) = x(3ik+ld) * mu where u is prescribed on the
// element, else the prescribed traction; FI(3i+ld) = prescribed u where an adjacent
// element prescribes it (first in ke order: the uknown/vp lookup), else x.
__global__ void reorganize_dfi_kernel(int ne, const int* nconec, const int* kconec, const int* kode,
                                      const double* bc, const double* X, double mu, double* DFI) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 27 * (int64_t)ne) return;
  const int e = (int)(i / 27), q = (int)(i % 27), k = q / 3, ld = q % 3;
  double v = 0.0;
  if (k < nconec[e]) {
    if (kode[3 * e + ld] == 0)
      v = X[3 * (int64_t)(kconec[k + 9 * e] - 1) + ld] * mu;
    else
      v = bc[i];
  }
  DFI[i] = v;
}

__global__ void reorganize_fi_kernel(int n3, const int* uknown, const double* vp, const double* X, double* FI) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) FI[i] = uknown[i] ? vp[i] : X[i];
}

int launch_reorganize(bem_ctx* c) {
  BEM_CUDA(c, c->DFI.alloc(27 * (size_t)c->ne));
  const int64_t nd = 27 * (int64_t)c->ne;
  reorganize_dfi_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, c->stream>>>(c->ne, c->nconec.p, c->kconec.p,
                                                                             c->kode.p, c->bc.p, c->X.p, c->mat.mu,
                                                                             c->DFI.p);
  BEM_LAUNCH_CHECK(c);
  const int n3 = 3 * c->n;
  BEM_CUDA(c, c->U.alloc(n3));
  reorganize_fi_kernel<<<(n3 + 255) / 256, 256, 0, c->stream>>>(n3, c->uknown.p, c->vp.p, c->X.p, c->U.p);
  BEM_LAUNCH_CHECK(c);
  return BEM_OK;
}

}  // namespace bem
