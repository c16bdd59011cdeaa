// LU, substitution and refinement of a batch of systems (batch.cu), panel by panel over all
// systems at once.
//
// A batch has systems of very different orders, and the largest bound its time when each one
// ran on its own CTA (2,598 unknowns: 150 ms for the FP32 LU, 4 ms for one substitution of
// eight load cases, whatever the other SMs did).  Here every launch covers one step of every
// system that still has one, the systems ordered by size:
//   LU, two 32-column panels a step (LAPACK's right-looking dgetrf with 64 columns a step):
//     batch_panel_kernel   the panel of a system on one cluster (panel_cluster.cuh)
//     batch_swap_kernel    its interchanges on the other columns, and its rows of U12
//     batch_update_kernel  after the first panel the second one's columns, after the second
//                          A22 -= L21 U12, in register-tiled FMA tiles
//     Bound: the panel's 32 exchanges (about 50 us for a system of 2,598 with four rows per
//     thread) while few systems remain, the update's traffic (the trailing matrices read and
//     written once a step; one panel a step moved twice as much) for many.
//   Systems above the cluster's capacity take the one-CTA LU (batch_lu_kernel).
//   Substitution, 128 rows a step, FP64 arithmetic on the factors, all load cases at once:
//     the diagonal blocks are inverted once (batch_inv_kernel); at step k every block row
//     subtracts the tile times the block solved by the step before, and block k's CTA
//     multiplies by its inverse (batch_step_kernel).
//   Residual: one CTA per 128 rows, the columns streamed once for all load cases.
// Measured on 96 boxes of 78 to 2,598 unknowns with eight load cases: FP32 LU 155 -> 14.2 ms, ten
// sweeps 42 -> 6.8 ms, residuals 15.9 -> 2.7 ms.
#include <math_constants.h>

#include <algorithm>
#include <climits>

#include "batch_dev.cuh"
#include "panel_cluster.cuh"
#include "tri_inv.cuh"

namespace bem {
namespace {

constexpr int kLuNB = 32;  // panel width
constexpr int kPanelNT = 256;

// ---- LU ----------------------------------------------------------------------------------

template <typename T, int LPT>
__global__ void __launch_bounds__(kPanelNT, 1)
    batch_panel_kernel(const SysDev* __restrict__ sys, const int* __restrict__ order, T* F, int j0, int C, int* piv,
                       int* info, int* moved, int* err, unsigned long long wait_ns, int withhold) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Sm = PanelSmem<T, LPT, kPanelNT>;
  Sm& sm = *reinterpret_cast<Sm*>(smem_raw);
  const int tid = threadIdx.x;
  const int s = order[blockIdx.x / C], rank = blockIdx.x % C;
  const int N = sys[s].N, w = min(kLuNB, N - j0);
  const int64_t lda = sys[s].lda;
  T* A = F + sys[s].f_off;
  const int base = j0 + rank * Sm::kLines, nl = max(0, min(Sm::kLines, N - base));
  const PanelStep P{N, j0, w, piv + sys[s].piv_off, info + s, wait_ns, withhold};
  const bool ok = panel_on_cluster<T, LPT, kPanelNT>(P, sm, C, rank, base, nl, [&](T(&v)[LPT][kPanelW]) {
#pragma unroll
    for (int q = 0; q < LPT; ++q)
#pragma unroll
      for (int j = 0; j < kPanelW; ++j)
        v[q][j] = (tid + q * kPanelNT < nl && j < w) ? A[base + tid + q * kPanelNT + (int64_t)(j0 + j) * lda] : T(0);
  });
  if (!ok) {
    if (tid == 0) atomicCAS(err, 0, BEM_ERR_TIMEOUT);
    return;
  }
  int* top = moved + 64 * s;  // the rows that end at j0 + q; [32..): where row j0 + q ends
  for (int c = tid; c < nl; c += kPanelNT) {
    const int p = sm.pos[c], row = base + c;
    for (int j = 0; j < w; ++j) A[p + (int64_t)(j0 + j) * lda] = sm.val[j * Sm::kPitchL + c];
    if (p < j0 + w) top[p - j0] = row;
    if (row < j0 + w) top[32 + row - j0] = p;
  }
}

// One column per thread: the interchanges of the panel at j0 (a row of its block that leaves it
// ends where a pivot came from), then, from column t0 on, its rows of U12: for the second panel
// of a step (jp = j0 - 32 the first one's columns, else -1) less the first panel's part, then
// the unit lower solve.  part 0: all columns but the panel's own and, with jp >= 0, the first
// panel's, which part 1 has interchanged by then.
template <typename T, bool SECOND>
__global__ void __launch_bounds__(128) batch_swap_kernel(const SysDev* __restrict__ sys, const int* __restrict__ order,
                                                         T* F, int j0, int t0, int part,
                                                         const int* __restrict__ moved) {
  constexpr int V = 16 / sizeof(T), LP = kLuNB + V;
  struct alignas(16) Vec {
    T v[V];
  };
  __shared__ int s_src[kLuNB], s_dst[kLuNB];
  __shared__ __align__(16) T s_L[kLuNB][LP];  // rows, read as 16-byte broadcasts
  __shared__ __align__(16) T s_P[SECOND ? kLuNB : 1][LP];  // the first panel's multipliers
  const int s = order[blockIdx.y], tid = threadIdx.x, jp = j0 - kLuNB;
  const int N = sys[s].N, w = min(kLuNB, N - j0), b1 = j0 + w;
  if ((int)blockIdx.x * 128 >= N) return;
  const int64_t lda = sys[s].lda;
  T* A = F + sys[s].f_off;
  bool any = false;
  if (tid < kLuNB) {
    s_src[tid] = tid < w ? checked_index(moved[64 * s + tid], j0, N, j0 + tid) : j0 + tid;
    s_dst[tid] = tid < w ? checked_index(moved[64 * s + 32 + tid], j0, N, j0 + tid) : j0 + tid;
    any = s_src[tid] != j0 + tid;
  }
  for (int i = tid; i < kLuNB * kLuNB; i += 128) {
    const int r = i % kLuNB, c = i / kLuNB;
    s_L[r][c] = (r < w && c < r) ? A[j0 + r + (int64_t)(j0 + c) * lda] : T(0);
    if (SECOND && part == 0) s_P[r][c] = r < w ? A[j0 + r + (int64_t)(jp + c) * lda] : T(0);
  }
  any = __syncthreads_or(any);
  const int c = part == 1 ? jp + tid : (int)blockIdx.x * 128 + tid;
  if (part == 1 ? tid >= kLuNB || !any : c >= N || (c >= (SECOND ? jp : j0) && c < b1) || (c < t0 && !any)) return;
  T* col = A + (int64_t)c * lda;
  // rows j0 .. j0 + 31: lda is a multiple of 32, so they lie in the column even where w < 32
  T x[kLuNB];
#pragma unroll
  for (int q = 0; q < kLuNB; q += V) {
    const Vec v = *reinterpret_cast<const Vec*>(col + j0 + q);
#pragma unroll
    for (int u = 0; u < V; ++u) x[q + u] = v.v[u];
  }
  if (any) {
    T y[kLuNB];
#pragma unroll
    for (int q = 0; q < kLuNB; ++q) y[q] = (q >= w || s_src[q] < b1) ? T(0) : col[s_src[q]];
    // rows that leave the block; within it they move between registers
#pragma unroll
    for (int q = 0; q < kLuNB; ++q)
      if (q < w && s_dst[q] >= b1) col[s_dst[q]] = x[q];
#pragma unroll
    for (int q = 0; q < kLuNB; ++q)
      if (s_src[q] < b1 && q < w) y[q] = col[s_src[q]];  // as they were: the block is written last
#pragma unroll
    for (int q = 0; q < kLuNB; ++q) x[q] = q < w ? y[q] : x[q];
  }
  if (c >= t0) {
    if constexpr (SECOND) {
      T u1[kLuNB];
#pragma unroll
      for (int q = 0; q < kLuNB; q += V) {
        const Vec v = *reinterpret_cast<const Vec*>(col + jp + q);
#pragma unroll
        for (int u = 0; u < V; ++u) u1[q + u] = v.v[u];
      }
#pragma unroll
      for (int q = 0; q < kLuNB; ++q)
#pragma unroll
        for (int t = 0; t < kLuNB; t += V) {
          const Vec l = *reinterpret_cast<const Vec*>(&s_P[q][t]);
#pragma unroll
          for (int u = 0; u < V; ++u) x[q] = fma(-l.v[u], u1[t + u], x[q]);
        }
    }
#pragma unroll
    for (int q = 1; q < kLuNB; ++q) {
      T v = x[q];
#pragma unroll
      for (int t = 0; t < q; t += V) {
        const Vec l = *reinterpret_cast<const Vec*>(&s_L[q][t]);
#pragma unroll
        for (int u = 0; u < V; ++u)
          if (t + u < q) v -= l.v[u] * x[t + u];
      }
      x[q] = v;
    }
  }
#pragma unroll
  for (int q = 0; q < kLuNB; q += V) {
    Vec v;
#pragma unroll
    for (int u = 0; u < V; ++u) v.v[u] = x[q + u];
    *reinterpret_cast<Vec*>(col + j0 + q) = v;
  }
}

// A(t0.., t0..cend) -= A(t0.., j0..j0+k) A(j0..j0+k, t0..cend), k 32 or 64: tiles of
// 16 M x 16 M entries, M x M per thread in 16-byte vectors of rows.  Bound by the loads of a tile
// that no arithmetic covers, so all of them are under way at once: the tile itself to registers,
// the operand tiles of both 32-step halves to shared memory (cp.async; U12 as it lies, its steps
// along the fast index).  FP32: two CTAs per SM at 128 registers.  The 81 launches of the batch
// above: 18.9 ms with one CTA per SM and loads through registers, 13.6 ms with two, 10.8 ms with
// two panels a step, 8.4 ms with every load ahead (the inner loop rolled: unrolled twice it spills,
// 9.2 ms).
template <typename T>
struct UpdateTile {
  static constexpr int V = 16 / sizeof(T);           // entries per vector
  static constexpr int M = sizeof(T) == 4 ? 8 : 4;   // entries per thread and direction
  static constexpr int TILE = 16 * M;
  static constexpr int KU = 8 / sizeof(T);           // steps per load of U12
  static constexpr int PB = kLuNB + V;               // a column's pitch in s_b
  struct Half {                                      // operands of 32 steps
    T a[kLuNB][TILE];  // [step][row]
    T b[TILE][PB];     // [column][step]
  };
};
// 16 bytes global -> shared, zeros unless `in`
__device__ __forceinline__ void copy_16(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
template <typename T>
__global__ void __launch_bounds__(256, 2) batch_update_kernel(const SysDev* __restrict__ sys,
                                                              const int* __restrict__ order, T* F, int j0, int k,
                                                              int t0, int cend) {
  using U = UpdateTile<T>;
  constexpr int V = U::V, M = U::M, TILE = U::TILE, H = M / V, KU = U::KU;
  struct alignas(16) Vec {
    T v[V];
  };
  struct alignas(8) Steps {
    T v[KU];
  };
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typename U::Half* sm = reinterpret_cast<typename U::Half*>(smem_raw);  // [k / 32]
  const int s = order[blockIdx.y];
  const int N = sys[s].N, tiles = (N - t0 + TILE - 1) / TILE, C = min(N, cend);
  if ((int)blockIdx.x >= tiles * ((C - t0 + TILE - 1) / TILE)) return;
  const int64_t lda = sys[s].lda;
  T* A = F + sys[s].f_off;
  const int rb = t0 + (blockIdx.x % tiles) * TILE, cb = t0 + (blockIdx.x / tiles) * TILE;
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  // rows up to lda (a multiple of 32, zero beyond N) and columns up to C
  const int halves = k / kLuNB;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h < halves) {
      const int k0 = j0 + h * kLuNB;
#pragma unroll
      for (int u = 0; u < kLuNB * TILE / V / 256; ++u) {
        const int i = tid + u * 256, q = i / (TILE / V), r = (i % (TILE / V)) * V;
        const bool in = rb + r < lda;
        copy_16(&sm[h].a[q][r], in ? A + rb + r + (int64_t)(k0 + q) * lda : A, in);
      }
#pragma unroll
      for (int u = 0; u < kLuNB * TILE / V / 256; ++u) {
        const int i = tid + u * 256, c = i / (kLuNB / V), q = (i % (kLuNB / V)) * V;
        const bool in = cb + c < C;
        copy_16(&sm[h].b[c][q], in ? A + k0 + q + (int64_t)(cb + c) * lda : A, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  T acc[M][M];  // [column][row]
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const int c = cb + ty + 16 * j;
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int r = rb + h * 16 * V + tx * V;
      Vec x{};
      if (c < C && r < lda) x = *reinterpret_cast<const Vec*>(A + r + (int64_t)c * lda);
#pragma unroll
      for (int u = 0; u < V; ++u) acc[j][h * V + u] = x.v[u];
    }
  }
  for (int h = 0; h < halves; ++h) {
    if (h == 0) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const typename U::Half& S = sm[h];
#pragma unroll 1
    for (int q = 0; q < kLuNB; q += KU) {
      Steps b[M];
#pragma unroll
      for (int j = 0; j < M; ++j) b[j] = *reinterpret_cast<const Steps*>(&S.b[ty + 16 * j][q]);
#pragma unroll
      for (int w = 0; w < KU; ++w) {
        T a[M];
#pragma unroll
        for (int g = 0; g < H; ++g) {
          const Vec va = *reinterpret_cast<const Vec*>(&S.a[q + w][g * 16 * V + tx * V]);
#pragma unroll
          for (int u = 0; u < V; ++u) a[g * V + u] = va.v[u];
        }
#pragma unroll
        for (int j = 0; j < M; ++j)
#pragma unroll
          for (int i = 0; i < M; ++i) acc[j][i] = fma(-a[i], b[j].v[w], acc[j][i]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const int c = cb + ty + 16 * j;
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int r = rb + h * 16 * V + tx * V;
      Vec x;
#pragma unroll
      for (int u = 0; u < V; ++u) x.v[u] = acc[j][h * V + u];
      if (c < C && r < lda) *reinterpret_cast<Vec*>(A + r + (int64_t)c * lda) = x;
    }
  }
}

// The largest system that one cluster holds: 16 CTAs of 256 threads with LPT rows each.
template <typename T>
constexpr int kMaxLpt = sizeof(T) == 4 ? 4 : 2;

template <typename T, int LPT>
bool panel_step(BatchSolve& b, T* F, int j0, int active, int C) {
  ++b.launches;
  return launch_clusters(batch_panel_kernel<T, LPT>, active, C, kPanelNT, sizeof(PanelSmem<T, LPT, kPanelNT>),
                         b.stream, b.sys, b.order, F, j0, C, b.piv, b.info, b.moved, b.err, b.wait_ns,
                         b.withhold_pivot) == cudaSuccess;
}

// systems (the first ones in order) of at least n rows
int active_from(const BatchSolve& b, int n) {
  return (int)(std::upper_bound(b.N.begin(), b.N.end(), n, [](int v, int x) { return v > x; }) - b.N.begin());
}

// the panel at j0, its interchanges and its rows of U12 from column t0 on
template <typename T, bool SECOND>
bool panel_and_rows(BatchSolve& b, T* F, int j0, int t0) {
  const int maxN = b.N[0], active = active_from(b, j0 + 1), rows = maxN - j0;
  // the fewest rows per thread (the shortest steps) with which all clusters run at once; else as
  // many as fit, so that fewer waves of clusters are needed
  auto ctas = [&](int l) {
    int c = 1;
    while (c * kPanelNT * l < rows) c *= 2;
    return c;
  };
  int lpt = 1;
  for (; lpt < kMaxLpt<T>; lpt *= 2)
    if (ctas(lpt) <= kMaxCluster && active * ctas(lpt) <= b.sm_count) break;
  const int C = ctas(lpt);
  bool ok = true;
  if (lpt == 1) ok = panel_step<T, 1>(b, F, j0, active, C);
  else if (lpt == 2) ok = panel_step<T, 2>(b, F, j0, active, C);
  else if constexpr (kMaxLpt<T> >= 4) ok = panel_step<T, 4>(b, F, j0, active, C);
  if (!ok) return false;
  if (SECOND) {  // the first panel's multipliers, which the launch below reads
    batch_swap_kernel<T, SECOND><<<dim3(1, active), 128, 0, b.stream>>>(b.sys, b.order, F, j0, t0, 1, b.moved);
    ++b.launches;
  }
  batch_swap_kernel<T, SECOND>
      <<<dim3((maxN + 127) / 128, active), 128, 0, b.stream>>>(b.sys, b.order, F, j0, t0, 0, b.moved);
  ++b.launches;
  return cudaGetLastError() == cudaSuccess;
}

// A(t0.., t0..cend) -= A(t0.., j0..j0+k) A(j0..j0+k, t0..cend) of every system that reaches t0
template <typename T>
bool update(BatchSolve& b, T* F, int j0, int k, int t0, int cend) {
  const int left = active_from(b, t0 + 1);
  if (left == 0) return true;
  constexpr int TILE = UpdateTile<T>::TILE;
  const int rt = (b.N[0] - t0 + TILE - 1) / TILE, ct = (std::min(b.N[0], cend) - t0 + TILE - 1) / TILE;
  batch_update_kernel<T><<<dim3(rt * ct, left), 256, (k / kLuNB) * sizeof(typename UpdateTile<T>::Half), b.stream>>>(
      b.sys, b.order, F, j0, k, t0, cend);
  ++b.launches;
  return cudaGetLastError() == cudaSuccess;
}

template <typename T>
bool lu_steps(BatchSolve& b, T* F) {
  for (int j0 = 0; j0 < b.N[0]; j0 += 2 * kLuNB) {
    const int j1 = j0 + kLuNB, j2 = j1 + kLuNB;
    if (!panel_and_rows<T, false>(b, F, j0, j1) || !update<T>(b, F, j0, kLuNB, j1, j2)) return false;
    if (j1 >= b.N[0]) break;
    if (!panel_and_rows<T, true>(b, F, j1, j2) || !update<T>(b, F, j0, 2 * kLuNB, j2, INT_MAX)) return false;
  }
  return true;
}

// ---- one-CTA LU, for systems above the cluster's capacity -----------------------------------

constexpr int kBigNT = 512;
constexpr int kTM = 128, kTN = 64;  // trailing-update tile (kTM x kTN)

__device__ __forceinline__ void take_max(double& bv, int& bi, double v, int i) {
  if (v > bv || (v == bv && i < bi)) {
    bv = v;
    bi = i;
  }
}

// dynamic shared memory: the L21 (kLuNB x kTM) and U12 (kLuNB x kTN) tiles
template <typename T>
constexpr size_t big_smem() {
  return (size_t)kLuNB * (kTM + kTN) * sizeof(T);
}

template <typename T, int NT>
__device__ void cta_getrf(T* A, int64_t lda, int N, int* ipiv, int* info, T* s_a, T* s_b) {
  __shared__ double s_v[NT / 32];
  __shared__ int s_i[NT / 32];
  __shared__ int s_piv[kLuNB];
  __shared__ int s_rows[2 * kLuNB], s_src[2 * kLuNB], s_nrows;
  __shared__ T s_row[kLuNB];
  __shared__ T s_L[kLuNB][kLuNB + 1];
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  if (tid == 0) *info = 0;
  for (int j0 = 0; j0 < N; j0 += kLuNB) {
    const int jb = min(kLuNB, N - j0);
    // ---- panel: columns j0 .. j0+jb-1 ------------------------------------------------
    for (int j = j0; j < j0 + jb; ++j) {
      double bv = -1.0;
      int bi = INT_MAX;
      for (int i = j + tid; i < N; i += NT) take_max(bv, bi, pivot_size((double)A[i + (int64_t)j * lda]), i);
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, bv, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        take_max(bv, bi, ov, oi);
      }
      if (lane == 0) {
        s_v[wp] = bv;
        s_i[wp] = bi;
      }
      __syncthreads();
      if (tid == 0) {
        for (int w = 1; w < NT / 32; ++w) take_max(bv, bi, s_v[w], s_i[w]);
        s_piv[j - j0] = bi;
        ipiv[j] = bi;
        if (bv == 0.0 && *info == 0) *info = j + 1;
      }
      __syncthreads();
      const int p = s_piv[j - j0];
      if (p != j && tid < jb) {
        T* a = A + j + (int64_t)(j0 + tid) * lda;
        T* b = A + p + (int64_t)(j0 + tid) * lda;
        const T t = *a;
        *a = *b;
        *b = t;
      }
      __syncthreads();
      const T piv = A[j + (int64_t)j * lda];
      if (tid < jb) s_row[tid] = A[j + (int64_t)(j0 + tid) * lda];
      __syncthreads();
      if (piv != T(0)) {
        for (int i = j + 1 + tid; i < N; i += NT) {
          T* ri = A + i;
          const T l = ri[(int64_t)j * lda] / piv;
          ri[(int64_t)j * lda] = l;
          for (int c = j + 1 - j0; c < jb; ++c) ri[(int64_t)(j0 + c) * lda] -= l * s_row[c];
        }
      }
      __syncthreads();
    }
    // ---- the panel's interchanges on the other columns, as one gather per column ---
    if (tid == 0) {
      int nr = 0;
      for (int q = 0; q < jb; ++q) {  // rows touched: j0+q and their pivots
        const int cand[2] = {j0 + q, s_piv[q]};
        for (int u = 0; u < 2; ++u) {
          int f = -1;
          for (int m = 0; m < nr; ++m)
            if (s_rows[m] == cand[u]) f = m;
          if (f < 0) {
            s_rows[nr] = cand[u];
            s_src[nr] = cand[u];
            ++nr;
          }
        }
      }
      for (int q = 0; q < jb; ++q) {  // apply the swaps to the labels in order
        int a = -1, b = -1;
        for (int m = 0; m < nr; ++m) {
          if (s_rows[m] == j0 + q) a = m;
          if (s_rows[m] == s_piv[q]) b = m;
        }
        const int t = s_src[a];
        s_src[a] = s_src[b];
        s_src[b] = t;
      }
      s_nrows = nr;
    }
    __syncthreads();
    {
      const int nr = s_nrows;
      for (int c = wp; c < N; c += NT / 32) {
        if (c >= j0 && c < j0 + jb) continue;
        T* col = A + (int64_t)c * lda;
        T v0 = T(0), v1 = T(0);
        if (lane < nr) v0 = col[s_src[lane]];
        if (lane + 32 < nr) v1 = col[s_src[lane + 32]];
        __syncwarp();
        if (lane < nr) col[s_rows[lane]] = v0;
        if (lane + 32 < nr) col[s_rows[lane + 32]] = v1;
      }
    }
    __syncthreads();
    const int t0 = j0 + jb;
    if (t0 >= N) break;
    // ---- U12 = L11^{-1} A12 (unit lower), one column per thread -------------------
    for (int idx = tid; idx < jb * jb; idx += NT) {
      const int r = idx % jb, c = idx / jb;
      s_L[r][c] = A[j0 + r + (int64_t)(j0 + c) * lda];
    }
    __syncthreads();
    for (int c = t0 + tid; c < N; c += NT) {
      T* col = A + j0 + (int64_t)c * lda;
      T x[kLuNB];
#pragma unroll
      for (int q = 0; q < kLuNB; ++q) {
        if (q < jb) {
          T v = col[q];
#pragma unroll
          for (int t = 0; t < q; ++t) v -= s_L[q][t] * x[t];
          x[q] = v;
        }
      }
#pragma unroll
      for (int q = 0; q < kLuNB; ++q)
        if (q < jb) col[q] = x[q];
    }
    __syncthreads();
    // ---- A22 -= L21 U12, tiles of kTM x kTN: the tile of C is loaded with the operand
    //      tiles, so a tile costs one memory round trip before its FMAs ---------------
    const int m = N - t0;
    const int tm = (m + kTM - 1) / kTM, tn = (m + kTN - 1) / kTN;
    constexpr int CPT = kTM * kTN / NT;  // columns per thread
    const int r = tid % kTM, cg = tid / kTM;
    for (int tt = 0; tt < tm * tn; ++tt) {
      const int ti = tt % tm, tj = tt / tm;
      const int rb = t0 + ti * kTM, cb = t0 + tj * kTN;
      for (int idx = tid; idx < kLuNB * kTM; idx += NT) {
        const int rr = idx % kTM, k = idx / kTM;  // L21(rb + rr, j0 + k)
        s_a[k * kTM + rr] = (k < jb && rb + rr < N) ? A[rb + rr + (int64_t)(j0 + k) * lda] : T(0);
      }
      for (int idx = tid; idx < kLuNB * kTN; idx += NT) {
        const int kk = idx % kLuNB, cc = idx / kLuNB;  // U12(j0 + kk, cb + cc)
        s_b[kk * kTN + cc] = (kk < jb && cb + cc < N) ? A[j0 + kk + (int64_t)(cb + cc) * lda] : T(0);
      }
      T acc[CPT];
      const bool row_ok = rb + r < N;
#pragma unroll
      for (int q = 0; q < CPT; ++q) {
        const int cc = cb + cg * CPT + q;
        acc[q] = (row_ok && cc < N) ? A[rb + r + (int64_t)cc * lda] : T(0);
      }
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < kLuNB; ++k) {
        const T l = s_a[k * kTM + r];
#pragma unroll
        for (int q = 0; q < CPT; ++q) acc[q] = fma(-l, s_b[k * kTN + cg * CPT + q], acc[q]);
      }
      if (row_ok) {
#pragma unroll
        for (int q = 0; q < CPT; ++q) {
          const int cc = cb + cg * CPT + q;
          if (cc < N) A[rb + r + (int64_t)cc * lda] = acc[q];
        }
      }
      __syncthreads();
    }
  }
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT) batch_lu_kernel(const SysDev* __restrict__ sys, const int* __restrict__ order,
                                                      int nsys, T* F, int* piv, int* info, unsigned* counter) {
  extern __shared__ __align__(16) unsigned char lu_dyn[];
  T* s_a = reinterpret_cast<T*>(lu_dyn);
  T* s_b = s_a + kLuNB * kTM;
  __shared__ int s_item;
  for (;;) {
    if (threadIdx.x == 0) s_item = (int)atomicAdd(counter, 1u);
    __syncthreads();
    const int it = s_item;
    __syncthreads();
    if (it >= nsys) return;
    const int s = order[it];
    const SysDev S = sys[s];
    cta_getrf<T, NT>(F + S.f_off, S.lda, S.N, piv + S.piv_off, info + s, s_a, s_b);
    __syncthreads();
  }
}

// ---- substitution ---------------------------------------------------------------------------

// the row gather of P^T: perm[i] is the row that the interchanges bring to i
__global__ void __launch_bounds__(256) batch_perm_kernel(const SysDev* __restrict__ sys, const int* __restrict__ piv,
                                                         int* __restrict__ perm) {
  extern __shared__ int s_p[];  // N pivots, N labels
  const SysDev& S = sys[blockIdx.x];
  int* s_l = s_p + S.N;
  for (int i = threadIdx.x; i < S.N; i += blockDim.x) {
    s_p[i] = piv[S.piv_off + i];
    s_l[i] = i;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int j = 0; j < S.N; ++j) {
      const int p = checked_index(s_p[j], j, S.N, j);
      if (p != j) {
        const int t = s_l[j];
        s_l[j] = s_l[p];
        s_l[p] = t;
      }
    }
  __syncthreads();
  for (int i = threadIdx.x; i < S.N; i += blockDim.x) perm[S.piv_off + i] = s_l[i];
}

constexpr int kBlk = 128;

// dinv[2 b] = inverse of the unit lower triangle of diagonal block b, dinv[2 b + 1] of the upper
// one (diagonal included): with W the inverse of a unit upper triangle, L^{-1} = W^T for W =
// (L^T)^{-1}, and U = D N gives U^{-1} = W D^{-1} for W = N^{-1}.
template <typename T>
__global__ void __launch_bounds__(kTriThreads) batch_inv_kernel(const SysDev* __restrict__ sys,
                                                                const T* __restrict__ F, double* __restrict__ dinv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* U = reinterpret_cast<double*>(smem_raw);
  constexpr int P = kTriPitch<double>;
  __shared__ double dg[kBlk];
  const SysDev& S = sys[blockIdx.z];
  const int k0 = blockIdx.x * kBlk, m = min(kBlk, S.N - k0);
  if (m <= 0) return;
  const bool lower = blockIdx.y == 0;
  const int64_t lda = S.lda;
  const T* D = F + S.f_off + k0 + (int64_t)k0 * lda;
  const int tid = threadIdx.x;
  if (tid < kBlk) dg[tid] = tid < m ? (double)D[tid + (int64_t)tid * lda] : 1.0;
  __syncthreads();
  for (int base = tid; base < kBlk * kBlk; base += 16 * kTriThreads) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int i = (base + u * kTriThreads) % kBlk, j = (base + u * kTriThreads) / kBlk;  // entry (i, j) of D
      v[u] = (i < m && j < m && (lower ? j < i : i < j)) ? (double)D[i + (int64_t)j * lda] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int i = (base + u * kTriThreads) % kBlk, j = (base + u * kTriThreads) / kBlk;
      if (lower) U[j + i * P] = v[u];
      else U[i + j * P] = i < j ? v[u] / dg[i] : 0.0;
    }
  }
  unit_upper_inverse<double, kTriThreads>(U, U + 128 * P);
  double* V = dinv + (2 * (S.inv_off + blockIdx.x) + blockIdx.y) * (int64_t)(kBlk * kBlk);
  for (int idx = tid; idx < kBlk * kBlk; idx += kTriThreads) {
    const int i = idx % kBlk, j = idx / kBlk;
    double v = 0.0;
    if (i < m && j < m) {
      if (lower) v = j <= i ? U[j + i * P] : 0.0;
      else v = i <= j ? U[i + j * P] / dg[j] : 0.0;
    }
    V[idx] = v;
  }
}

__global__ void __launch_bounds__(256) batch_gather_kernel(const SysDev* __restrict__ sys, const int* __restrict__ perm,
                                                           const double* __restrict__ R, double* __restrict__ W,
                                                           const int* __restrict__ conv, const int* __restrict__ info) {
  const int s = blockIdx.y;
  if (conv[s] || info[s]) return;
  const SysDev& S = sys[s];
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= S.N) return;
  const int p = perm[S.piv_off + i];
  double* w = W + (S.piv_off + i) * kMaxRhs;
#pragma unroll
  for (int r = 0; r < kMaxRhs; ++r) w[r] = r < S.nrhs ? R[S.v_off + p + (int64_t)r * S.N] : 0.0;
}

constexpr int kStepNT = 256;  // two threads per row

// acc (8 load cases) of row tid % 128 over the half of 128 columns that tid / 128 names:
// M(row, c) y[c], 32 loads in flight
template <typename T>
__device__ __forceinline__ void tile_product(const T* M, int64_t ldm, int rows, int cols, const double (*y)[kMaxRhs],
                                             double* acc) {
  const int r = threadIdx.x % kBlk, c0 = (threadIdx.x / kBlk) * (kBlk / 2);
#pragma unroll
  for (int q = 0; q < kMaxRhs; ++q) acc[q] = 0.0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = c0 + 32 * h;
    T v[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) v[u] = (r < rows && c + u < cols) ? M[r + (int64_t)(c + u) * ldm] : T(0);
#pragma unroll
    for (int u = 0; u < 32; ++u) {
      const double m = (double)v[u];
#pragma unroll
      for (int q = 0; q < kMaxRhs; ++q) acc[q] = fma(m, y[c + u][q], acc[q]);
    }
  }
}

// Step `step` of the forward (UP = false) or backward substitution: block row i subtracts its
// tile times the block solved by the previous step, and the step's own block is solved; the
// backward steps add their blocks to X.
template <typename T, bool UP>
__global__ void __launch_bounds__(kStepNT, 2) batch_step_kernel(const SysDev* __restrict__ sys,
                                                                const int* __restrict__ order, const T* __restrict__ F,
                                                                const double* __restrict__ dinv, double* __restrict__ W,
                                                                double* __restrict__ X, int step,
                                                                const int* __restrict__ conv,
                                                                const int* __restrict__ info) {
  const int s = order[blockIdx.y];
  if (conv[s] || info[s]) return;
  const SysDev& S = sys[s];
  const int N = S.N, nblk = (N + kBlk - 1) / kBlk;
  const int k = UP ? nblk - 1 - step : step;         // the step's block
  const int i = UP ? k - (int)blockIdx.x : k + (int)blockIdx.x;  // this CTA's block row
  if (i < 0 || i >= nblk) return;
  __shared__ __align__(16) double s_y[kBlk][kMaxRhs];
  __shared__ __align__(16) double s_h[kBlk][kMaxRhs];  // the second half's sums
  const int tid = threadIdx.x, r = tid % kBlk;
  const int rows = min(kBlk, N - i * kBlk);
  double* Wi = W + (S.piv_off + i * kBlk) * kMaxRhs;
  double acc[kMaxRhs];
  // the rows' sums over the halves, in the first half's threads
  auto combine = [&]() {
    if (tid >= kBlk)
#pragma unroll
      for (int q = 0; q < kMaxRhs; ++q) s_h[r][q] = acc[q];
    __syncthreads();
    if (tid < kBlk)
#pragma unroll
      for (int q = 0; q < kMaxRhs; ++q) acc[q] += s_h[r][q];
  };
  if (step > 0) {
    const int kp = UP ? k + 1 : k - 1, cols = min(kBlk, N - kp * kBlk);
    const double* Wk = W + (S.piv_off + kp * kBlk) * kMaxRhs;
    for (int t = tid; t < kBlk * kMaxRhs; t += kStepNT) (&s_y[0][0])[t] = t < cols * kMaxRhs ? Wk[t] : 0.0;
    __syncthreads();
    tile_product(F + S.f_off + i * kBlk + (int64_t)kp * kBlk * S.lda, S.lda, rows, cols, s_y, acc);
    combine();
  } else {
#pragma unroll
    for (int q = 0; q < kMaxRhs; ++q) acc[q] = 0.0;
  }
  if (tid < kBlk)
#pragma unroll
    for (int q = 0; q < kMaxRhs; ++q) acc[q] = r < rows ? Wi[r * kMaxRhs + q] - acc[q] : 0.0;
  if (i == k) {
    __syncthreads();  // s_y and s_h have been read
    if (tid < kBlk)
#pragma unroll
      for (int q = 0; q < kMaxRhs; ++q) s_y[r][q] = acc[q];
    __syncthreads();
    tile_product(dinv + (2 * (S.inv_off + k) + (UP ? 1 : 0)) * (int64_t)(kBlk * kBlk), kBlk, rows, rows, s_y, acc);
    combine();
    if (UP && tid < rows)
#pragma unroll
      for (int q = 0; q < kMaxRhs; ++q)
        if (q < S.nrhs) X[S.v_off + k * kBlk + r + (int64_t)q * N] += acc[q];
  }
  if (tid < rows)
#pragma unroll
    for (int q = 0; q < kMaxRhs; ++q) Wi[r * kMaxRhs + q] = acc[q];
}

template <typename T>
bool substitute(BatchSolve& b, const T* F, const double* rhs) {
  const int maxN = b.N[0], nblk = (maxN + kBlk - 1) / kBlk;
  batch_gather_kernel<<<dim3((maxN + 255) / 256, b.nsys), 256, 0, b.stream>>>(b.sys, b.perm, rhs, b.W, b.conv, b.info);
  ++b.launches;
  for (int up = 0; up < 2; ++up)
    for (int k = 0; k < nblk; ++k) {
      const dim3 grid(nblk - k, active_from(b, k * kBlk + 1));
      if (up) batch_step_kernel<T, true><<<grid, kStepNT, 0, b.stream>>>(b.sys, b.order, F, b.dinv, b.W, b.X, k, b.conv, b.info);
      else batch_step_kernel<T, false><<<grid, kStepNT, 0, b.stream>>>(b.sys, b.order, F, b.dinv, b.W, b.X, k, b.conv, b.info);
      ++b.launches;
    }
  return cudaGetLastError() == cudaSuccess;
}

// ---- residual ---------------------------------------------------------------------------------

__device__ __forceinline__ void max_into(double* p, double v) {  // v >= 0: ordered as an integer
  atomicMax(reinterpret_cast<unsigned long long*>(p), (unsigned long long)__double_as_longlong(v));
}

// R = B - A X (FP64) of 128 rows and their maxima: |R|, |X|, |B| per load case, row sums of |A|
__global__ void __launch_bounds__(256) batch_residual_kernel(const SysDev* __restrict__ sys,
                                                             const double* __restrict__ A, const double* __restrict__ B,
                                                             const double* __restrict__ X, double* __restrict__ R,
                                                             double* __restrict__ red, const int* __restrict__ conv,
                                                             const int* __restrict__ info) {
  const int s = blockIdx.y;
  if (conv[s] || info[s]) return;
  const SysDev& S = sys[s];
  const int N = S.N, nrhs = S.nrhs, r0 = blockIdx.x * kBlk;
  if (r0 >= N) return;
  __shared__ __align__(16) double s_x[kBlk][kMaxRhs];
  __shared__ __align__(16) double s_h[kBlk][kMaxRhs + 1];
  const int tid = threadIdx.x, r = tid % kBlk, c0 = (tid / kBlk) * (kBlk / 2), lane = tid & 31;
  const int row = r0 + r;
  const double* As = A + S.a_off + row;
  double acc[kMaxRhs], asum = 0.0;
#pragma unroll
  for (int q = 0; q < kMaxRhs; ++q) acc[q] = 0.0;
  for (int b0 = 0; b0 < N; b0 += kBlk) {
    __syncthreads();
    for (int t = tid; t < kBlk * kMaxRhs; t += 256) {
      const int c = t % kBlk, q = t / kBlk;
      s_x[c][q] = (b0 + c < N && q < nrhs) ? X[S.v_off + b0 + c + (int64_t)q * N] : 0.0;
    }
    __syncthreads();
    for (int c = c0; c < c0 + kBlk / 2; c += 16) {
      double a[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) a[u] = (row < N && b0 + c + u < N) ? As[(int64_t)(b0 + c + u) * S.lda] : 0.0;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        asum += fabs(a[u]);
#pragma unroll
        for (int q = 0; q < kMaxRhs; ++q) acc[q] = fma(a[u], s_x[c + u][q], acc[q]);
      }
    }
  }
  __syncthreads();
  if (tid >= kBlk) {
#pragma unroll
    for (int q = 0; q < kMaxRhs; ++q) s_h[r][q] = acc[q];
    s_h[r][kMaxRhs] = asum;
  }
  __syncthreads();
  if (tid >= kBlk) return;
  asum = row < N ? asum + s_h[r][kMaxRhs] : 0.0;
  double* m = red + s * (3 * kMaxRhs + 1);
  for (int q = 0; q < nrhs; ++q) {
    double rv = 0.0, xv = 0.0, bv = 0.0;
    if (row < N) {
      const int64_t at = S.v_off + row + (int64_t)q * N;
      bv = B[at];
      xv = fabs(X[at]);
      rv = bv - (acc[q] + s_h[r][q]);
      R[at] = rv;
      rv = rv == rv ? fabs(rv) : CUDART_INF;  // fmax would pass over a NaN
      bv = fabs(bv);
    }
    for (int off = 16; off > 0; off >>= 1) {
      rv = fmax(rv, __shfl_xor_sync(0xffffffffu, rv, off));
      xv = fmax(xv, __shfl_xor_sync(0xffffffffu, xv, off));
      bv = fmax(bv, __shfl_xor_sync(0xffffffffu, bv, off));
    }
    if (lane == 0) {
      max_into(m + q, rv);
      max_into(m + kMaxRhs + q, xv);
      max_into(m + 2 * kMaxRhs + q, bv);
    }
  }
  for (int off = 16; off > 0; off >>= 1) asum = fmax(asum, __shfl_xor_sync(0xffffffffu, asum, off));
  if (lane == 0) max_into(m + 3 * kMaxRhs, asum);
}

// backward error max_r ||R_r|| / (||A|| ||X_r|| + ||B_r||) (infinity norms; infinite where a residual
// is NaN); conv = 1 once it is
// <= tol, 2 once a sweep gains less than 10 %; the maxima are cleared for the next pass
__global__ void batch_conv_kernel(const SysDev* __restrict__ sys, int nsys, double* __restrict__ red,
                                  double* __restrict__ berr, int* __restrict__ conv, const int* __restrict__ info,
                                  double tol, int first) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys || conv[s] || info[s]) return;
  double* m = red + s * (3 * kMaxRhs + 1);
  double be = 0.0;
  for (int q = 0; q < sys[s].nrhs; ++q) {
    const double den = m[3 * kMaxRhs] * m[kMaxRhs + q] + m[2 * kMaxRhs + q];
    be = fmax(be, m[q] == CUDART_INF ? CUDART_INF : den > 0.0 ? m[q] / den : 0.0);
  }
  for (int q = 0; q < 3 * kMaxRhs + 1; ++q) m[q] = 0.0;
  const double prev = berr[s];
  berr[s] = be;
  if (!first) {
    if (be <= tol) conv[s] = 1;
    else if (be > 0.9 * prev) conv[s] = 2;
  }
}

bool residual(BatchSolve& b, double tol, int first) {
  batch_residual_kernel<<<dim3((b.N[0] + kBlk - 1) / kBlk, b.nsys), 256, 0, b.stream>>>(b.sys, b.A, b.FI, b.X, b.R,
                                                                                       b.red, b.conv, b.info);
  batch_conv_kernel<<<(b.nsys + 127) / 128, 128, 0, b.stream>>>(b.sys, b.nsys, b.red, b.berr, b.conv, b.info, tol,
                                                                 first);
  b.launches += 2;
  return cudaGetLastError() == cudaSuccess;
}

// X = 0: the residual is the right-hand side, its backward error 1
__global__ void __launch_bounds__(256) batch_start_kernel(const SysDev* __restrict__ sys, const double* __restrict__ B,
                                                          double* __restrict__ X, double* __restrict__ R,
                                                          double* __restrict__ berr) {
  const SysDev& S = sys[blockIdx.y];
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i == 0) berr[blockIdx.y] = 1.0;
  if (i >= S.N) return;
  for (int q = 0; q < S.nrhs; ++q) {
    const int64_t at = S.v_off + i + (int64_t)q * S.N;
    X[at] = 0.0;
    R[at] = B[at];
  }
}

template <typename T>
__global__ void batch_copy_kernel(const SysDev* __restrict__ sys, const double* __restrict__ A, T* __restrict__ F) {
  const SysDev& S = sys[blockIdx.y];
  const int64_t total = (int64_t)S.N * S.lda;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x)
    F[S.f_off + k] = (T)A[S.a_off + k];
}

constexpr size_t perm_smem(int n) { return 2 * (size_t)n * sizeof(int); }

// Shared-memory limits, once per device at the most that any batch takes: they are the process's,
// and a batch that lowered one to its own need would fail another thread's launch.
template <typename T>
bool attributes() {
  static DeviceOnce set;
  if (!set.pending()) return true;
  if (cudaFuncSetAttribute(batch_inv_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(kTriElems<double> * sizeof(double))) != cudaSuccess ||
      cudaFuncSetAttribute(batch_update_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           2 * (int)sizeof(typename UpdateTile<T>::Half)) != cudaSuccess ||
      cudaFuncSetAttribute(batch_perm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)perm_smem(kMaxOrder)) != cudaSuccess)
    return false;
  set.mark();
  return true;
}

}  // namespace

template <typename T>
int batch_lu_max_order() {
  static DeviceOnce asked, yes;
  if (asked.pending()) {
    bool ok = cluster_fits(batch_panel_kernel<T, 1>, kPanelNT, sizeof(PanelSmem<T, 1, kPanelNT>)) &&
              cluster_fits(batch_panel_kernel<T, 2>, kPanelNT, sizeof(PanelSmem<T, 2, kPanelNT>));
    if constexpr (kMaxLpt<T> >= 4)
      ok = ok && cluster_fits(batch_panel_kernel<T, 4>, kPanelNT, sizeof(PanelSmem<T, 4, kPanelNT>));
    if (ok) yes.mark();
    asked.mark();
  }
  return yes.pending() ? 0 : kMaxCluster * kPanelNT * kMaxLpt<T>;
}

template <typename T>
bool batch_solve_enqueue(BatchSolve& b, T* F, double tol, int sweeps) {
  const int maxN = b.N[0], nblk = (maxN + kBlk - 1) / kBlk;
  if (!attributes<T>()) return false;
  if (cudaMemsetAsync(b.info, 0, b.nsys * sizeof(int), b.stream) != cudaSuccess ||
      cudaMemsetAsync(b.conv, 0, b.nsys * sizeof(int), b.stream) != cudaSuccess ||
      cudaMemsetAsync(b.red, 0, (size_t)b.nsys * (3 * kMaxRhs + 1) * sizeof(double), b.stream) != cudaSuccess ||
      cudaMemsetAsync(b.err, 0, 2 * sizeof(int), b.stream) != cudaSuccess)
    return false;
  batch_copy_kernel<T><<<dim3(64, b.nsys), 256, 0, b.stream>>>(b.sys, b.A, F);
  ++b.launches;
  if (maxN <= batch_lu_max_order<T>()) {
    if (!lu_steps<T>(b, F)) return false;
  } else {
    if (cudaFuncSetAttribute(batch_lu_kernel<T, kBigNT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)big_smem<T>()) != cudaSuccess)
      return false;
    batch_lu_kernel<T, kBigNT><<<std::min(b.nsys, b.sm_count), kBigNT, big_smem<T>(), b.stream>>>(
        b.sys, b.order, b.nsys, F, b.piv, b.info, reinterpret_cast<unsigned*>(b.err + 1));
    ++b.launches;
  }
  batch_perm_kernel<<<b.nsys, 256, perm_smem(maxN), b.stream>>>(b.sys, b.piv, b.perm);
  batch_inv_kernel<T><<<dim3(nblk, 2, b.nsys), kTriThreads, kTriElems<double> * sizeof(double), b.stream>>>(b.sys, F, b.dinv);
  batch_start_kernel<<<dim3((maxN + 255) / 256, b.nsys), 256, 0, b.stream>>>(b.sys, b.FI, b.X, b.R, b.berr);
  b.launches += 3;
  if (cudaGetLastError() != cudaSuccess) return false;
  if (sweeps == 0) return substitute<T>(b, F, b.FI) && residual(b, tol, 1);
  for (int it = 0; it < sweeps; ++it)
    if (!substitute<T>(b, F, b.R) || !residual(b, tol, 0)) return false;
  return true;
}

template bool batch_solve_enqueue<float>(BatchSolve&, float*, double, int);
template bool batch_solve_enqueue<double>(BatchSolve&, double*, double, int);
template int batch_lu_max_order<float>();
template int batch_lu_max_order<double>();

}  // namespace bem
