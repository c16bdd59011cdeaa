// FP64 partial-pivot sub-panel of the dense LU on one cluster (panel_cluster.cuh): w <= 32
// columns of T = S^T, so that a line is a column of S and its values the contiguous S(r0 .. r0
// + w, c), c in [r0, n).  Up to 8,192 lines at one per thread, 12,288 at two.
//
// Measured per 32-column sub-panel: 36 us at 2,598 lines (8 CTAs), 58 us at 11,526 (16 CTAs,
// two lines per thread), where the grid-synchronised panel_kernel takes 109 and 125 us
// (seven CTA barriers and a grid barrier through L2 per pivot).  One CTA alone (up to 256
// lines) takes 27 us.  More CTAs than the lines need do not help: the step is the chain of
// latencies above, about 1 us, not the update.
#include "panel_cluster.cuh"

namespace bem {
namespace {

struct PanelArgs {
  PanelStep st;
  double* S;
  int64_t lda;
  int* status;  // [0] error code, [1] info
  int* moved;   // [q]: the line that ends at position r0 + q; [32 + q]: where line r0 + q ends
};

template <int LPT, int NT>
__global__ void __launch_bounds__(NT, 1) panel_cluster_kernel(PanelArgs P, int C) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Sm = PanelSmem<double, LPT, NT>;
  Sm& sm = *reinterpret_cast<Sm*>(smem_raw);
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int r0 = P.st.r0, w = P.st.w;
  const int rank = C > 1 ? (int)blockIdx.x : 0;  // the grid is one cluster
  const int base = r0 + rank * Sm::kLines;       // line i of this CTA is column base + i of S
  const int nl = max(0, min(Sm::kLines, P.st.n - base));
  for (int c = wp; c < nl; c += NW)  // a line's values: one coalesced 256 B read per warp
    sm.val[lane * Sm::kPitchL + c] = lane < w ? P.S[(int64_t)(base + c) * P.lda + r0 + lane] : 0.0;
  __syncthreads();
  const bool ok = panel_on_cluster<double, LPT, NT>(P.st, sm, C, rank, base, nl, [&](double(&v)[LPT][kPanelW]) {
#pragma unroll
    for (int q = 0; q < LPT; ++q)
#pragma unroll
      for (int j = 0; j < kPanelW; ++j) v[q][j] = tid + q * NT < nl ? sm.val[j * Sm::kPitchL + tid + q * NT] : 0.0;
  });
  if (!ok) {
    if (tid == 0) atomicCAS(P.status, 0, BEM_ERR_TIMEOUT);
    return;
  }
  for (int c = tid; c < nl; c += NT) {
    const int p = sm.pos[c], line = base + c;
    if (p < r0 + w) P.moved[p - r0] = line;
    if (line < r0 + w) P.moved[kPanelW + line - r0] = p;
  }
  for (int c = wp; c < nl; c += NW)
    if (lane < w) P.S[(int64_t)sm.pos[c] * P.lda + r0 + lane] = sm.val[lane * Sm::kPitchL + c];
}

// One row of S per thread, outside the sub-panel: its interchanges (a column of the sub-panel
// that leaves it ends where a pivot came from), all loads before the first store, and for the
// panel's rows below, [r0 + w, q1), the solve with the unit upper triangle of S(r0.., r0..).
// (The interchanges one after the other, each a dependent exchange, and a launch of its own for
// the solve took 9.5 us where this takes 6.)
__global__ void __launch_bounds__(128) panel_rows_kernel(double* S, int64_t lda, int n, int r0, int w, int q1,
                                                         const int* __restrict__ moved) {
  constexpr int W = kPanelW;
  __shared__ int s_src[W], s_dst[W];
  __shared__ __align__(16) double s_U[W][W + 2];  // [column][row], read as 16-byte broadcasts
  const int tid = threadIdx.x, b1 = r0 + w;
  bool any = false;
  if (tid < W) {
    s_src[tid] = tid < w ? checked_index(moved[tid], r0, n, r0 + tid) : r0 + tid;
    s_dst[tid] = tid < w ? checked_index(moved[W + tid], r0, n, r0 + tid) : r0 + tid;
    any = s_src[tid] != r0 + tid;
  }
  for (int i = tid; i < W * W; i += 128) {
    const int a = i % W, b = i / W;
    s_U[b][a] = (b < w && a < b) ? S[r0 + a + (int64_t)(r0 + b) * lda] : 0.0;
  }
  any = __syncthreads_or(any);
  const int i = blockIdx.x * 128 + tid, r = i < r0 ? i : i + w;
  const bool solve = r >= b1 && r < q1;
  if (r >= n || (!any && !solve)) return;
  double x[W];
#pragma unroll
  for (int q = 0; q < W; ++q) x[q] = q < w ? S[r + (int64_t)(r0 + q) * lda] : 0.0;
  if (any) {
    double y[W];
#pragma unroll
    for (int q = 0; q < W; ++q) y[q] = q < w ? S[r + (int64_t)s_src[q] * lda] : 0.0;
#pragma unroll
    for (int q = 0; q < W; ++q)
      if (q < w && s_dst[q] >= b1) S[r + (int64_t)s_dst[q] * lda] = x[q];
#pragma unroll
    for (int q = 0; q < W; ++q) x[q] = y[q];
  }
  if (solve) {
#pragma unroll
    for (int b = 1; b < W; ++b) {
      double v = x[b];
#pragma unroll
      for (int a = 0; a < b; a += 2) {
        const double2 u = *reinterpret_cast<const double2*>(&s_U[b][a]);
        v = fma(-x[a], u.x, v);
        if (a + 1 < b) v = fma(-x[a + 1], u.y, v);
      }
      x[b] = v;
    }
  }
#pragma unroll
  for (int q = 0; q < W; ++q)
    if (q < w) S[r + (int64_t)(r0 + q) * lda] = x[q];
}

template <int LPT, int NT>
int launch(bem_ctx* c, const PanelArgs& P, int C) {
  BEM_CUDA(c, launch_clusters(panel_cluster_kernel<LPT, NT>, 1, C, NT, sizeof(PanelSmem<double, LPT, NT>), c->stream,
                              P, C));
  ++c->launches;
  return BEM_OK;
}

template <int LPT, int NT>
bool fits() {
  return cluster_fits(panel_cluster_kernel<LPT, NT>, NT, sizeof(PanelSmem<double, LPT, NT>));
}

}  // namespace

// Lines the cluster kernel takes on this device (0: not at all); asked once per device.
int panel_cluster_lines() {
  static DeviceOnce asked, yes;
  if (asked.pending()) {
    if (fits<1, 256>() && fits<1, 512>() && fits<2, 384>()) yes.mark();
    asked.mark();
  }
  return yes.pending() ? 0 : kMaxCluster * 768;
}

// The sub-panel rows [r0, r0 + w) of S, pivoting over the columns [r0, n): n - r0 at most
// panel_cluster_lines().  moved (64 ints) receives its interchanges as panel_rows takes them.
int panel_cluster_launch(bem_ctx* c, double* S, int64_t lda, int n, int r0, int w, int* piv, int* status,
                         int* moved) {
  const PanelArgs P{{n, r0, w, piv, status + 1, c->wait_ns, c->withhold_pivot}, S, lda, status, moved};
  const int lines = n - r0;
  if (lines > kMaxCluster * 512) return launch<2, 384>(c, P, kMaxCluster);
  if (lines > kMaxCluster * 256) return launch<1, 512>(c, P, kMaxCluster);
  int C = 1;
  while (C * 256 < lines) C *= 2;
  return launch<1, 256>(c, P, C);
}

// The sub-panel's interchanges on every other row of S and the solve of the rows [r0 + w, q1).
int panel_rows_launch(bem_ctx* c, double* S, int64_t lda, int n, int r0, int w, int q1, const int* moved) {
  if (n == w) return BEM_OK;
  panel_rows_kernel<<<(n - w + 127) / 128, 128, 0, c->stream>>>(S, lda, n, r0, w, q1, moved);
  BEM_LAUNCH_CHECK(c);
  return BEM_OK;
}

}  // namespace bem
