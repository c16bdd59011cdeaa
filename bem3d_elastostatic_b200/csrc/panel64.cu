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
  for (int c = wp; c < nl; c += NW)
    if (lane < w) P.S[(int64_t)sm.pos[c] * P.lda + r0 + lane] = sm.val[lane * Sm::kPitchL + c];
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
// panel_cluster_lines().
int panel_cluster_launch(bem_ctx* c, double* S, int64_t lda, int n, int r0, int w, int* piv, int* status) {
  const PanelArgs P{{n, r0, w, piv, status + 1, c->wait_ns}, S, lda, status};
  const int lines = n - r0;
  if (lines > kMaxCluster * 512) return launch<2, 384>(c, P, kMaxCluster);
  if (lines > kMaxCluster * 256) return launch<1, 512>(c, P, kMaxCluster);
  int C = 1;
  while (C * 256 < lines) C *= 2;
  return launch<1, 256>(c, P, C);
}

}  // namespace bem
