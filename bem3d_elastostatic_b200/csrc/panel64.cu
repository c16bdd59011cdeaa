// FP64 partial-pivot sub-panel on one thread-block cluster (see lu.cuh for the layout).
//
// The sub-panel is w <= 32 columns of T = S^T: line c (a column of S, a row of T) holds its
// w values S(r0 .. r0 + w, c), c in [r0, n).  A pivot step is a search over the lines and
// one rank-1 update; its cost is the exchange of the pivot line, so the lines live in the
// registers of one cluster of up to 16 CTAs (8,192 lines at one per thread, 12,288 at two)
// and the exchange stays in distributed shared memory:
//   * a line never moves: a thread keeps its line's current position instead of swapping
//     contents, ties go to the smallest position (dgetrf's row order);
//   * a line's values are shifted by one register every step, so that the current column is
//     always v[0] and every index is static although the step loop is not unrolled; the
//     multipliers, and a pivoted line's rest of its U row, go to shared memory;
//   * every warp finds its candidate by three integer warp reductions (the high and low
//     words of |v| and the position), and warp d of a CTA sends the CTA's candidate line to
//     CTA d with st.async, which completes on that CTA's mbarrier: one one-way trip per
//     pivot, no cluster barrier.  Two slots by step parity suffice: a CTA sends step t + 1
//     only after its threads have read step t - 1's line.
// Measured per 32-column sub-panel: 36 us at 2,598 lines (8 CTAs), 58 us at 11,526 (16 CTAs,
// two lines per thread), where the grid-synchronised panel_kernel takes 109 and 125 us
// (seven CTA barriers and a grid barrier through L2 per pivot).  One CTA alone (up to 256
// lines) takes 27 us.  More CTAs than the lines need do not help: the step is the chain of
// latencies above, about 1 us, not the update.
// Waits are bounded by the context's limit; on a timeout the CTA records BEM_ERR_TIMEOUT,
// ends its steps and meets the others at the final cluster barrier.
#include <climits>

#include "lu.cuh"

namespace bem {
namespace {

constexpr int kMaxCluster = 16;

struct alignas(16) Key {
  unsigned hi, lo;
  int pos, pad;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void st_async_f64(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void st_async_key(unsigned addr, const Key& k, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   addr),
               "r"(k.hi), "r"(k.lo), "r"((unsigned)k.pos), "r"(0u), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned phase) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(phase)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ unsigned long long timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A lane that holds the largest key of the warp, the smallest position first among equals.
// The high words nearly always decide.
__device__ __forceinline__ int warp_pick(unsigned hi, unsigned lo, int pos) {
  unsigned at = __ballot_sync(0xffffffffu, hi == __reduce_max_sync(0xffffffffu, hi));
  if ((at & (at - 1)) != 0) {
    const bool top = (at >> (threadIdx.x & 31)) & 1u;
    const unsigned l = __reduce_max_sync(0xffffffffu, top ? lo : 0u);
    const bool eq = top && lo == l;
    const unsigned p = __reduce_min_sync(0xffffffffu, eq ? (unsigned)pos : (unsigned)INT_MAX);
    at = __ballot_sync(0xffffffffu, eq && (unsigned)pos == p);
  }
  return __ffs(at) - 1;
}

// 1 / x for normal x: the hardware's approximation y of the leading bits and one third-order
// step, y (1 + e + e^2) with e = 1 - x y (Newton's iteration with one more term).
__device__ __forceinline__ double reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// kept out of line: as a select it would be computed for every multiplier
__device__ __noinline__ double plain_quotient(double v, double pv) { return pv != 0.0 ? v / pv : v; }

template <int LPT, int NT>
struct PanelSmem {
  static constexpr int kLines = LPT * NT;
  static constexpr int kPitchL = kLines + 1;  // odd: the transposed accesses meet every bank
  double val[kPanelW * kPitchL];              // [column of T][line]
  double cand[2][NT / 32][kPanelW];           // the warps' candidate lines
  double slot[2][kMaxCluster][kPanelW];       // the CTAs' candidate lines, sent by them
  Key cand_key[2][NT / 32];
  Key slot_key[2][kMaxCluster];
  int abort[2];                               // by step parity: set in the wait of the step before
  int pos[kLines];
  unsigned long long bar[2];
};

struct PanelArgs {
  double* S;
  int64_t lda;
  int n, r0, w;
  int* piv;
  int* status;
  unsigned long long wait_ns;
};

// Steps [t0, t0 + 8) with LEN = 32 - t0 values left per line: the update shrinks with the
// panel in four lengths.  A step is a chain of latencies: the warp's search, the CTA's, the
// send, the search over the CTAs, the multiplier and the update, whose pivot line every
// warp reads from shared memory.
//
// A warp whose lines are all pivoted (or beyond the matrix) keeps only the barriers and the
// sends.  Returns false, in all threads of the CTA, once a wait has run out.
constexpr unsigned kMsgBytes = kPanelW * 8 + 16;  // line, key
template <int LPT, int NT, int LEN>
__device__ __forceinline__ bool panel_steps(const PanelArgs& P, PanelSmem<LPT, NT>& sm, int C, int rank,
                                            double (&v)[LPT][kPanelW], int (&pos)[LPT], bool (&done)[LPT]) {
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int t0 = kPanelW - LEN;
  constexpr int kDest = (kMaxCluster + NW - 1) / NW;  // CTAs a warp sends to
  const unsigned own = smem_u32(&sm);
  unsigned remote[kDest];
#pragma unroll
  for (int i = 0; i < kDest; ++i) remote[i] = wp + i * NW < C ? mapa(own, wp + i * NW) : 0u;
#pragma unroll 1
  for (int t = t0; t < t0 + 8 && t < P.w; ++t) {
    const int k = P.r0 + t, par = t & 1;
    // the warp's candidate
    bool mine = false;
#pragma unroll
    for (int q = 0; q < LPT; ++q) mine |= !done[q];
    const bool live = __any_sync(0xffffffffu, mine);
    if (live) {
      unsigned hi = 0, lo = 0;
      int cp = INT_MAX;
#pragma unroll
      for (int q = 0; q < LPT; ++q) {
        const double a = fabs(v[q][0]);
        const unsigned long long b = a == a ? (unsigned long long)__double_as_longlong(a) : 0ull;  // NaN as zero
        const unsigned ah = (unsigned)(b >> 32), al = (unsigned)b;
        const bool better =
            !done[q] && (cp == INT_MAX || ah > hi || (ah == hi && (al > lo || (al == lo && pos[q] < cp))));
        if (better) {
          hi = ah;
          lo = al;
          cp = pos[q];
        }
      }
      if (lane == warp_pick(hi, lo, cp)) {
        sm.cand_key[par][wp] = Key{hi, lo, cp, 0};
#pragma unroll
        for (int q = 0; q < LPT; ++q)
          if (LPT == 1 || (!done[q] && pos[q] == cp))
#pragma unroll
            for (int j = 0; j < LEN; j += 2)
              *reinterpret_cast<double2*>(&sm.cand[par][wp][j]) = make_double2(v[q][j], v[q][j + 1]);
      }
    } else if (lane == 0) {
      sm.cand_key[par][wp] = Key{0u, 0u, INT_MAX, 0};
    }
    __syncthreads();
    if (*(volatile int*)&sm.abort[par]) return false;
    // the CTA's candidate
    Key kk{0u, 0u, INT_MAX, 0};
    if (lane < NW) kk = sm.cand_key[par][lane];
    int wl = min(warp_pick(kk.hi, kk.lo, kk.pos), NW - 1);
    const double* line = sm.cand[par][wl];
    int p;
    if (C > 1) {
      const double x = line[lane];
      const Key best = sm.cand_key[par][wl];
#pragma unroll
      for (int i = 0; i < kDest; ++i)
        if (wp + i * NW < C) {
          const unsigned rb = remote[i] + (smem_u32(&sm.bar[par]) - own);
          st_async_f64(remote[i] + (smem_u32(&sm.slot[par][rank][lane]) - own), x, rb);
          if (lane == 0) st_async_key(remote[i] + (smem_u32(&sm.slot_key[par][rank]) - own), best, rb);
        }
      const unsigned ph = (t >> 1) & 1;
      if (!mbar_try(smem_u32(&sm.bar[par]), ph)) {
        const unsigned long long s = timer_ns();
        unsigned spins = 0;
        while (!mbar_try(smem_u32(&sm.bar[par]), ph))
          if ((++spins & 63u) == 0 && timer_ns() - s > P.wait_ns) {
            *(volatile int*)&sm.abort[par ^ 1] = 1;  // seen after the next step's barrier
            break;
          }
      }
      Key sk{0u, 0u, INT_MAX, 0};
      if (lane < C) sk = sm.slot_key[par][lane];
      wl = min(warp_pick(sk.hi, sk.lo, sk.pos), kMaxCluster - 1);
      line = sm.slot[par][wl];
      p = sm.slot_key[par][wl].pos;
    } else {
      p = sm.cand_key[par][wl].pos;
    }
    const double pv = line[0];
    if (live) {
      // v / pv: the product with the reciprocal and one correction by its remainder; far from
      // the ends of the exponent range only
      const bool nz = pv != 0.0;
      const bool plain = fabs(pv) < 1e290 && fabs(pv) > 1e-290;
      const double rc = reciprocal(pv);
      unsigned own_pivot[LPT];
      double m[LPT];
#pragma unroll
      for (int q = 0; q < LPT; ++q) {
        double l = v[q][0] * rc;
        l = fma(fma(-l, pv, v[q][0]), rc, l);
        if (!plain) l = plain_quotient(v[q][0], pv);
        const bool here = !done[q] && pos[q] == p;  // the pivot line: position k from now on
        own_pivot[q] = __ballot_sync(0xffffffffu, here);
        if (!done[q] && pos[q] == k) pos[q] = p;
        if (here) pos[q] = k;
        done[q] |= here;
        if (!done[q]) sm.val[t * PanelSmem<LPT, NT>::kPitchL + tid + q * NT] = l;
        m[q] = nz ? l : 0.0;
      }
#pragma unroll
      for (int j = 0; j < LEN - 1; ++j) {
        const double u = line[j + 1];
#pragma unroll
        for (int q = 0; q < LPT; ++q) v[q][j] = fma(-m[q], u, v[q][j + 1]);
      }
#pragma unroll
      for (int q = 0; q < LPT; ++q)  // its values are row k of U, written by its warp's lanes
        if (own_pivot[q] && t + lane < kPanelW)
          sm.val[(t + lane) * PanelSmem<LPT, NT>::kPitchL + wp * 32 + q * NT + __ffs(own_pivot[q]) - 1] = line[lane];
    }
    if (tid == 0) {
      if (C > 1 && t + 2 < P.w && mbar_try(smem_u32(&sm.bar[par]), (t >> 1) & 1))
        mbar_expect(smem_u32(&sm.bar[par]), (unsigned)C * kMsgBytes);  // for step t + 2
      if (rank == 0 && p < P.n) {
        P.piv[k] = p;
        if (pv == 0.0 && P.status[1] == 0) P.status[1] = k + 1;
      }
    }
  }
  return true;
}

template <int LPT, int NT>
__global__ void __launch_bounds__(NT, 1) panel_cluster_kernel(PanelArgs P, int C) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Sm = PanelSmem<LPT, NT>;
  Sm& sm = *reinterpret_cast<Sm*>(smem_raw);
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int rank = C > 1 ? (int)blockIdx.x : 0;  // the grid is one cluster
  const int base = P.r0 + rank * Sm::kLines;     // line i of this CTA is column base + i of S
  const int nl = max(0, min(Sm::kLines, P.n - base));
  for (int c = wp; c < nl; c += NW)  // a line's values: one coalesced 256 B read per warp
    sm.val[lane * Sm::kPitchL + c] = lane < P.w ? P.S[(int64_t)(base + c) * P.lda + P.r0 + lane] : 0.0;
  for (int i = tid; i < 2 * NW * kPanelW; i += NT) (&sm.cand[0][0][0])[i] = 0.0;
  if (tid == 0) {
    mbar_init(smem_u32(&sm.bar[0]), 1);
    mbar_init(smem_u32(&sm.bar[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect(smem_u32(&sm.bar[0]), (unsigned)C * kMsgBytes);
    mbar_expect(smem_u32(&sm.bar[1]), (unsigned)C * kMsgBytes);
    sm.abort[0] = sm.abort[1] = 0;
  }
  __syncthreads();
  if (C > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  double v[LPT][kPanelW];
  int pos[LPT];
  bool done[LPT];
#pragma unroll
  for (int q = 0; q < LPT; ++q) {
    const int c = tid + q * NT;
    done[q] = c >= nl;
    pos[q] = c < nl ? base + c : INT_MAX;
#pragma unroll
    for (int j = 0; j < kPanelW; ++j) v[q][j] = c < nl ? sm.val[j * Sm::kPitchL + c] : 0.0;
  }
  // a thread reads and writes only its own lines of sm.val until the last barrier
  bool ok = panel_steps<LPT, NT, 32>(P, sm, C, rank, v, pos, done);
  if (ok && P.w > 8) ok = panel_steps<LPT, NT, 24>(P, sm, C, rank, v, pos, done);
  if (ok && P.w > 16) ok = panel_steps<LPT, NT, 16>(P, sm, C, rank, v, pos, done);
  if (ok && P.w > 24) ok = panel_steps<LPT, NT, 8>(P, sm, C, rank, v, pos, done);
#pragma unroll
  for (int q = 0; q < LPT; ++q) sm.pos[tid + q * NT] = pos[q];
  __syncthreads();
  const bool failed = !ok || *(volatile int*)&sm.abort[0] || *(volatile int*)&sm.abort[1];
  if (C > 1) {  // no CTA leaves while another may still send to it
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (failed) {
    if (tid == 0) atomicCAS(P.status, 0, BEM_ERR_TIMEOUT);
    return;
  }
  for (int c = wp; c < nl; c += NW)
    if (lane < P.w) P.S[(int64_t)sm.pos[c] * P.lda + P.r0 + lane] = sm.val[lane * Sm::kPitchL + c];
}

template <int LPT, int NT>
int launch(bem_ctx* c, const PanelArgs& P, int C) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = sizeof(PanelSmem<LPT, NT>);
  cfg.stream = c->stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = C;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  BEM_CUDA(c, cudaLaunchKernelEx(&cfg, panel_cluster_kernel<LPT, NT>, P, C));
  ++c->launches;
  return BEM_OK;
}

// whether a cluster of 16 such CTAs fits the device (attributes set on the way)
template <int LPT, int NT>
bool resident() {
  if (cudaFuncSetAttribute(panel_cluster_kernel<LPT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(PanelSmem<LPT, NT>)) != cudaSuccess ||
      cudaFuncSetAttribute(panel_cluster_kernel<LPT, NT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
          cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kMaxCluster);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = sizeof(PanelSmem<LPT, NT>);
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kMaxCluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int num = 0;
  if (cudaOccupancyMaxActiveClusters(&num, panel_cluster_kernel<LPT, NT>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return num >= 1;
}

}  // namespace

// Lines the cluster kernel takes on this device (0: not at all); asked once per device.
int panel_cluster_lines() {
  static DeviceOnce asked, fits;
  if (asked.pending()) {
    if (resident<1, 256>() && resident<1, 512>() && resident<2, 384>()) fits.mark();
    asked.mark();
  }
  return fits.pending() ? 0 : kMaxCluster * 768;
}

// The sub-panel rows [r0, r0 + w) of S, pivoting over the columns [r0, n): n - r0 at most
// panel_cluster_lines().
int panel_cluster_launch(bem_ctx* c, double* S, int64_t lda, int n, int r0, int w, int* piv, int* status) {
  const PanelArgs P{S, lda, n, r0, w, piv, status, c->wait_ns};
  const int lines = n - r0;
  if (lines > kMaxCluster * 512) return launch<2, 384>(c, P, kMaxCluster);
  if (lines > kMaxCluster * 256) return launch<1, 512>(c, P, kMaxCluster);
  int C = 1;
  while (C * 256 < lines) C *= 2;
  return launch<1, 256>(c, P, C);
}

}  // namespace bem
