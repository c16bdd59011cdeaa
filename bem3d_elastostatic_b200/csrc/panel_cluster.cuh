// Partial-pivot sub-panel on one thread-block cluster.
//
// A sub-panel is w <= 32 columns; a line is one of its rows, identified by its position in
// [r0, n).  A pivot step is a search over the lines and one rank-1 update; its cost is the
// exchange of the pivot line, so the lines live in the registers of one cluster of up to 16
// CTAs (LPT per thread) and the exchange stays in distributed shared memory:
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
// Waits are bounded by the caller's limit; on a timeout the CTA records it, ends its steps before
// it sends again and meets the others at the final cluster barrier: no message is younger than the
// limit then.  The launches that follow run all the same, so the readers of a panel's pivots and
// interchanges take them through checked_index (lu.cuh).
#pragma once

#include <cuda_runtime.h>
#include <climits>

#include "common.cuh"
#include "lu.cuh"
#include "recip.cuh"

namespace bem {

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

__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, float v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
               "r"(__float_as_uint(v)), "r"(bar)
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

// |v| as an ordered integer, NaN as zero
__device__ __forceinline__ void magnitude(double v, unsigned& hi, unsigned& lo) {
  const double a = fabs(v);
  const unsigned long long b = a == a ? (unsigned long long)__double_as_longlong(a) : 0ull;
  hi = (unsigned)(b >> 32);
  lo = (unsigned)b;
}
__device__ __forceinline__ void magnitude(float v, unsigned& hi, unsigned& lo) {
  const float a = fabsf(v);
  hi = a == a ? __float_as_uint(a) : 0u;
  lo = 0u;
}

// far from the ends of the exponent range
__device__ __forceinline__ bool mid_range(double a) { return fabs(a) < 1e290 && fabs(a) > 1e-290; }
__device__ __forceinline__ bool mid_range(float a) { return fabsf(a) < 1e30f && fabsf(a) > 1e-30f; }

// kept out of line: as a select it would be computed for every multiplier
template <typename T>
__device__ __noinline__ T plain_quotient(T v, T pv) {
  return pv != T(0) ? v / pv : v;
}

template <typename T, int LPT, int NT>
struct PanelSmem {
  static constexpr int kLines = LPT * NT;
  static constexpr int kPitchL = kLines + 1;  // odd: the transposed accesses meet every bank
  alignas(16) T val[kPanelW * kPitchL];       // [column][line]
  alignas(16) T cand[2][NT / 32][kPanelW];    // the warps' candidate lines
  alignas(16) T slot[2][kMaxCluster][kPanelW];       // the CTAs' candidate lines, sent by them
  Key cand_key[2][NT / 32];
  Key slot_key[2][kMaxCluster];
  int abort[2];                               // by step parity: set in the wait of the step before
  int pos[kLines];
  unsigned long long bar[2];
};

// The steps' view of a sub-panel: positions [r0, n), w columns; piv[k] and *info (the 1-based
// step of the first exactly zero pivot, if still 0) are written by the cluster's first CTA.
struct PanelStep {
  int n, r0, w;
  int* piv;
  int* info;
  unsigned long long wait_ns;
  int withhold;  // failure injection: the step whose line the first CTA does not send (-1: none)
};

// Steps [t0, t0 + 8) with LEN = 32 - t0 values left per line: the update shrinks with the
// panel in four lengths.  A step is a chain of latencies: the warp's search, the CTA's, the
// send, the search over the CTAs, the multiplier and the update, whose pivot line every
// warp reads from shared memory.
//
// A warp whose lines are all pivoted (or beyond the matrix) keeps only the barriers and the
// sends.  Returns false, in all threads of the CTA, once a wait has run out.
template <typename T>
constexpr unsigned kMsgBytes = kPanelW * sizeof(T) + 16;  // line, key
template <typename T, int LPT, int NT, int LEN>
__device__ __forceinline__ bool panel_steps(const PanelStep& P, PanelSmem<T, LPT, NT>& sm, int C, int rank,
                                            T (&v)[LPT][kPanelW], int (&pos)[LPT], bool (&done)[LPT]) {
  constexpr int NW = NT / 32, kVec = 16 / sizeof(T), kPitchL = PanelSmem<T, LPT, NT>::kPitchL;
  struct alignas(16) Vec {
    T v[kVec];
  };
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int t0 = kPanelW - LEN;
  constexpr int kDest = (kMaxCluster + NW - 1) / NW;  // CTAs a warp sends to
  const unsigned own = smem_u32(&sm);
  const int hold = rank == 0 ? P.withhold : -1;
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
        unsigned ah, al;
        magnitude(v[q][0], ah, al);
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
            for (int j = 0; j < LEN; j += kVec) {
              Vec x;
#pragma unroll
              for (int u = 0; u < kVec; ++u) x.v[u] = v[q][j + u];
              *reinterpret_cast<Vec*>(&sm.cand[par][wp][j]) = x;
            }
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
    const T* line = sm.cand[par][wl];
    int p;
    if (C > 1) {
      const T x = line[lane];
      const Key best = sm.cand_key[par][wl];
#pragma unroll
      for (int i = 0; i < kDest; ++i)
        if (wp + i * NW < C && k != hold) {
          const unsigned rb = remote[i] + (smem_u32(&sm.bar[par]) - own);
          st_async(remote[i] + (smem_u32(&sm.slot[par][rank][lane]) - own), x, rb);
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
    const T pv = line[0];
    if (live) {
      // v / pv from the reciprocal far from the ends of the exponent range only
      const bool nz = pv != T(0);
      const bool plain = mid_range(pv);
      const T rc = reciprocal(pv);
      unsigned own_pivot[LPT];
      T m[LPT];
#pragma unroll
      for (int q = 0; q < LPT; ++q) {
        T l = corrected_quotient(v[q][0], pv, rc);
        if (!plain) l = plain_quotient(v[q][0], pv);
        const bool here = !done[q] && pos[q] == p;  // the pivot line: position k from now on
        own_pivot[q] = __ballot_sync(0xffffffffu, here);
        if (!done[q] && pos[q] == k) pos[q] = p;
        if (here) pos[q] = k;
        done[q] |= here;
        if (!done[q]) sm.val[t * kPitchL + tid + q * NT] = l;
        m[q] = nz ? l : T(0);
      }
#pragma unroll
      for (int j = 0; j < LEN - 1; ++j) {
        const T u = line[j + 1];
#pragma unroll
        for (int q = 0; q < LPT; ++q) v[q][j] = fma(-m[q], u, v[q][j + 1]);
      }
#pragma unroll
      for (int q = 0; q < LPT; ++q)  // its values are row k of U, written by its warp's lanes
        if (own_pivot[q] && t + lane < kPanelW)
          sm.val[(t + lane) * kPitchL + wp * 32 + q * NT + __ffs(own_pivot[q]) - 1] = line[lane];
    }
    if (tid == 0) {
      if (C > 1 && t + 2 < P.w && mbar_try(smem_u32(&sm.bar[par]), (t >> 1) & 1))
        mbar_expect(smem_u32(&sm.bar[par]), (unsigned)C * kMsgBytes<T>);  // for step t + 2
      if (rank == 0 && p >= k && p < P.n) {
        P.piv[k] = p;
        if (pv == T(0) && *P.info == 0) *P.info = k + 1;
      }
    }
  }
  return true;
}

// The sub-panel of the cluster's lines: load(v) fills the registers of this CTA's lines [base,
// base + nl) (line tid + q NT in v[q]), the steps run, and on success every line's values are
// in sm.val and its final position in sm.pos (all threads return true).
template <typename T, int LPT, int NT, typename Load>
__device__ __forceinline__ bool panel_on_cluster(const PanelStep& P, PanelSmem<T, LPT, NT>& sm, int C, int rank,
                                                 int base, int nl, Load load) {
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x;
  for (int i = tid; i < 2 * NW * kPanelW; i += NT) (&sm.cand[0][0][0])[i] = T(0);
  if (tid == 0) {
    mbar_init(smem_u32(&sm.bar[0]), 1);
    mbar_init(smem_u32(&sm.bar[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect(smem_u32(&sm.bar[0]), (unsigned)C * kMsgBytes<T>);
    mbar_expect(smem_u32(&sm.bar[1]), (unsigned)C * kMsgBytes<T>);
    sm.abort[0] = sm.abort[1] = 0;
  }
  __syncthreads();
  if (C > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  T v[LPT][kPanelW];
  int pos[LPT];
  bool done[LPT];
#pragma unroll
  for (int q = 0; q < LPT; ++q) {
    const int c = tid + q * NT;
    done[q] = c >= nl;
    pos[q] = c < nl ? base + c : INT_MAX;
  }
  load(v);
  // a thread reads and writes only its own lines of sm.val until the last barrier
  bool ok = panel_steps<T, LPT, NT, 32>(P, sm, C, rank, v, pos, done);
  if (ok && P.w > 8) ok = panel_steps<T, LPT, NT, 24>(P, sm, C, rank, v, pos, done);
  if (ok && P.w > 16) ok = panel_steps<T, LPT, NT, 16>(P, sm, C, rank, v, pos, done);
  if (ok && P.w > 24) ok = panel_steps<T, LPT, NT, 8>(P, sm, C, rank, v, pos, done);
#pragma unroll
  for (int q = 0; q < LPT; ++q) sm.pos[tid + q * NT] = pos[q];
  __syncthreads();
  const bool failed = !ok || *(volatile int*)&sm.abort[0] || *(volatile int*)&sm.abort[1];
  if (C > 1) {  // no CTA leaves, or writes lines back, while another may still send or read
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  return !failed;
}

// Launch of a kernel whose grid is `clusters` clusters of C CTAs along x.
template <typename... Params, typename... Args>
cudaError_t launch_clusters(void (*kernel)(Params...), int clusters, int C, int threads, size_t smem,
                            cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(clusters * C);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = C;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Whether a cluster of 16 CTAs of the kernel fits the device (its attributes are set here).
template <typename... Params>
bool cluster_fits(void (*kernel)(Params...), int threads, size_t smem) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kMaxCluster);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kMaxCluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int num = 0;
  if (cudaOccupancyMaxActiveClusters(&num, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return num >= 1;
}

}  // namespace bem
