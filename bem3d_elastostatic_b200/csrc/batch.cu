// Many small systems in few launches: each system is a boundary mesh of its own
// (size, material, supports) with nrhs load cases (sets of prescribed values).
//
//   geometry    one etaxja launch over the elements of every system
//   assembly    H (rigid-body diagonal included) and G of every system in two
//               launches (assembly.cu: a persistent work queue over (system, 32-node
//               tile) items for the regular pairs, one warp per node for the singular
//               ones)
//   combine     per system: FI of every load case, FI_r = G[:, t known] t_r -
//               H[:, u known] u_r, then A in place of H by the column swap of
//               assembly_mod.f90:125-218 (A(:, dof) = H(:, dof) unless u is known there,
//               minus mu G for every element that prescribes u at that node), then
//               the pinned rows
//   solve       batch_lu.cu: the LU of all systems panel by panel (LAPACK dgetrf: row
//               pivoting of A), in FP32 (refined) or FP64 (plain), then the substitution
//               for all load cases and the FP64 residual / backward error of each system,
//               for a fixed number of refinement sweeps in which converged systems skip
//               their work.  The whole solve is captured once in a CUDA graph and replayed.
//
// The column swap is formed from H and G, so a node's prescribed displacement must be
// the same in every element that prescribes it (the single-system path takes each
// element's own value); bem_batch_add rejects meshes that break this.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <string>
#include <vector>

#include "asm_args.cuh"
#include "batch_dev.cuh"
#include "common.cuh"

namespace bem {
namespace {

// ---------------------------------------------------------------------------------
// combine
// ---------------------------------------------------------------------------------

// FI_r = sum_terms coef[t][r] * M_t(:, col_t), M = G (kind 0) or H (kind 1)
__global__ void batch_fi_kernel(const SysDev* __restrict__ sys, const double* __restrict__ H,
                                const double* __restrict__ G, const int2* __restrict__ terms,
                                const double* __restrict__ coef, double* __restrict__ FI) {
  const SysDev S = sys[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.N) return;
  double acc[kMaxRhs];
  for (int r = 0; r < kMaxRhs; ++r) acc[r] = 0.0;
  const double* Hs = H + S.a_off;
  const double* Gs = G + S.g_off;
  for (int64_t t = 0; t < S.nfl; ++t) {
    const int2 tm = terms[S.fl_off + t];
    const double m = tm.x == 0 ? Gs[i + tm.y * S.ldg] : Hs[i + tm.y * S.lda];
    const double* cf = coef + (S.fl_off + t) * kMaxRhs;
    for (int r = 0; r < S.nrhs; ++r) acc[r] = fma(m, cf[r], acc[r]);
  }
  double* F = FI + S.v_off;
  for (int r = 0; r < S.nrhs; ++r) F[i + (int64_t)r * S.N] = acc[r];
}

// A(:, dof) = (u known at dof ? 0 : H(:, dof)) - mu * sum of the dof's G columns, in
// place of H; one CTA per (system, dof).  ukcsr holds per system the N u-known flags
// and the N + 1 offsets of the dof's entries in the (dof, G column) list cs.
__global__ void batch_a_kernel(const SysDev* __restrict__ sys, double* __restrict__ HA,
                               const double* __restrict__ G, const int2* __restrict__ cs,
                               const int* __restrict__ ukcsr) {
  const SysDev S = sys[blockIdx.y];
  const int d = blockIdx.x;
  if (d >= S.N) return;
  double* col = HA + S.a_off + (int64_t)d * S.lda;
  const double* Gs = G + S.g_off;
  const int* uk = ukcsr + S.uk_off;
  const int beg = uk[S.N + d], end = uk[S.N + d + 1];
  const bool known = uk[d] != 0;
  for (int i = threadIdx.x; i < S.N; i += blockDim.x) {
    double a = known ? 0.0 : col[i];
    for (int q = beg; q < end; ++q) a -= S.mu * Gs[i + (int64_t)cs[S.cs_off + q].y * S.ldg];
    col[i] = a;
  }
}

__global__ void batch_pins_kernel(const SysDev* __restrict__ sys, const int* __restrict__ pins,
                                  double* __restrict__ A, double* __restrict__ FI) {
  const SysDev S = sys[blockIdx.y];
  if (blockIdx.x >= S.npins) return;
  const int p = pins[S.pin_off + blockIdx.x];
  double* As = A + S.a_off;
  for (int c = threadIdx.x; c < S.N; c += blockDim.x) As[p + (int64_t)c * S.lda] = (c == p) ? 1.0 : 0.0;
  if (threadIdx.x < S.nrhs) FI[S.v_off + p + (int64_t)threadIdx.x * S.N] = 0.0;
}

}  // namespace
}  // namespace bem

// =====================================================================================
// host side
// =====================================================================================

struct bem_batch {
  int device = 0;
  int sm_count = 148;
  cudaStream_t stream = nullptr;
  std::string err;
  long long launches = 0;
  int nrhs = 0;
  struct Sys {
    int n, ne, npins;
    double mu, nu;
    std::vector<double> x, y, z, bc;
    std::vector<int> nconec, kconec, kode, pins;
  };
  std::vector<Sys> sys;
  std::vector<bem::SysDev> hdev;
  std::vector<int> order;  // systems by decreasing order
  bool packed = false, assembled = false, factored = false;
  int factored_precision = -1;
  // device storage
  bem::DBuf<double> x, y, z, ref, tab, H, G, vec, berr, A64f;
  bem::DBuf<double> W, dinv, red;  // solve: the sweeps' vectors, diagonal-block inverses, maxima
  bem::DBuf<int> perm, moved, lu_err;
  int64_t rows = 0, inv_blocks = 0;  // of all systems
  bem::DBuf<float> A32;
  bem::DBuf<int> nconec, kconec_loc, kconec_glob, nesim, ke, batches, node_off, piv, info, conv, uk_csr, ord;
  bem::DBuf<int2> tiles, cs, terms;
  bem::DBuf<double> coef;
  bem::DBuf<int> pins;
  bem::DBuf<bem::AsmArgs> args;
  bem::DBuf<bem::SysDev> dsys;
  bem::DBuf<unsigned> counters;
  int ntiles = 0, total_nodes = 0, total_elems = 0;
  // solve graph
  cudaGraphExec_t graph = nullptr;
  int graph_key[3] = {-1, -1, -1};
  double graph_tol = -1.0;
  long long graph_launches = 0;
  unsigned long long wait_ns = 2000000000ull;  // BEM_OPT_WAIT_LIMIT_MS
  int withhold_pivot = -1;                     // BEM_OPT_WITHHOLD_PIVOT
  int lu_threads = 0;  // CTA size of the LU the solve took
  // the solutions of the latest solve on the host (pinned), fetched with the first one asked for
  double* host_x = nullptr;
  size_t host_cap = 0;
  bool host_valid = false;
  std::mutex host_lock;  // of the three above: threads may fetch solutions at the same time
  ~bem_batch() {
    if (host_x) cudaFreeHost(host_x);
    if (graph) cudaGraphExecDestroy(graph);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

int bfail(bem_batch* b, int code, const std::string& msg) {
  if (b) b->err = msg;
  return code;
}
#define BB_CUDA(b, call)                                                                      \
  do {                                                                                        \
    cudaError_t _e = (call);                                                                  \
    if (_e != cudaSuccess) return bfail((b), BEM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
  } while (0)

template <typename T>
int up(bem_batch* b, bem::DBuf<T>& d, const std::vector<T>& h) {
  BB_CUDA(b, d.alloc(std::max<size_t>(1, h.size())));
  if (!h.empty()) BB_CUDA(b, cudaMemcpyAsync(d.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, b->stream));
  return BEM_OK;
}

}  // namespace

extern "C" {

int bem_batch_create(bem_batch** out, int device) {
  if (!out) return BEM_ERR_ARG;
  *out = nullptr;
  bem_batch* b = new bem_batch();
  b->device = device;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&b->sm_count, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) {
    delete b;
    return BEM_ERR_CUDA;
  }
  *out = b;
  return BEM_OK;
}

int bem_batch_destroy(bem_batch* b) {
  if (!b) return BEM_OK;
  cudaSetDevice(b->device);
  cudaStreamSynchronize(b->stream);
  delete b;
  return BEM_OK;
}

const char* bem_batch_last_error(const bem_batch* b) { return b ? b->err.c_str() : "null batch"; }

int bem_batch_add(bem_batch* b, int n, int ne, const double* x, const double* y, const double* z, const int* nconec,
                  const int* kconec, double mu, double nu, const int* kode, int nrhs, const double* bc, int npins,
                  const int* pins) {
  if (!b || n <= 0 || ne <= 0 || !x || !y || !z || !nconec || !kconec || !kode || !bc || nrhs < 1 ||
      nrhs > bem::kMaxRhs || npins < 0 || (npins > 0 && !pins) || !(mu > 0.0))
    return bfail(b, BEM_ERR_ARG, "batch_add: bad arguments");
  if (b->nrhs == 0) b->nrhs = nrhs;
  if (nrhs != b->nrhs) return bfail(b, BEM_ERR_ARG, "batch_add: every system needs the same number of load cases");
  bem_batch::Sys s;
  s.n = n;
  s.ne = ne;
  s.mu = mu;
  s.nu = nu;
  s.npins = npins;
  s.x.assign(x, x + n);
  s.y.assign(y, y + n);
  s.z.assign(z, z + n);
  s.nconec.assign(nconec, nconec + ne);
  s.kconec.assign(kconec, kconec + 9 * (size_t)ne);
  s.kode.assign(kode, kode + 3 * (size_t)ne);
  s.bc.assign(bc, bc + 27 * (size_t)ne * nrhs);
  s.pins.assign(pins, pins + npins);
  std::vector<int> cnt(n, 0);
  for (int e = 0; e < ne; ++e) {
    if (nconec[e] != 9 && nconec[e] != 6) return bfail(b, BEM_ERR_MESH, "batch_add: nconec must be 6 or 9");
    for (int m = 0; m < 9; ++m) {
      if (m >= nconec[e]) {
        s.kconec[m + 9 * (size_t)e] = 1;
        continue;
      }
      const int k = kconec[m + 9 * (size_t)e];
      if (k < 1 || k > n) return bfail(b, BEM_ERR_MESH, "batch_add: kconec references a node out of range");
      if (++cnt[k - 1] > 8) return bfail(b, BEM_ERR_MESH, "batch_add: a node lies in more than 8 elements");
    }
    for (int ld = 0; ld < 3; ++ld)
      if (kode[3 * e + ld] != 0 && kode[3 * e + ld] != 1) return bfail(b, BEM_ERR_ARG, "batch_add: kode must be 0 or 1");
  }
  // a node's prescribed displacement must agree over the elements that prescribe it
  for (int r = 0; r < nrhs; ++r) {
    std::vector<double> val(3 * (size_t)n, 0.0);
    std::vector<char> set(3 * (size_t)n, 0);
    const double* bcr = bc + 27 * (size_t)ne * r;
    for (int e = 0; e < ne; ++e)
      for (int ld = 0; ld < 3; ++ld)
        if (kode[3 * e + ld] == 0)
          for (int m = 0; m < nconec[e]; ++m) {
            const size_t d = 3 * (size_t)(kconec[m + 9 * (size_t)e] - 1) + ld;
            const double v = bcr[3 * m + ld + 27 * (size_t)e];
            if (set[d] && val[d] != v)
              return bfail(b, BEM_ERR_MESH, "batch_add: elements prescribe different displacements at one node");
            set[d] = 1;
            val[d] = v;
          }
  }
  for (int i = 0; i < npins; ++i)
    if (pins[i] < 0 || pins[i] >= 3 * n) return bfail(b, BEM_ERR_ARG, "batch_add: pin out of range");
  b->sys.push_back(std::move(s));
  b->packed = b->assembled = b->factored = b->host_valid = false;
  if (b->graph) {  // captured for the systems so far
    cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
  }
  return (int)b->sys.size() - 1;
}

}  // extern "C"

namespace {

// The systems' arrays, lists and schedules, packed and uploaded; done again only after a system
// was added (a batch's systems do not change).
int pack(bem_batch* b) {
  const int ns = (int)b->sys.size(), nrhs = b->nrhs;
  // host packing
  std::vector<double> hx, hy, hz;
  std::vector<int> hnc, hkl, hkg, hnesim, hke, hbatch, hnode_off(ns + 1, 0), hpins;
  std::vector<int2> htiles, hcs, hterms;
  std::vector<double> hcoef;
  std::vector<int> huk;  // per system: N u-known flags, then N + 1 row pointers of the cs list
  std::vector<bem::SysDev> hs(ns);
  int64_t a_off = 0, g_off = 0, v_off = 0, piv_off = 0, inv_off = 0, elem_off = 0, batch_off = 0;
  std::vector<int64_t> elem_offs(ns), batch_offs(ns), node_offs(ns);
  std::vector<int> nbatches(ns);
  for (int si = 0; si < ns; ++si) {
    const auto& S = b->sys[si];
    const int n = S.n, ne = S.ne, N = 3 * n;
    bem::SysDev& D = hs[si];
    D.n = n;
    D.ne = ne;
    D.N = N;
    D.nrhs = nrhs;
    D.lda = ((int64_t)N + 31) / 32 * 32;
    D.ldg = D.lda;
    D.a_off = a_off;
    a_off += D.lda * N;
    D.g_off = g_off;
    g_off += D.ldg * 27 * (int64_t)ne;
    D.f_off = D.a_off;
    D.v_off = v_off;
    v_off += (int64_t)N * nrhs;
    D.piv_off = piv_off;
    piv_off += N;
    D.inv_off = inv_off;
    inv_off += (N + 127) / 128;
    D.mu = S.mu;
    node_offs[si] = hx.size();
    hnode_off[si] = (int)hx.size();
    hx.insert(hx.end(), S.x.begin(), S.x.end());
    hy.insert(hy.end(), S.y.begin(), S.y.end());
    hz.insert(hz.end(), S.z.begin(), S.z.end());
    elem_offs[si] = elem_off;
    elem_off += ne;
    hnc.insert(hnc.end(), S.nconec.begin(), S.nconec.end());
    for (size_t k = 0; k < S.kconec.size(); ++k) {
      hkl.push_back(S.kconec[k]);
      hkg.push_back(S.kconec[k] + (int)node_offs[si]);
    }
    // adjacency (io_mod.f90:125-135)
    std::vector<int> nes(n, 0), kel(8 * (size_t)n, 0);
    for (int e = 0; e < ne; ++e)
      for (int m = 0; m < S.nconec[e]; ++m) {
        const int in = S.kconec[m + 9 * (size_t)e] - 1;
        kel[nes[in]++ + 8 * (size_t)in] = e + 1;
      }
    hnesim.insert(hnesim.end(), nes.begin(), nes.end());
    hke.insert(hke.end(), kel.begin(), kel.end());
    // conflict-free element batches of the regular kernel (elements sharing no node)
    {
      std::vector<int> sched;
      std::vector<char> used(ne, 0);
      int left = ne, start = 0;
      while (left > 0) {
        std::vector<int> batch;
        std::vector<int> touched;
        for (int e = start; e < ne && (int)batch.size() < bem::kBatch; ++e) {
          if (used[e]) continue;
          bool clash = false;
          for (int m = 0; m < S.nconec[e] && !clash; ++m)
            for (int t : touched)
              if (t == S.kconec[m + 9 * (size_t)e]) clash = true;
          if (clash) continue;
          batch.push_back(e);
          used[e] = 1;
          --left;
          for (int m = 0; m < S.nconec[e]; ++m) touched.push_back(S.kconec[m + 9 * (size_t)e]);
        }
        while (start < ne && used[start]) ++start;
        for (int w = 0; w < bem::kBatch; ++w) sched.push_back(w < (int)batch.size() ? batch[w] : -1);
      }
      nbatches[si] = (int)sched.size() / bem::kBatch;
      batch_offs[si] = batch_off;
      batch_off += sched.size();
      hbatch.insert(hbatch.end(), sched.begin(), sched.end());
    }
    for (int t = 0; t < (n + 31) / 32; ++t) htiles.push_back(make_int2(si, t));
    // column swap: per dof, G columns of the elements prescribing u there; u-known flags
    std::vector<std::vector<int>> lists(N);
    std::vector<int> uk(N, 0);
    std::vector<double> vp(3 * (size_t)n * nrhs, 0.0);
    for (int in = 0; in < n; ++in)  // first element in ke order prescribing u (as build_lookup)
      for (int ld = 0; ld < 3; ++ld)
        for (int i = 0; i < nes[in] && i < 8 && !uk[3 * in + ld]; ++i) {
          const int e = kel[i + 8 * (size_t)in] - 1;
          if (S.kode[3 * e + ld] == 0)
            for (int m = 0; m < S.nconec[e]; ++m)
              if (S.kconec[m + 9 * (size_t)e] - 1 == in) {
                uk[3 * in + ld] = 1;
                for (int r = 0; r < nrhs; ++r)
                  vp[3 * in + ld + 3 * (size_t)n * r] = S.bc[3 * m + ld + 27 * (size_t)e + 27 * (size_t)ne * r];
                break;
              }
        }
    D.fl_off = (int64_t)hterms.size();
    for (int e = 0; e < ne; ++e)
      for (int k = 0; k < S.nconec[e]; ++k)
        for (int ld = 0; ld < 3; ++ld) {
          const int dof = 3 * (S.kconec[k + 9 * (size_t)e] - 1) + ld;
          const int gcol = 27 * e + 3 * k + ld;
          if (S.kode[3 * e + ld] == 0) {
            lists[dof].push_back(gcol);
          } else {  // traction known: FI += G(:, gcol) t
            bool any = false;
            double cf[bem::kMaxRhs] = {0};
            for (int r = 0; r < nrhs; ++r) {
              cf[r] = S.bc[3 * k + ld + 27 * (size_t)e + 27 * (size_t)ne * r];
              any |= cf[r] != 0.0;
            }
            if (any) {
              hterms.push_back(make_int2(0, gcol));
              hcoef.insert(hcoef.end(), cf, cf + bem::kMaxRhs);
            }
          }
        }
    for (int d = 0; d < N; ++d)  // u known: FI -= H(:, dof) u
      if (uk[d]) {
        bool any = false;
        double cf[bem::kMaxRhs] = {0};
        for (int r = 0; r < nrhs; ++r) {
          cf[r] = -vp[d + 3 * (size_t)n * r];
          any |= cf[r] != 0.0;
        }
        if (any) {
          hterms.push_back(make_int2(1, d));
          hcoef.insert(hcoef.end(), cf, cf + bem::kMaxRhs);
        }
      }
    D.nfl = (int64_t)hterms.size() - D.fl_off;
    D.cs_off = (int64_t)hcs.size();
    D.uk_off = (int64_t)huk.size();
    huk.insert(huk.end(), uk.begin(), uk.end());
    int acc = 0;
    for (int d = 0; d < N; ++d) {
      huk.push_back(acc);
      for (int gcol : lists[d]) hcs.push_back(make_int2(d, gcol));
      acc += (int)lists[d].size();
    }
    huk.push_back(acc);
    D.ncs = acc;
    D.pin_off = (int64_t)hpins.size();
    D.npins = S.npins;
    hpins.insert(hpins.end(), S.pins.begin(), S.pins.end());
  }
  hnode_off[ns] = (int)hx.size();
  b->total_nodes = (int)hx.size();
  b->total_elems = (int)elem_off;
  // the regular work items, largest systems first
  std::vector<int> ordsys(ns);
  for (int i = 0; i < ns; ++i) ordsys[i] = i;
  std::stable_sort(ordsys.begin(), ordsys.end(), [&](int a, int c) {
    return (int64_t)b->sys[a].n * b->sys[a].ne > (int64_t)b->sys[c].n * b->sys[c].ne;
  });
  std::vector<int2> sorted_tiles;
  for (int si : ordsys)
    for (int t = 0; t < (b->sys[si].n + 31) / 32; ++t) sorted_tiles.push_back(make_int2(si, t));
  b->ntiles = (int)sorted_tiles.size();
  b->order = ordsys;
  std::stable_sort(b->order.begin(), b->order.end(), [&](int a, int c) { return b->sys[a].n > b->sys[c].n; });
  // device
  int rc;
  if ((rc = up(b, b->x, hx)) || (rc = up(b, b->y, hy)) || (rc = up(b, b->z, hz)) || (rc = up(b, b->nconec, hnc)) ||
      (rc = up(b, b->kconec_loc, hkl)) || (rc = up(b, b->kconec_glob, hkg)) || (rc = up(b, b->nesim, hnesim)) ||
      (rc = up(b, b->ke, hke)) || (rc = up(b, b->batches, hbatch)) || (rc = up(b, b->node_off, hnode_off)) ||
      (rc = up(b, b->tiles, sorted_tiles)) || (rc = up(b, b->cs, hcs)) || (rc = up(b, b->terms, hterms)) ||
      (rc = up(b, b->coef, hcoef)) || (rc = up(b, b->uk_csr, huk)) || (rc = up(b, b->pins, hpins)) ||
      (rc = up(b, b->ord, b->order)))
    return rc;
  const size_t ng = (size_t)bem::kGp * elem_off;
  BB_CUDA(b, b->ref.alloc(16 * ng));
  BB_CUDA(b, b->tab.alloc((size_t)bem::kTabStride * elem_off));
  BB_CUDA(b, b->H.alloc((size_t)std::max<int64_t>(1, a_off)));
  BB_CUDA(b, b->G.alloc((size_t)std::max<int64_t>(1, g_off)));
  BB_CUDA(b, b->vec.alloc((size_t)3 * std::max<int64_t>(1, v_off)));  // FI, X, R
  BB_CUDA(b, b->piv.alloc((size_t)std::max<int64_t>(1, piv_off)));
  BB_CUDA(b, b->info.alloc(ns));
  BB_CUDA(b, b->conv.alloc(ns));
  BB_CUDA(b, b->berr.alloc(ns));
  BB_CUDA(b, b->counters.alloc(64));
  b->rows = piv_off;
  b->inv_blocks = inv_off;
  // per-system assembly arguments (mode HG)
  std::vector<bem::AsmArgs> hargs(ns);
  for (int si = 0; si < ns; ++si) {
    const auto& S = b->sys[si];
    bem::AsmArgs& P = hargs[si];
    P = bem::AsmArgs{};
    P.n = S.n;
    P.ne = S.ne;
    P.nbatches = nbatches[si];
    P.in0 = 0;
    P.nrows_nodes = S.n;
    P.batches = b->batches.p + batch_offs[si];
    P.nconec = b->nconec.p + elem_offs[si];
    P.kconec = b->kconec_loc.p + 9 * elem_offs[si];
    P.nesim = b->nesim.p + node_offs[si];
    P.ke = b->ke.p + 8 * node_offs[si];
    P.x = b->x.p + node_offs[si];
    P.y = b->y.p + node_offs[si];
    P.z = b->z.p + node_offs[si];
    P.tab = b->tab.p + (size_t)bem::kTabStride * elem_offs[si];
    P.mat = bem::make_material(S.mu, S.nu);
    P.A = b->H.p + hs[si].a_off;
    P.lda = hs[si].lda;
    P.G = b->G.p + hs[si].g_off;
    P.ldg = hs[si].ldg;
  }
  if ((rc = up(b, b->args, hargs)) || (rc = up(b, b->dsys, hs))) return rc;
  b->hdev = hs;
  BB_CUDA(b, cudaStreamSynchronize(b->stream));  // the host vectors end here
  b->packed = true;
  return BEM_OK;
}

}  // namespace

extern "C" {

int bem_batch_assemble(bem_batch* b) {
  if (!b || b->sys.empty()) return bfail(b, BEM_ERR_STATE, "batch_assemble: no systems");
  BB_CUDA(b, cudaSetDevice(b->device));
  int rc;
  if (!b->packed && (rc = pack(b))) return rc;
  const int ns = (int)b->sys.size();
  const int64_t elem_off = b->total_elems;
  const auto& hs = b->hdev;
  // geometry of every element, then H and G of every system
  if (bem::launch_geometry_arrays(b->stream, (int)elem_off, b->x.p, b->y.p, b->z.p, b->nconec.p, b->kconec_glob.p,
                                  b->ref.p, b->tab.p))
    return bfail(b, BEM_ERR_CUDA, "batch geometry launch failed");
  ++b->launches;
  BB_CUDA(b, cudaMemsetAsync(b->H.p, 0, b->H.bytes(), b->stream));
  if (bem::launch_batch_hg(b->stream, b->sm_count, b->args.p, b->tiles.p, b->ntiles, b->counters.p, b->node_off.p,
                           ns, b->total_nodes, &b->launches))
    return bfail(b, BEM_ERR_CUDA, "batch assembly launch failed");
  // FI of every load case, then A in place of H, then the pinned rows
  int maxN = 0, maxp = 1;
  for (auto& D : hs) {
    maxN = std::max(maxN, D.N);
    maxp = std::max<int>(maxp, (int)D.npins);
  }
  bem::batch_fi_kernel<<<dim3((maxN + 127) / 128, ns), 128, 0, b->stream>>>(b->dsys.p, b->H.p, b->G.p, b->terms.p,
                                                                             b->coef.p, b->vec.p);
  bem::batch_a_kernel<<<dim3(maxN, ns), 128, 0, b->stream>>>(b->dsys.p, b->H.p, b->G.p, b->cs.p, b->uk_csr.p);
  bem::batch_pins_kernel<<<dim3(maxp, ns), 256, 0, b->stream>>>(b->dsys.p, b->pins.p, b->H.p, b->vec.p);
  BB_CUDA(b, cudaGetLastError());
  b->launches += 3;
  BB_CUDA(b, cudaStreamSynchronize(b->stream));
  b->assembled = true;
  b->factored = b->host_valid = false;
  return BEM_OK;
}

}  // extern "C"

// bem_batch_info: include/bem3d_b200.h

extern "C" {

int bem_batch_set_option(bem_batch* b, int option, int64_t value) {
  if (!b) return BEM_ERR_ARG;
  if (option == BEM_OPT_WAIT_LIMIT_MS) {
    if (value < 1 || value > 60000) return bfail(b, BEM_ERR_ARG, "batch_set_option: wait limit must be 1..60000 ms");
    b->wait_ns = (unsigned long long)value * 1000000ull;
  } else if (option == BEM_OPT_WITHHOLD_PIVOT) {
    if (value < -1 || value > INT32_MAX) return bfail(b, BEM_ERR_ARG, "batch_set_option: bad pivot index");
    b->withhold_pivot = (int)value;
  } else {
    return bfail(b, BEM_ERR_ARG, "batch_set_option: unknown option");
  }
  if (b->graph) {  // captured with the former value
    cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
  }
  return BEM_OK;
}

int bem_batch_solve(bem_batch* b, int precision, double tol, int max_iter, bem_batch_info* info) {
  if (!b || !b->assembled) return bfail(b, BEM_ERR_STATE, "batch_solve before batch_assemble");
  b->host_valid = false;
  if (precision != BEM_PREC_FP64 && precision != BEM_PREC_FP32_IR)
    return bfail(b, BEM_ERR_ARG, "batch_solve: precision must be BEM_PREC_FP64 or BEM_PREC_FP32_IR");
  if (max_iter < 1 || max_iter > 30) return bfail(b, BEM_ERR_ARG, "batch_solve: max_iter must be in 1..30");
  for (const auto& D : b->hdev)
    if (D.N > bem::kMaxOrder) return bfail(b, BEM_ERR_TOO_LARGE, "batch_solve: a system of order above 25,600");
  BB_CUDA(b, cudaSetDevice(b->device));
  int rc;
  const int ns = (int)b->sys.size();
  const int sweeps = precision == BEM_PREC_FP64 ? 0 : max_iter;
  if (precision == BEM_PREC_FP64) {
    if (b->A64f.count < b->H.count) BB_CUDA(b, b->A64f.alloc(b->H.count));
  } else {
    if (b->A32.count < b->H.count) BB_CUDA(b, b->A32.alloc(b->H.count));
  }
  BB_CUDA(b, b->W.alloc((size_t)b->rows * bem::kMaxRhs));
  BB_CUDA(b, b->dinv.alloc((size_t)b->inv_blocks * 2 * 128 * 128));
  BB_CUDA(b, b->red.alloc((size_t)ns * (3 * bem::kMaxRhs + 1)));
  BB_CUDA(b, b->perm.alloc((size_t)b->rows));
  BB_CUDA(b, b->moved.alloc((size_t)ns * 64));
  BB_CUDA(b, b->lu_err.alloc(2));
  // the solve as one CUDA graph, captured once per (precision, sweeps, tol)
  if (!b->graph || b->graph_key[0] != precision || b->graph_key[1] != sweeps || b->graph_tol != tol) {
    if (b->graph) {
      cudaGraphExecDestroy(b->graph);
      b->graph = nullptr;
    }
    bem::BatchSolve S{};
    const int64_t nv = b->vec.count / 3;
    S.stream = b->stream;
    S.sm_count = b->sm_count;
    S.sys = b->dsys.p;
    S.order = b->ord.p;
    for (int i : b->order) S.N.push_back(b->hdev[i].N);
    S.A = b->H.p;
    S.FI = b->vec.p;
    S.X = b->vec.p + nv;
    S.R = b->vec.p + 2 * nv;
    S.W = b->W.p;
    S.dinv = b->dinv.p;
    S.red = b->red.p;
    S.berr = b->berr.p;
    S.piv = b->piv.p;
    S.perm = b->perm.p;
    S.info = b->info.p;
    S.conv = b->conv.p;
    S.moved = b->moved.p;
    S.err = b->lu_err.p;
    S.wait_ns = b->wait_ns;
    S.withhold_pivot = b->withhold_pivot;
    S.nsys = ns;
    const int cap = precision == BEM_PREC_FP64 ? bem::batch_lu_max_order<double>() : bem::batch_lu_max_order<float>();
    b->lu_threads = S.N[0] <= cap ? 256 : 512;
    BB_CUDA(b, cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    const bool queued = (precision == BEM_PREC_FP64) ? bem::batch_solve_enqueue<double>(S, b->A64f.p, tol, 0)
                                                     : bem::batch_solve_enqueue<float>(S, b->A32.p, tol, sweeps);
    rc = queued ? BEM_OK
                : bfail(b, BEM_ERR_CUDA, std::string("batch solve launch failed: ") + cudaGetErrorString(cudaGetLastError()));
    b->graph_launches = S.launches;
    cudaGraph_t g = nullptr;
    cudaError_t ce = cudaStreamEndCapture(b->stream, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (ce != cudaSuccess) return bfail(b, BEM_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(ce));
    ce = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) return bfail(b, BEM_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(ce));
    b->graph_key[0] = precision;
    b->graph_key[1] = sweeps;
    b->graph_tol = tol;
  }
  b->factored = false;  // until this solve has succeeded: it writes over the last one's vectors
  cudaEvent_t e0, e1;
  BB_CUDA(b, cudaEventCreate(&e0));
  BB_CUDA(b, cudaEventCreate(&e1));
  BB_CUDA(b, cudaEventRecord(e0, b->stream));
  BB_CUDA(b, cudaGraphLaunch(b->graph, b->stream));
  BB_CUDA(b, cudaEventRecord(e1, b->stream));
  BB_CUDA(b, cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  b->launches += b->graph_launches;
  int lerr = 0;
  BB_CUDA(b, cudaMemcpy(&lerr, b->lu_err.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (lerr != 0) return bfail(b, lerr, "batch_solve: a wait of the panel factorisation timed out");
  std::vector<int> hconv(ns), hinfo(ns);
  std::vector<double> hbe(ns);
  BB_CUDA(b, cudaMemcpy(hconv.data(), b->conv.p, ns * sizeof(int), cudaMemcpyDeviceToHost));
  BB_CUDA(b, cudaMemcpy(hinfo.data(), b->info.p, ns * sizeof(int), cudaMemcpyDeviceToHost));
  BB_CUDA(b, cudaMemcpy(hbe.data(), b->berr.p, ns * sizeof(double), cudaMemcpyDeviceToHost));
  bem_batch_info st{};
  st.systems = ns;
  st.sweeps = sweeps;
  for (int s = 0; s < ns; ++s) {
    if (hinfo[s]) ++st.singular;
    else {
      st.max_backward_error = std::max(st.max_backward_error, hbe[s]);
      if (hconv[s] == 1 || hbe[s] <= tol) ++st.converged;
    }
  }
  st.solve_seconds = ms * 1e-3;
  st.lu_threads = b->lu_threads;
  if (info) *info = st;
  b->factored = true;
  b->factored_precision = precision;
  return st.singular ? BEM_ERR_NOCONV : BEM_OK;
}

int bem_batch_get_solution(bem_batch* b, int i, double* x) {
  if (!b) return BEM_ERR_ARG;
  std::lock_guard<std::mutex> lock(b->host_lock);
  if (!b->factored || i < 0 || i >= (int)b->sys.size() || !x)
    return bfail(b, BEM_ERR_ARG, "batch_get_solution: bad arguments or no solve");
  const auto& D = b->hdev[i];
  const int64_t nv = b->vec.count / 3;
  const size_t mine = (size_t)D.N * D.nrhs;
  // one copy of all solutions instead of one per system (28 us each); large batches, or without
  // pinned memory, directly
  constexpr size_t kHostMost = size_t(32) << 20;  // doubles
  if (!b->host_valid && (size_t)nv <= kHostMost) {
    if (b->host_cap < (size_t)nv) {
      if (b->host_x) cudaFreeHost(b->host_x);
      b->host_x = nullptr;
      b->host_cap = 0;
      if (cudaMallocHost(&b->host_x, (size_t)nv * sizeof(double)) == cudaSuccess) b->host_cap = (size_t)nv;
      else cudaGetLastError();
    }
    if (b->host_cap >= (size_t)nv) {
      BB_CUDA(b, cudaMemcpy(b->host_x, b->vec.p + nv, (size_t)nv * sizeof(double), cudaMemcpyDeviceToHost));
      b->host_valid = true;
    }
  }
  if (b->host_valid) std::copy(b->host_x + D.v_off, b->host_x + D.v_off + mine, x);
  else BB_CUDA(b, cudaMemcpy(x, b->vec.p + nv + D.v_off, mine * sizeof(double), cudaMemcpyDeviceToHost));
  return BEM_OK;
}

int bem_batch_get_system(bem_batch* b, int i, double* A, double* FI) {
  if (!b || !b->assembled || i < 0 || i >= (int)b->sys.size())
    return bfail(b, BEM_ERR_ARG, "batch_get_system: bad arguments or no assembly");
  const auto& D = b->hdev[i];
  if (A)
    BB_CUDA(b, cudaMemcpy2D(A, (size_t)D.N * sizeof(double), b->H.p + D.a_off, (size_t)D.lda * sizeof(double),
                            (size_t)D.N * sizeof(double), D.N, cudaMemcpyDeviceToHost));
  if (FI)
    BB_CUDA(b, cudaMemcpy(FI, b->vec.p + D.v_off, (size_t)D.N * D.nrhs * sizeof(double), cudaMemcpyDeviceToHost));
  return BEM_OK;
}

long long bem_batch_launches(const bem_batch* b) { return b ? b->launches : -1; }

}  // extern "C"
