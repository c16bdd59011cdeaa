// compute_internal_points (stress_mod.f90:511-886) on the GPU: Somigliana
// displacement and stress identities at internal points, with the reference's
// two-tier quadrature (the element's own 6x6 / 4x4 table when the point is farther
// than 3.5 element radii from its centroid, a 40x40 Gauss-Legendre table otherwise)
// and calc_principal_and_vm (:299-359).
//
// Kernels
//   far_table / near_table  pre-weighted Gauss-point tables (:580-726), 18 doubles per
//                           point: x, y, z, n1, n2, n3, u*w (3), t*w (3) and the six
//                           products of n and u*w that the stress identity adds
//   far_kernel              a CTA takes a tile of 256 internal points and a share of the
//                           elements, whose tables it streams through a double-buffered
//                           shared-memory ring (cp.async) and reads as broadcasts; near
//                           elements are skipped
//   near_count / near_scan / near_fill   the (point, near element) pairs, point by point
//                           and, as index lists, element by element
//   near_kernel             a CTA takes one element and up to 256 of its near points, so
//                           that the element's 1600 points are staged once for all of
//                           them; every pair's sums go to its own place
//   finish_kernel           adds a point's far shares and near pairs in their order and
//                           forms the principal stresses
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "recip.cuh"
#include "shape.cuh"
#include "stress.cuh"

namespace bem {

constexpr int kNearN = 40;
constexpr int kNear = kNearN * kNearN;
constexpr int kRec = 18;   // doubles per table point
constexpr int kChunk = 4;  // elements staged per shared-memory chunk (20.7 KB)

__constant__ double c_ome6[6] = {kOmeQuad[0], kOmeQuad[1], kOmeQuad[2], kOmeQuad[3], kOmeQuad[4], kOmeQuad[5]};
__constant__ double c_omei4[4] = {kOmeiTri[0], kOmeiTri[1], kOmeiTri[2], kOmeiTri[3]};
__constant__ double c_omej4[4] = {kOmejTri[0], kOmejTri[1], kOmejTri[2], kOmejTri[3]};

// the 40-point rule, passed to near_table_kernel by value
struct NearRule {
  double x[kNearN], w[kNearN];
};

// gauss_legendre_1d (stress_mod.f90:475-503): Newton iteration on P_n from the
// Chebyshev-like first guess, to |dz| <= 1e-15.
static void gauss_legendre(int n, double* x, double* w) {
  const int m = (n + 1) / 2;
  for (int i = 1; i <= m; ++i) {
    double z = std::cos(kPi * ((double)i - 0.25) / ((double)n + 0.5));
    double p1 = 0, p2 = 0, p3 = 0, pp = 0;
    for (int it = 0; it < 100; ++it) {
      p1 = 1.0;
      p2 = 0.0;
      for (int j = 1; j <= n; ++j) {
        p3 = p2;
        p2 = p1;
        p1 = ((2.0 * j - 1.0) * z * p2 - (j - 1.0) * p3) / j;
      }
      pp = n * (z * p1 - p2) / (z * z - 1.0);
      const double z1 = z;
      z = z1 - p1 / pp;
      if (std::fabs(z - z1) <= 1.0e-15) break;
    }
    x[i - 1] = -z;
    x[n - i] = z;
    w[i - 1] = 2.0 / ((1.0 - z * z) * pp * pp);
    w[n - i] = w[i - 1];
  }
}

// element centroid and near threshold 3.5^2 * max |node - centroid|^2 (:584-604)
__global__ void einfo_kernel(int ne, const double* x, const double* y, const double* z, const int* nconec,
                             const int* kconec, double* einfo) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int nc = nconec[e];
  double xj[9], yj[9], zj[9], cx = 0, cy = 0, cz = 0;
  for (int m = 0; m < nc; ++m) {
    const int k = kconec[m + 9 * e] - 1;
    xj[m] = x[k];
    yj[m] = y[k];
    zj[m] = z[k];
    cx += xj[m];
    cy += yj[m];
    cz += zj[m];
  }
  cx /= nc;
  cy /= nc;
  cz /= nc;
  double d2 = 0.0;
  for (int m = 0; m < nc; ++m) {
    const double dx = xj[m] - cx, dy = yj[m] - cy, dz = zj[m] - cz;
    d2 = fmax(d2, dx * dx + dy * dy + dz * dz);
  }
  einfo[4 * e + 0] = cx;
  einfo[4 * e + 1] = cy;
  einfo[4 * e + 2] = cz;
  einfo[4 * e + 3] = (3.5 * 3.5) * d2;
}

// the record's normal, weighted u and t, and the products of n and b = u w: n_i b_i
// (xx, yy, zz), n_i b_j + n_j b_i (xy, yz, zx)
__device__ __forceinline__ void table_tail(double* P, const double* nr, const double* ug, const double* tg, double wg) {
  double b[3];
  for (int c = 0; c < 3; ++c) {
    b[c] = ug[c] * wg;
    P[3 + c] = nr[c];
    P[6 + c] = b[c];
    P[9 + c] = tg[c] * wg;
    P[12 + c] = nr[c] * b[c];
  }
  P[15] = nr[0] * b[1] + nr[1] * b[0];
  P[16] = nr[1] * b[2] + nr[2] * b[1];
  P[17] = nr[2] * b[0] + nr[0] * b[2];
}

// far table (:606-650), fixed stride of 36 points per element
__global__ void far_table_kernel(int ne, const int* nconec, const int* kconec, const double* eta1,
                                 const double* eta2, const double* eta3, const double* xja, const double* xg1,
                                 const double* xg2, const double* xg3, const double* ff, const double* U,
                                 const double* DFI, double* far) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (int64_t)ne * kGp) return;
  const int e = (int)(gid / kGp), q = (int)(gid % kGp);
  const int nc = nconec[e];
  const int npg = (nc == 9) ? 6 : 4;
  double* P = far + gid * kRec;
  if (q >= npg * npg) {
    for (int v = 0; v < kRec; ++v) P[v] = 0.0;
    return;
  }
  const int i = q / npg, j = q % npg;
  const double wg = (nc == 9) ? c_ome6[i] * c_ome6[j] * xja[gid] : c_omei4[i] * c_omej4[j] * xja[gid];
  double ug[3] = {0, 0, 0}, tg[3] = {0, 0, 0};
  for (int m = 0; m < nc; ++m) {
    const int64_t ik = kconec[m + 9 * e] - 1;
    const double f = ff[m + 9 * gid];
    for (int c = 0; c < 3; ++c) {
      ug[c] += f * U[3 * ik + c];
      tg[c] += f * DFI[3 * m + c + 27 * (int64_t)e];
    }
  }
  P[0] = xg1[gid];
  P[1] = xg2[gid];
  P[2] = xg3[gid];
  const double nr[3] = {eta1[gid], eta2[gid], eta3[gid]};
  table_tail(P, nr, ug, tg, wg);
}

// near table (:654-726): 40 x 40 Gauss-Legendre, Duffy map on tri6
__global__ void near_table_kernel(int ne, const double* x, const double* y, const double* z, const int* nconec,
                                  const int* kconec, const double* U, const double* DFI, NearRule rule, double* near) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (int64_t)ne * kNear) return;
  const int e = (int)(gid / kNear), q = (int)(gid % kNear), i = q / kNearN, j = q % kNearN;
  const int nc = nconec[e];
  double g1, g2, tj;
  if (nc == 9) {
    g1 = rule.x[i];
    g2 = rule.x[j];
    tj = 1.0;
  } else {
    g1 = 0.5 * (1.0 + rule.x[i]);
    g2 = 0.25 * (1.0 - rule.x[i]) * (1.0 + rule.x[j]);
    tj = 0.125 * (1.0 - rule.x[i]);
  }
  double f[9], fd1[9], fd2[9];
  shape_fn<double>(nc, g1, g2, f, fd1, fd2);
  double xg[3] = {0, 0, 0}, d1[3] = {0, 0, 0}, d2[3] = {0, 0, 0}, ug[3] = {0, 0, 0}, tg[3] = {0, 0, 0};
  for (int m = 0; m < nc; ++m) {
    const int64_t ik = kconec[m + 9 * e] - 1;
    const double p[3] = {x[ik], y[ik], z[ik]};
    for (int c = 0; c < 3; ++c) {
      xg[c] += f[m] * p[c];
      d1[c] += fd1[m] * p[c];
      d2[c] += fd2[m] * p[c];
      ug[c] += f[m] * U[3 * ik + c];
      tg[c] += f[m] * DFI[3 * m + c + 27 * (int64_t)e];
    }
  }
  const double c0 = d1[1] * d2[2] - d1[2] * d2[1];
  const double c1 = d1[2] * d2[0] - d1[0] * d2[2];
  const double c2 = d1[0] * d2[1] - d1[1] * d2[0];
  const double jac = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
  const double wg = rule.w[i] * rule.w[j] * tj * jac;
  double* P = near + gid * kRec;
  P[0] = xg[0];
  P[1] = xg[1];
  P[2] = xg[2];
  const double nr[3] = {c0 / jac, c1 / jac, c2 / jac};
  table_tail(P, nr, ug, tg, wg);
}

// The identities' constants.  cD = 1 / (8 pi (1 - nu)) and the others by their use in
// SomAcc::add: cU = cD / (2 mu), cS = 2 mu cD.
struct SomConst {
  double cU, cU4, cD, cDc6, cS, cS3nu, cSc6, m3c6, mc6, k15c6, pr4, asg, asgc6;
};

// Sums of the displacement and stress identities at one point.
struct SomAcc {
  double u[3] = {0.0, 0.0, 0.0};
  double d[3] = {0.0, 0.0, 0.0};  // half the diagonal stresses without their common part
  double o[3] = {0.0, 0.0, 0.0};  // xy, yz, zx
  double tr = 0.0;                // the common part

  // accumulate_somigliana_range's body (:807-885) for one table point.  With a the unit
  // vector to it, n its normal, b = u w, t = t w, the stress kernels D t - S b are
  //   a_i w_j + a_j w_i - cS c6 / r^3 (n_i b_j + n_j b_i) + delta_ij tr,
  //   w = cD c6 / r^2 t - 3 nu cS / r^3 ((a.n) b + (a.b) n) + alpha a,
  // and the displacement ones a combination of t, a, b and n with scalar factors: about 92
  // FP64 operations, where the identities written out component by component take twice
  // that (the kernels are bound by the FP64 pipe).
  __device__ __forceinline__ void add(const SomConst& K, const double* P, double xx, double yy, double zz) {
    const double2* P2 = reinterpret_cast<const double2*>(P);
    const double2 p0 = P2[0], p1 = P2[1], p2 = P2[2], p3 = P2[3], p4 = P2[4], p5 = P2[5], p6 = P2[6], p7 = P2[7],
                  p8 = P2[8];
    const double rx = p0.x - xx, ry = p0.y - yy, rz = p1.x - zz;
    const double n0 = p1.y, n1 = p2.x, n2 = p2.y;
    const double b0 = p3.x, b1 = p3.y, b2 = p4.x;
    const double t0 = p4.y, t1 = p5.x, t2 = p5.y;
    const double ir = rsqrt_h3(fma(rx, rx, fma(ry, ry, rz * rz)));
    const double a0 = rx * ir, a1 = ry * ir, a2 = rz * ir;
    const double rdn = fma(a0, n0, fma(a1, n1, a2 * n2));
    const double rdu = fma(a0, b0, fma(a1, b1, a2 * b2));
    const double rdt = fma(a0, t0, fma(a1, t1, a2 * t2));
    const double nuv = p6.x + p6.y + p7.x;
    const double ir2 = ir * ir, ir3 = ir2 * ir;
    const double fD = K.cD * ir2, fS = K.cS * ir3;
    const double q = K.cDc6 * ir2, fS6 = K.cSc6 * ir3, z = K.cS3nu * ir3;
    const double h = rdn * rdu;
    // displacement
    const double g1 = K.cU4 * ir;
    const double g2 = fma(fD, fma(3.0, h, K.asgc6 * nuv), (K.cU * ir) * rdt);
    const double g3 = q * rdn, g4 = (K.asg * q) * rdu;
    u[0] = fma(g1, t0, fma(g2, a0, fma(g3, b0, fma(g4, n0, u[0]))));
    u[1] = fma(g1, t1, fma(g2, a1, fma(g3, b1, fma(g4, n1, u[1]))));
    u[2] = fma(g1, t2, fma(g2, a2, fma(g3, b2, fma(g4, n2, u[2]))));
    // stress
    const double p_b = z * rdn, p_n = z * rdu;
    const double x1 = fD * rdt, x2 = fS * h, x4 = fS * nuv;
    const double al = fma(7.5, x2, fma(1.5, x1, K.k15c6 * x4));
    tr = fma(K.mc6, x1, fma(K.m3c6, x2, fma(K.pr4, x4, tr)));
    const double w0 = fma(q, t0, fma(p_b, b0, fma(p_n, n0, al * a0)));
    const double w1 = fma(q, t1, fma(p_b, b1, fma(p_n, n1, al * a1)));
    const double w2 = fma(q, t2, fma(p_b, b2, fma(p_n, n2, al * a2)));
    d[0] = fma(a0, w0, fma(-fS6, p6.x, d[0]));
    d[1] = fma(a1, w1, fma(-fS6, p6.y, d[1]));
    d[2] = fma(a2, w2, fma(-fS6, p7.x, d[2]));
    o[0] = fma(a0, w1, fma(a1, w0, fma(-fS6, p7.y, o[0])));
    o[1] = fma(a1, w2, fma(a2, w1, fma(-fS6, p8.x, o[1])));
    o[2] = fma(a2, w0, fma(a0, w2, fma(-fS6, p8.y, o[2])));
  }

  // value c of u (3), sigma (xx, yy, zz, xy, yz, zx)
  __device__ __forceinline__ double value(int c) const {
    if (c < 3) return u[c];
    return c < 6 ? fma(2.0, d[c - 3], tr) : o[c - 6];
  }
};

static SomConst som_const(const Material& m, int flags) {
  const double nu = m.nu, mu = m.mu, c6 = 1.0 - 2.0 * nu, asg = (flags & BEM_IP_KELVIN_CONSISTENT) ? -1.0 : 1.0;
  SomConst K;
  K.cD = 1.0 / (8.0 * kPi * (1.0 - nu));
  K.cU = 1.0 / (16.0 * kPi * (1.0 - nu) * mu);
  K.cU4 = K.cU * (3.0 - 4.0 * nu);
  K.cDc6 = K.cD * c6;
  K.cS = mu / (4.0 * kPi * (1.0 - nu));
  K.cS3nu = -3.0 * nu * K.cS;
  K.cSc6 = K.cS * c6;
  K.m3c6 = -3.0 * c6;
  K.mc6 = -c6;
  K.k15c6 = -1.5 * c6;
  K.pr4 = 1.0 - 4.0 * nu;
  K.asg = -asg;
  K.asgc6 = asg * c6;
  return K;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem)
               : "memory");
}

constexpr int kFarThreads = 256;
constexpr int kChunkDoubles = kChunk * kGp * kRec;  // one staged chunk of element tables

// Far pass: CTA (x, y) sums the element chunks [nchunks y / S, nchunks (y + 1) / S) of S =
// gridDim.y shares at the points [256 x, 256 (x + 1)), one per thread, into part[y][9][l].
// The shares give a call with few points enough CTAs (a single tile alone fills one SM)
// and even out the last wave.  Bound: FP64 pipe, 83 % active (16 warps per SM at 126
// registers).  100,003 points x 960 elements: 49.6 -> 21.2 ms by SomAcc::add; 3,001 points x
// 484 elements: 8.3 -> 0.35 ms, the rest by the shares.  counters[0] accumulates the table points evaluated (far
// Gauss points x internal points).
__global__ void __launch_bounds__(kFarThreads, 2)
    far_kernel(int l, const double* __restrict__ cx, const double* __restrict__ cy, const double* __restrict__ cz,
               int ne, const int* __restrict__ nconec, const double* __restrict__ einfo,
               const double* __restrict__ far, SomConst K, double* __restrict__ part, unsigned long long* counters) {
  __shared__ __align__(16) double s_tab[2][kChunkDoubles];
  __shared__ __align__(16) double s_info[2][kChunk][4];
  __shared__ int s_npt[2][kChunk];
  const int tid = threadIdx.x;
  const int nchunks = (ne + kChunk - 1) / kChunk;
  const int ch0 = (int)((int64_t)nchunks * blockIdx.y / gridDim.y);
  const int ch1 = (int)((int64_t)nchunks * (blockIdx.y + 1) / gridDim.y);
  const int ip = blockIdx.x * kFarThreads + tid;
  const bool act = ip < l;
  const double xx = act ? cx[ip] : 0.0, yy = act ? cy[ip] : 0.0, zz = act ? cz[ip] : 0.0;
  SomAcc acc;
  unsigned long long evals = 0;
  auto stage = [&](int ch, int buf) {  // issue the copies of chunk ch into buffer buf
    const int e0 = ch * kChunk, ce = min(kChunk, ne - e0);
    const double* src = far + (int64_t)e0 * kGp * kRec;
    double* dst = s_tab[buf];
    for (int i = tid; i < ce * kGp * kRec / 2; i += kFarThreads) cp_async16(dst + 2 * i, src + 2 * i);
    const double* isrc = einfo + 4 * (int64_t)e0;
    if (tid < ce * 2) cp_async16(&s_info[buf][0][0] + 2 * tid, isrc + 2 * tid);
    if (tid < ce) s_npt[buf][tid] = (nconec[e0 + tid] == 9) ? 36 : 16;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (ch0 < ch1) stage(ch0, 0);
  for (int ch = ch0; ch < ch1; ++ch) {
    const int buf = (ch - ch0) & 1;
    if (ch + 1 < ch1) {
      stage(ch + 1, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int ce = min(kChunk, ne - ch * kChunk);
    for (int ee = 0; ee < ce; ++ee) {
      const double* inf = s_info[buf][ee];
      const double dx = xx - inf[0], dy = yy - inf[1], dz = zz - inf[2];
      if (!act || !(dx * dx + dy * dy + dz * dz > inf[3])) continue;
      const int np = s_npt[buf][ee];
      const double* Pt = s_tab[buf] + ee * kGp * kRec;
#pragma unroll 2
      for (int q = 0; q < np; ++q) acc.add(K, Pt + q * kRec, xx, yy, zz);
      evals += (unsigned long long)np;
    }
    __syncthreads();  // buffer buf is refilled by the next iteration's stage
  }
  if (act)
#pragma unroll
    for (int c = 0; c < 9; ++c) part[((int64_t)blockIdx.y * 9 + c) * l + ip] = acc.value(c);
  // one addition per warp
  for (int off = 16; off > 0; off >>= 1) evals += __shfl_xor_sync(0xffffffffu, evals, off);
  if ((tid & 31) == 0 && evals) atomicAdd(counters, evals);
}

// ---- near pairs ----------------------------------------------------------------------
// A point and an element whose centroid lies within the near radius form a pair.  Pairs are
// numbered point by point, elements ascending, so that finish_kernel adds a point's pairs
// in a fixed order; elist lists them by element for near_kernel.

constexpr int kNearThreads = 256;

// One warp per point: the lanes test 32 elements at a time, f(e, near) with e ascending from
// lane to lane (near = false past the last element).  A thread per point needed the whole
// element list one after the other, which with a few thousand points left most SMs idle
// (0.24 ms for the lists of 3,001 points and 484 elements).
template <typename F>
__device__ __forceinline__ void for_near(int ip, const double* cx, const double* cy, const double* cz, int ne,
                                         const double* einfo, F f) {
  const double xx = __ldg(cx + ip), yy = __ldg(cy + ip), zz = __ldg(cz + ip);
  for (int e0 = 0; e0 < ne; e0 += 32) {
    const int e = e0 + (threadIdx.x & 31);
    bool near = false;
    if (e < ne) {
      const double2 i0 = __ldg(reinterpret_cast<const double2*>(einfo) + 2 * (int64_t)e);
      const double2 i1 = __ldg(reinterpret_cast<const double2*>(einfo) + 2 * (int64_t)e + 1);
      const double dx = xx - i0.x, dy = yy - i0.y, dz = zz - i1.x;
      near = !(dx * dx + dy * dy + dz * dz > i1.y);
    }
    f(e, near);
  }
}

// pairs of every point (pcnt) and of every element (ecnt, zeroed by the caller)
__global__ void __launch_bounds__(kNearThreads)
    near_count_kernel(int l, const double* __restrict__ cx, const double* __restrict__ cy,
                      const double* __restrict__ cz, int ne, const double* __restrict__ einfo, int* pcnt, int* ecnt) {
  const int ip = (int)(((int64_t)blockIdx.x * kNearThreads + threadIdx.x) >> 5);
  if (ip >= l) return;
  int cnt = 0;
  for_near(ip, cx, cy, cz, ne, einfo, [&](int e, bool near) {
    cnt += __popc(__ballot_sync(0xffffffffu, near));
    if (near) atomicAdd(ecnt + e, 1);
  });
  if ((threadIdx.x & 31) == 0) pcnt[ip] = cnt;
}

// Exclusive sums: pair offsets of the points (poff, l + 1) and of the elements (eoff, ne +
// 1), work items of the elements (ioff, ne + 1; one per kNearThreads pairs).  tot: pairs,
// items, points with a pair.  One CTA of 1024 threads.
__device__ __forceinline__ long long block_exclusive(long long v, long long* s_w, long long& total) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  long long x = v;
  for (int off = 1; off < 32; off <<= 1) {
    const long long o = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += o;
  }
  if (lane == 31) s_w[wp] = x;
  __syncthreads();
  if (wp == 0) {
    long long y = s_w[lane];
    for (int off = 1; off < 32; off <<= 1) {
      const long long o = __shfl_up_sync(0xffffffffu, y, off);
      if (lane >= off) y += o;
    }
    s_w[lane] = y;
  }
  __syncthreads();
  const long long base = wp ? s_w[wp - 1] : 0;
  total = s_w[31];
  __syncthreads();
  return base + x - v;
}

__global__ void __launch_bounds__(1024) near_scan_kernel(int l, const int* pcnt, long long* poff, int ne,
                                                         const int* ecnt, long long* eoff, int* ioff, long long* tot) {
  __shared__ long long s_w[32];
  const int tid = threadIdx.x;
  long long run = 0, total, nearp = 0;
  for (int i0 = 0; i0 < l; i0 += 4 * 1024) {
    int v[4];
    long long sum = 0;
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + 4 * tid + u;
      v[u] = i < l ? pcnt[i] : 0;
      sum += v[u];
      nearp += v[u] > 0;
    }
    long long at = run + block_exclusive(sum, s_w, total);
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + 4 * tid + u;
      if (i < l) poff[i] = at;
      at += v[u];
    }
    run += total;
  }
  block_exclusive(nearp, s_w, total);
  if (tid == 0) {
    poff[l] = run;
    tot[0] = run;
    tot[2] = total;
  }
  long long erun = 0, irun = 0;
  for (int e0 = 0; e0 < ne; e0 += 1024) {
    const int e = e0 + tid, v = e < ne ? ecnt[e] : 0;
    const long long at = erun + block_exclusive(v, s_w, total);
    erun += total;
    const long long it = irun + block_exclusive((v + kNearThreads - 1) / kNearThreads, s_w, total);
    irun += total;
    if (e < ne) {
      eoff[e] = at;
      ioff[e] = (int)it;
    }
  }
  if (tid == 0) {
    eoff[ne] = erun;
    ioff[ne] = (int)irun;
    tot[1] = irun;
  }
}

// the pairs' points (pt) and the elements' pair lists (elist; the order within a list is
// that of the atomics, which no result depends on); cur: ne zeros
__global__ void __launch_bounds__(kNearThreads)
    near_fill_kernel(int l, const double* __restrict__ cx, const double* __restrict__ cy,
                     const double* __restrict__ cz, int ne, const double* __restrict__ einfo,
                     const long long* __restrict__ poff, const long long* __restrict__ eoff, int* cur, int* pt,
                     int* elist) {
  const int ip = (int)(((int64_t)blockIdx.x * kNearThreads + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (ip >= l) return;
  long long j0 = poff[ip];
  for_near(ip, cx, cy, cz, ne, einfo, [&](int e, bool near) {
    const unsigned b = __ballot_sync(0xffffffffu, near);
    if (near) {
      const long long j = j0 + __popc(b & ((1u << lane) - 1));
      pt[j] = ip;
      elist[eoff[e] + atomicAdd(cur + e, 1)] = (int)j;
    }
    j0 += __popc(b);
  });
}

// Near pass: work item (element, up to 256 of its pairs).  The CTA's 8 warps take the item's
// pairs in groups of 32, one per lane; an element with fewer than 5 groups has 2, 4 or 8
// warps share a group, each over its slice of the 1600 points (as many for all items of an
// element, so that a pair's sums do not depend on its place in the list), and their sums
// meet in shared memory.  The table streams through shared memory in chunks of 160 points
// (160 / slices of every slice) and is read as broadcasts: one warp per point read 96 B
// records lane by lane and was bound by that: 103 -> 33.7 ms for 100,003 points of a plate of
// 960 elements, now at the FP64 pipe (82 % active).
constexpr int kNearChunk = 160;
constexpr int kNearChunks = kNear / kNearChunk;
constexpr size_t kNearSmem = 2 * (size_t)kNearChunk * kRec * sizeof(double);

__global__ void __launch_bounds__(kNearThreads, 2)
    near_kernel(int nitems, const double* __restrict__ cx, const double* __restrict__ cy,
                const double* __restrict__ cz, int ne, const double* __restrict__ near, SomConst K,
                const int* __restrict__ ioff, const long long* __restrict__ eoff, const int* __restrict__ elist,
                const int* __restrict__ pt, double* __restrict__ acc_out) {
  extern __shared__ __align__(16) double s_near[];  // [2][kNearChunk][kRec], then the slices' sums
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int item = blockIdx.x;
  int lo = 0, hi = ne - 1;  // largest e with ioff[e] <= item: the item's element
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(ioff + mid) <= item) lo = mid;
    else hi = mid - 1;
  }
  const int e = lo;
  const long long p0 = __ldg(eoff + e), p1 = __ldg(eoff + e + 1);
  const int cnt = (int)min((long long)kNearThreads, p1 - p0);  // pairs of the element's fullest item
  const int slices = cnt > 128 ? 1 : cnt > 64 ? 2 : cnt > 32 ? 4 : 8;
  const int ngrp = 8 / slices, grp = w % ngrp, sl = w / ngrp;
  const long long mine = p0 + (long long)(item - __ldg(ioff + e)) * kNearThreads + 32 * grp + lane;
  const bool act = mine < p1;
  const int j = act ? __ldg(elist + mine) : 0;
  const int ip = act ? __ldg(pt + j) : 0;
  const double xx = cx[ip], yy = cy[ip], zz = cz[ip];
  const bool any = __any_sync(0xffffffffu, act);
  const double* T = near + (int64_t)e * kNear * kRec;
  const int per = kNearChunk / slices;  // points of a slice in a chunk
  auto stage = [&](int ch, int buf) {
    for (int i = tid; i < kNearChunk * kRec / 2; i += kNearThreads) {
      const int r = i / (kRec / 2), o = i % (kRec / 2);
      const int q = (r / per) * (kNear / slices) + ch * per + r % per;
      cp_async16(s_near + (size_t)buf * kNearChunk * kRec + 2 * i, T + (int64_t)q * kRec + 2 * o);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  SomAcc acc;
  stage(0, 0);
  for (int ch = 0; ch < kNearChunks; ++ch) {
    const int buf = ch & 1;
    if (ch + 1 < kNearChunks) {
      stage(ch + 1, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (any) {
      const double* Pt = s_near + ((size_t)buf * kNearChunk + sl * per) * kRec;
#pragma unroll 2
      for (int q = 0; q < per; ++q) acc.add(K, Pt + q * kRec, xx, yy, zz);
    }
    __syncthreads();  // buffer buf is refilled next
  }
  if (slices > 1) {
    double* s_sum = s_near + (size_t)(w * 32 + lane) * 9;
#pragma unroll
    for (int c = 0; c < 9; ++c) s_sum[c] = acc.value(c);
    __syncthreads();
    if (sl == 0 && act)
      for (int c = 0; c < 9; ++c) {
        double v = 0.0;
        for (int s = 0; s < slices; ++s) v += s_near[(size_t)((grp + s * ngrp) * 32 + lane) * 9 + c];
        acc_out[(int64_t)j * 9 + c] = v;
      }
  } else if (act) {
#pragma unroll
    for (int c = 0; c < 9; ++c) acc_out[(int64_t)j * 9 + c] = acc.value(c);
  }
}

// A point's far shares and near pairs added in their order, and its principal stresses:
// warp c of a CTA adds component c of 32 points.
__global__ void __launch_bounds__(9 * 32)
    finish_kernel(int l, int shares, const double* __restrict__ part, const long long* __restrict__ poff,
                  const double* __restrict__ pairs, double* u, double* s, double* pr, double* vm) {
  __shared__ double s_v[9][33];
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ip = (int64_t)blockIdx.x * 32 + lane;
  if (ip < l) {
    double v = 0.0;
#pragma unroll 8
    for (int y = 0; y < shares; ++y) v += part[((int64_t)y * 9 + c) * l + ip];
    const long long j1 = poff[ip + 1];
#pragma unroll 4
    for (long long j = poff[ip]; j < j1; ++j) v += pairs[j * 9 + c];
    if (c < 3) u[3 * ip + c] = v;
    else s[6 * ip + c - 3] = v;
    s_v[c][lane] = v;
  }
  __syncthreads();
  if (c == 0 && ip < l) {
    double t[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) t[k] = s_v[3 + k][lane];
    principal_vm(t, pr + 3 * ip, vm + ip);
  }
}

// pairs evaluated at a time (their sums and lists take 80 B each)
constexpr long long kMaxPairs = 24LL << 20;

static cudaError_t at_least(DBuf<unsigned char>& b, size_t bytes) {
  return b.count >= bytes ? cudaSuccess : b.alloc(bytes);
}

// the tables and the workspace of a call, in the context's ip_ws
struct IpTables {
  const double *einfo, *far, *near;
  unsigned char* scratch;
  unsigned long long* counters;
};

// far-pass shares of l points: enough CTAs for eight waves of two CTAs per SM, as far as
// the elements go and the partial sums stay below 128 MB (one share above 1.8 M points)
static int far_shares(const bem_ctx* c, int l) {
  const int tiles = (l + kFarThreads - 1) / kFarThreads;
  const int nchunks = (c->ne + kChunk - 1) / kChunk;
  const int64_t want = (16LL * c->sm_count + tiles - 1) / tiles;
  const int64_t room = std::max<int64_t>(1, (int64_t)(size_t(128) << 20) / (72 * (int64_t)l));
  return (int)std::max<int64_t>(1, std::min({want, room, (int64_t)nchunks}));
}

static size_t up256(size_t b) { return (b + 255) / 256 * 256; }
static size_t scratch_bytes(const bem_ctx* c, int l) {
  return up256(sizeof(double) * 9 * (size_t)l * far_shares(c, l)) + up256(sizeof(long long) * ((size_t)l + 1)) +
         up256(sizeof(int) * (size_t)l);
}

// l points.  A range with more near pairs than kMaxPairs, or than there is memory for, is
// taken in two halves; the far shares are the whole call's.
static int run_points(bem_ctx* c, const IpTables& T, const SomConst& K, int shares, int l, const double* cx, const double* cy,
                      const double* cz, double* u, double* s, double* pr, double* vm) {
  const int ne = c->ne;
  unsigned char* p = T.scratch;
  double* part = reinterpret_cast<double*>(p);
  p += up256(sizeof(double) * 9 * (size_t)l * shares);
  long long* poff = reinterpret_cast<long long*>(p);
  p += up256(sizeof(long long) * ((size_t)l + 1));
  int* pcnt = reinterpret_cast<int*>(p);
  // counters: far evaluations; pairs, items, near points; then the elements' arrays
  long long* tot = reinterpret_cast<long long*>(T.counters) + 1;
  long long* eoff = tot + 3;
  int* ioff = reinterpret_cast<int*>(eoff + ne + 1);
  int *ecnt = ioff + ne + 1, *cur = ecnt + ne;
  BEM_CUDA(c, cudaMemsetAsync(ecnt, 0, 2 * (size_t)ne * sizeof(int), c->stream));
  const int blocks = (int)((32 * (int64_t)l + kNearThreads - 1) / kNearThreads);
  near_count_kernel<<<blocks, kNearThreads, 0, c->stream>>>(l, cx, cy, cz, ne, T.einfo, pcnt, ecnt);
  BEM_LAUNCH_CHECK(c);
  near_scan_kernel<<<1, 1024, 0, c->stream>>>(l, pcnt, poff, ne, ecnt, eoff, ioff, tot);
  BEM_LAUNCH_CHECK(c);
  long long ht[3];
  BEM_CUDA(c, cudaMemcpyAsync(ht, tot, sizeof(ht), cudaMemcpyDeviceToHost, c->stream));
  BEM_CUDA(c, cudaStreamSynchronize(c->stream));
  const long long npairs = ht[0];
  const int nitems = (int)ht[1];
  const size_t sums = up256(sizeof(double) * 9 * (size_t)npairs), list = up256(sizeof(int) * (size_t)npairs);
  const bool room = npairs <= kMaxPairs && (npairs == 0 || at_least(c->ip_pairs, sums + 2 * list) == cudaSuccess);
  if (!room) {
    cudaGetLastError();  // a failed allocation: fewer points at a time
    if (l == 1) return bem_fail(c, BEM_ERR_OOM, "allocating the near pairs of the internal points");
    const int h = l / 2;
    int rc = run_points(c, T, K, shares, h, cx, cy, cz, u, s, pr, vm);
    if (rc) return rc;
    return run_points(c, T, K, shares, l - h, cx + h, cy + h, cz + h, u + 3 * (int64_t)h, s + 6 * (int64_t)h,
                      pr + 3 * (int64_t)h, vm + h);
  }
  double* pairs = nullptr;
  if (npairs > 0) {
    pairs = reinterpret_cast<double*>(c->ip_pairs.p);
    int* elist = reinterpret_cast<int*>(c->ip_pairs.p + sums);
    int* pt = reinterpret_cast<int*>(c->ip_pairs.p + sums + list);
    near_fill_kernel<<<blocks, kNearThreads, 0, c->stream>>>(l, cx, cy, cz, ne, T.einfo, poff, eoff, cur, pt, elist);
    BEM_LAUNCH_CHECK(c);
    near_kernel<<<nitems, kNearThreads, kNearSmem, c->stream>>>(nitems, cx, cy, cz, ne, T.near, K, ioff, eoff, elist,
                                                                pt, pairs);
    BEM_LAUNCH_CHECK(c);
  }
  far_kernel<<<dim3((l + kFarThreads - 1) / kFarThreads, shares), kFarThreads, 0, c->stream>>>(
      l, cx, cy, cz, ne, c->nconec.p, T.einfo, T.far, K, part, T.counters);
  BEM_LAUNCH_CHECK(c);
  finish_kernel<<<(l + 31) / 32, 9 * 32, 0, c->stream>>>(l, shares, part, poff, pairs, u, s, pr, vm);
  BEM_LAUNCH_CHECK(c);
  c->prof.ip_near_points += ht[2];
  c->prof.ip_near_evals += (double)npairs * kNear;
  return BEM_OK;
}

int launch_internal_points(bem_ctx* c, int l, const double* cx, const double* cy, const double* cz, double* u,
                           double* s, double* pr, double* vm, int flags) {
  if (!c->have_geometry || c->DFI.count == 0 || c->U.count == 0)
    return bem_fail(c, BEM_ERR_STATE, "internal_points needs geometry and a reorganized solution");
  NearRule rule;
  gauss_legendre(kNearN, rule.x, rule.w);
  const int ne = c->ne;
  // one buffer: tables, element arrays and counters, the points' workspace
  const size_t b_info = up256(sizeof(double) * 4 * (size_t)ne), b_far = up256(sizeof(double) * kRec * kGp * (size_t)ne),
               b_near = up256(sizeof(double) * kRec * kNear * (size_t)ne),
               b_cnt = up256(8 * (4 + (size_t)ne + 1) + 4 * (3 * (size_t)ne + 1));
  if (at_least(c->ip_ws, b_info + b_far + b_near + b_cnt + scratch_bytes(c, l)) != cudaSuccess)
    return bem_fail(c, BEM_ERR_OOM, "allocating the internal points' tables and workspace");
  unsigned char* p = c->ip_ws.p;
  double* einfo = reinterpret_cast<double*>(p);
  double* far = reinterpret_cast<double*>(p += b_info);
  double* near = reinterpret_cast<double*>(p += b_far);
  IpTables T;
  T.counters = reinterpret_cast<unsigned long long*>(p += b_near);
  T.scratch = p + b_cnt;
  T.einfo = einfo;
  T.far = far;
  T.near = near;
  BEM_CUDA(c, cudaMemsetAsync(T.counters, 0, sizeof(unsigned long long), c->stream));
  einfo_kernel<<<(ne + 127) / 128, 128, 0, c->stream>>>(ne, c->x.p, c->y.p, c->z.p, c->nconec.p, c->kconec.p, einfo);
  BEM_LAUNCH_CHECK(c);
  const int64_t nf = (int64_t)ne * kGp;
  far_table_kernel<<<(unsigned)((nf + 127) / 128), 128, 0, c->stream>>>(
      ne, c->nconec.p, c->kconec.p, c->eta1.p, c->eta2.p, c->eta3.p, c->xja.p, c->xg1.p, c->xg2.p, c->xg3.p,
      c->ff.p, c->U.p, c->DFI.p, far);
  BEM_LAUNCH_CHECK(c);
  const int64_t nn = (int64_t)ne * kNear;
  near_table_kernel<<<(unsigned)((nn + 127) / 128), 128, 0, c->stream>>>(ne, c->x.p, c->y.p, c->z.p, c->nconec.p,
                                                                          c->kconec.p, c->U.p, c->DFI.p, rule, near);
  BEM_LAUNCH_CHECK(c);
  int rc = run_points(c, T, som_const(c->mat, flags), far_shares(c, l), l, cx, cy, cz, u, s, pr, vm);
  unsigned long long cnt = 0;
  if (rc == BEM_OK) {
    BEM_CUDA(c, cudaMemcpyAsync(&cnt, T.counters, sizeof(cnt), cudaMemcpyDeviceToHost, c->stream));
    BEM_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  // cudaFree waits for the work that uses the buffer
  if (c->ip_ws.count > kWsKeep) c->ip_ws.release();
  if (c->ip_pairs.count > kWsKeep) c->ip_pairs.release();
  if (rc) return rc;
  c->prof.ip_points += l;
  c->prof.ip_far_evals += (double)cnt;
  return BEM_OK;
}

}  // namespace bem
