// Device-side description of the systems of a batch, shared by batch.cu (assembly, host
// side) and batch_lu.cu (factorisation and solve).
#pragma once

#include "common.cuh"

namespace bem {

constexpr int kMaxRhs = 8;  // load cases per system
constexpr int kMaxOrder = 25600;  // of a system: its pivots and their gather fit in shared memory

struct SysDev {
  int n, ne, N, nrhs;
  int64_t lda;   // of H / A and of the factor copy
  int64_t ldg;   // of G
  int64_t a_off, g_off, f_off;  // A (FP64), G (FP64), factor (T) in their arenas
  int64_t v_off;                // FI, X, R: N x nrhs each (ld N) in the vector arena
  int64_t piv_off;              // pivots, the row gather and the solve's rows (N each)
  int64_t inv_off;              // diagonal-block inverses: 128-row block index of the first
  int64_t cs_off, ncs;          // column-swap list: (dof, G column) pairs
  int64_t fl_off, nfl;          // FI terms: (matrix, column) and nrhs coefficients each
  int64_t pin_off, npins;
  int64_t uk_off;               // u known per dof
  double mu;
};

// What the solve of a batch works on.
struct BatchSolve {
  cudaStream_t stream;
  int sm_count;
  const SysDev* sys;   // device
  const int* order;    // device: systems by decreasing order N
  std::vector<int> N;  // orders, decreasing
  const double* A;     // FP64 systems
  double *FI, *X, *R;  // right-hand sides, solutions, residuals
  double* W;           // [total rows][kMaxRhs]: the sweeps' vectors
  double* dinv;        // two 128 x 128 inverses per 128-row diagonal block
  double* red;         // [systems][3 kMaxRhs + 1] maxima of the residual pass
  double* berr;        // per system
  int *piv, *perm;     // per row
  int *info, *conv;    // per system
  int* moved;          // [systems][64]: the interchanges of the current panel
  int* err;            // one error word
  unsigned long long wait_ns;  // limit of the panels' waits
  int withhold_pivot;  // BEM_OPT_WITHHOLD_PIVOT
  int nsys;
  long long launches;  // counted by the calls below
};

// The whole solve, enqueued on the stream without host synchronisation: LU of F (T: FP32 or
// FP64, row pivoting, LAPACK's dgetrf), then either one solve (sweeps = 0) or `sweeps` steps of
// FP64 refinement from zero that a system leaves once its backward error is <= tol or gains
// less than 10 %.  Returns false when a launch failed.
template <typename T>
bool batch_solve_enqueue(BatchSolve& b, T* F, double tol, int sweeps);
// largest order whose LU runs panel by panel over all systems (0: none on this device)
template <typename T>
int batch_lu_max_order();

}  // namespace bem
