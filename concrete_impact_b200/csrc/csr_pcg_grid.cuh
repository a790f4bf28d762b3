// Jacobi-PCG of one or six right-hand sides in a single persistent launch (csr_pcg_grid.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cib {

constexpr int PCG_BLOCK_RHS = 6;  // right-hand sides of a block solve

struct CsrSystem {
  int64_t n;
  const int64_t* indptr;
  const int64_t* indices;
  const double* values;
  const uint8_t* free_mask;
  const double* dinv;
};

constexpr int PCG_GRID_MAX = 160;  // CTAs of a persistent solve
constexpr int PCG_GRID_DOTS = 5;

// Doubles of the partial sums and sums; results of a solve.
constexpr int pcg_grid_part(int rhs) { return 2 * PCG_GRID_DOTS * rhs * (PCG_GRID_MAX + 1); }
constexpr int pcg_grid_out(int rhs) { return 3 * rhs + 1; }

struct PcgGridWork {
  double *zlo, *zhi;  // rhs * n each
  double* part;       // pcg_grid_part(rhs), or rhs * n
  double* out;        // pcg_grid_out(rhs)
};

// Solves rhs = 1 or PCG_BLOCK_RHS systems A x_j = b_j (rows j of b and x).  Returns CIB_OK with
// status (0 converged, 1 iteration limit, 2 breakdown), iterations and relative residuals of
// each, CIB_ERANGE when the persistent launch does not take the system (the caller then solves
// it with a launch per phase), CIB_ECUDA.
int csr_pcg_grid(const CsrSystem& a, int rhs, const double* b, double* x, const PcgGridWork& w, double rtol,
                 int32_t maxit, int32_t* status, int32_t* iterations, double* relative_residual, cudaStream_t st);

}  // namespace cib
