// Driver for tests/test_profile_waits.py: one factorisation and solve of a CSR
// system with a given limit on the waits between its blocks.
#include <cuda_runtime.h>

#include "../../xara_gb300/csrc/xg_internal.h"

extern "C" int solve_with_limit(int n, const int *rowptr, const int *colidx, const double *vals,
                                const double *b, double *x, double wait_ms) {
  const size_t nnz = rowptr[n];
  int *rp, *ci;
  double *v, *db, *dx;
  if (cudaMalloc(&rp, (n + 1) * sizeof(int)) || cudaMalloc(&ci, nnz * sizeof(int)) ||
      cudaMalloc(&v, nnz * sizeof(double)) || cudaMalloc(&db, n * sizeof(double)) ||
      cudaMalloc(&dx, n * sizeof(double)))
    return -100;
  cudaMemcpy(rp, rowptr, (n + 1) * sizeof(int), cudaMemcpyHostToDevice);
  cudaMemcpy(ci, colidx, nnz * sizeof(int), cudaMemcpyHostToDevice);
  cudaMemcpy(v, vals, nnz * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, n * sizeof(double), cudaMemcpyHostToDevice);
  cudaStream_t s;
  cudaStreamCreate(&s);
  int e;
  {
    xg::ProfileSolver P;
    e = P.setup(n, rowptr, colidx, rp, ci, v, s);
    xg::ProfileSystem S = P.system();
    S.wait_ns = (unsigned long long)(wait_ms * 1e6);
    S.fwd_nrhs = 1;
    S.b[0] = db;
    S.x[0] = dx;
    if (!e) e = xg::profile_factor(S, s);
    if (!e) e = xg::profile_solve(S, 1, s, true);
    if (!e) e = xg::profile_status(S, s, nullptr);
    cudaMemcpy(x, dx, n * sizeof(double), cudaMemcpyDeviceToHost);
  }
  cudaStreamDestroy(s);
  for (void *p : {(void *)rp, (void *)ci, (void *)v, (void *)db, (void *)dx}) cudaFree(p);
  return e;
}
