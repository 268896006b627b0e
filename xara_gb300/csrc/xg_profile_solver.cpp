// xg_profile_solver.cpp -- the buffers and call sequence of the tiled
// envelope LDL' (xg_profile.cu): `system ProfileSPD` on the device,
// ProfileSPDLinDirectSolver::factor / solve
// (system_of_eqn/linearSOE/profileSPD/ProfileSPDLinDirectSolver.cpp:100-420)
// for the device model and for the standalone linear system.
#include <cuda_runtime.h>

#include <cstdio>
#include <vector>

#include "xg_internal.h"

namespace xg {

template <class T>
int ProfileSolver::Buf<T>::alloc(size_t count) {
  if (p) cudaFree(p);
  p = nullptr;
  if (count == 0) count = 1;
  return cudaMalloc(&p, count * sizeof(T)) == cudaSuccess ? 0 : XG_ENOMEM;
}

template <class T>
ProfileSolver::Buf<T>::~Buf() {
  if (p) cudaFree(p);
}

ProfileSolver::~ProfileSolver() = default;

int ProfileSolver::setup(int n, const int *rowptr, const int *colidx, const int *d_rowptr,
                         const int *d_colidx, const double *d_vals, cudaStream_t s) {
  ready_ = false;
  std::vector<int> ftile;
  int nt = 0, W = 0;
  if (int e = profile_plan(n, rowptr, colidx, ftile, nt, W)) return e;
  const size_t tiles = profile_tile_doubles(nt, W);
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
    record_error("ProfileSPD: cudaMemGetInfo failed");
    return XG_ECUDA;
  }
  int sms = 0;
  if (profile_device(&sms) != 0) {
    record_error("ProfileSPD: the device refuses the factorisation's shared memory");
    return XG_ECUDA;
  }
  const size_t dig = profile_digit_bytes(W);
  if ((tiles + (size_t)nt * 32 * 6) * sizeof(double) > free_b / 2) {
    char msg[160];
    snprintf(msg, sizeof msg,
             "ProfileSPD envelope needs %.1f GB (%d tile rows x %d): use the block-Jacobi PCG "
             "system", tiles * 8e-9, nt, W + 1);
    record_error(msg);
    return XG_ENOMEM;
  }
  std::vector<int> tasks, npairs;
  std::vector<int> rows, next, slot_row;   // first columns, then next rows, then the slots
  const int blocks = profile_rows(nt, ftile, sms, rows, next, slot_row);
  if (blocks > sms) {
    char msg[160];
    snprintf(msg, sizeof msg, "ProfileSPD: the factorisation needs %d SMs, the device has %d",
             blocks, sms);
    record_error(msg);
    return XG_ECUDA;
  }
  profile_tasks(nt, W, ftile, rows, tasks, npairs);
  rows.insert(rows.end(), next.begin(), next.end());
  rows.insert(rows.end(), slot_row.begin(), slot_row.end());
  const size_t nrow = (size_t)nt * 1024, nslot = (size_t)nt * (W + 1);
  // flags, task counter and tickets, then the per-tile and per-row counters
  const size_t ncount = 8 + 2 * nslot + 4 * (size_t)nt;
  int e = 0;
  e |= ftile_.alloc(ftile.size()) | tasks_.alloc(tasks.size()) | npairs_.alloc(npairs.size());
  e |= rows_.alloc(rows.size());
  e |= counters_.alloc(ncount) | dig_.alloc(dig) | stream_.alloc(5 * nrow);
  e |= L_.alloc(tiles) | Winv_.alloc(nrow) | F_.alloc(nrow) | G_.alloc(nrow);
  e |= E_.alloc(nrow) | H_.alloc(nrow) | Q_.alloc(nrow) | R_.alloc(nrow);
  e |= invD_.alloc((size_t)nt * 32) | piv_.alloc((size_t)nt * 32);
  e |= sweep_.alloc(4 * 4 * (size_t)nt * 32);
  if (e) {
    record_error("ProfileSPD: device allocation failed");
    return XG_ENOMEM;
  }
  if (cudaMemcpyAsync(ftile_.p, ftile.data(), ftile.size() * sizeof(int),
                      cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(tasks_.p, tasks.data(), tasks.size() * sizeof(int), cudaMemcpyHostToDevice,
                      s) != cudaSuccess ||
      cudaMemcpyAsync(rows_.p, rows.data(), rows.size() * sizeof(int), cudaMemcpyHostToDevice, s) !=
          cudaSuccess ||
      cudaMemcpyAsync(npairs_.p, npairs.data(), npairs.size() * sizeof(int),
                      cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    record_error("ProfileSPD: set-up copies failed");
    return XG_ECUDA;
  }
  S_ = ProfileSystem{};
  S_.n = n; S_.nt = nt; S_.W = W;
  S_.rowptr = d_rowptr; S_.colidx = d_colidx; S_.vals = d_vals;
  S_.ftile = ftile_.p; S_.L = L_.p; S_.invD = invD_.p; S_.piv = piv_.p;
  S_.Winv = Winv_.p; S_.F = F_.p; S_.G = G_.p;
  S_.E = E_.p; S_.H = H_.p; S_.Q = Q_.p; S_.R = R_.p;
  S_.sweep = sweep_.p;
  S_.tasks = reinterpret_cast<const int4 *>(tasks_.p);
  S_.ntasks = (int)(tasks.size() / 4);
  S_.flags = counters_.p; S_.next_task = S_.flags + 4;
  S_.upd = S_.flags + 8; S_.done = S_.upd + nslot;
  S_.cpl = S_.done + nslot; S_.cplq = S_.cpl + nt; S_.colcnt = S_.cplq + nt;
  S_.cplw = S_.colcnt + nt;
  S_.lstream = stream_.p; S_.wlstream = stream_.p + nrow;
  S_.w2stream = stream_.p + 3 * nrow;
  S_.own_first = rows_.p; S_.next_row = rows_.p + nt; S_.slot_row = rows_.p + 2 * nt;
  S_.nslots = (int)slot_row.size();
  S_.sms = sms;
  S_.counter_bytes = ncount * sizeof(int);
  S_.npairs = npairs_.p; S_.dig = dig_.p;
  S_.wait_ns = 2000000000ull;
  S_.min_diag_tol = 1.0e-12;   // ProfileSPDLinDirectSolver.h:49 default
  ready_ = true;
  return 0;
}

int ProfileSolver::solve(int nrhs, const double *const *b, double *const *x, cudaStream_t s) {
  if (!ready_) return XG_ESTATE;
  if (nrhs < 1 || nrhs > 4) return XG_EINVAL;
  ProfileSystem Sf = S_;
  for (int r = 0; r < nrhs; r++) {
    Sf.b[r] = b[r];
    Sf.x[r] = x[r];
  }
  if (int e = profile_solve(Sf, nrhs, s)) return e;
  return profile_status(Sf, s, nullptr);
}

int ProfileSolver::factor_forward(int nrhs, const double *const *b, cudaStream_t s) {
  if (!ready_) return XG_ESTATE;
  if (nrhs < 1 || nrhs > 4) return XG_EINVAL;
  fwd_nrhs_ = 0;
  ProfileSystem Sf = S_;
  Sf.fwd_nrhs = nrhs;
  for (int r = 0; r < nrhs; r++) Sf.b[r] = b[r];
  if (int e = profile_factor(Sf, s)) return e;
  fwd_nrhs_ = nrhs;
  return 0;
}

int ProfileSolver::solve_backward(int nrhs, double *const *x, cudaStream_t s, int *bad_eq) {
  *bad_eq = -1;
  if (!ready_) return XG_ESTATE;
  if (nrhs != fwd_nrhs_ || nrhs < 1) return XG_ESTATE;   // no matching forward sweep
  fwd_nrhs_ = 0;
  ProfileSystem Sf = S_;
  for (int r = 0; r < nrhs; r++) Sf.x[r] = x[r];
  if (int e = profile_solve(Sf, nrhs, s, true)) return e;
  return profile_status(Sf, s, bad_eq);
}

}  // namespace xg
