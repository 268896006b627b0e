// xg_band.cu -- `system ProfileSPD` for a model made of many small
// disconnected parts (a batch of frames): every part's LDL' in its own band,
// one block per part, all parts in one launch.  The reference runs each such
// model alone with ProfileSPDLinDirectSolver (system_of_eqn/linearSOE/
// profileSPD/ProfileSPDLinDirectSolver.cpp:100-256); its pivot checks are
// applied per part (the part's first pivot must be positive, later ones
// non-zero and above minDiagTol in magnitude).
//
// Storage: part c, local row i holds the entries (i, i-k), k = 0..b_c, at
// band[boff[c] + i*(b_c+1) + k] (b_c: the part's envelope width).
//
// Factor (k_band_factor): right-looking, the pivot chain one column ahead of
// the trailing update.  The rows column j touches, j..j+b, live in a ring of
// shared-memory rows; the rows beyond them are fetched kBandAhead columns
// early with cp.async, and a finished row goes back to the band.  The forward
// substitution and the diagonal scaling of up to four right-hand sides run
// inside the factorisation; the backward substitution (k_band_back) is one
// warp per part walking the band's rows upwards (x_i final, then the rows
// above take one FMA each from row i of L), rows prefetched the same way.
#include <cuda_runtime.h>

#include <algorithm>

#include "xg_internal.h"
#include "xg_rcp.h"

namespace xg {

namespace {

constexpr int kBandTrail = 6;           // trailing warps
constexpr int kBandWorkers = 32 * kBandTrail;
constexpr int kBandThreads = kBandWorkers + 64;
constexpr int kBandMaxWidth = 77;       // widest envelope band_plan accepts
constexpr int kBandAhead = 8;           // rows fetched ahead of use
constexpr int kBandMaxRhs = 4;

// reciprocal on the pivot chain (xg_rcp.h); the stored reciprocals are the
// correctly rounded ones
__device__ __forceinline__ double chain_rcp(double d) { return chain_reciprocal(d); }

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// the part's band from its CSR rows (lower triangle)
__device__ void band_fill(const BandSystem &S, int e0, int n, int ld, double *B) {
  for (long k = threadIdx.x; k < (long)n * ld; k += blockDim.x) B[k] = 0.0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int row = e0 + i;
    for (int q = S.rowptr[row]; q < S.rowptr[row + 1]; q++) {
      const int j = S.colidx[q] - e0;
      if (j <= i) B[(long)i * ld + (i - j)] = S.vals[q];
    }
  }
  __syncthreads();
}

// ProfileSPDLinDirectSolver.cpp:134-138 (first pivot), :189-199
__device__ __forceinline__ bool pivot_fails(const BandSystem &S, int j, double d) {
  return (j == 0) ? !(d > 0.0) : (d == 0.0 || fabs(d) <= S.min_diag_tol);
}

__device__ __forceinline__ void band_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void band_arrive(int id, int count) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// A window of 32 NB consecutive rows over a warp: row r sits in lane r % 32,
// register (r / 32) % NB.
template <int NB>
__device__ __forceinline__ double window_row(const double (&v)[NB], int r) {
  double t = v[0];
  if (NB == 2) t = (r & 32) ? v[NB - 1] : v[0];
  if (NB == 4) {
    const double a = (r & 32) ? v[1 % NB] : v[0], b = (r & 32) ? v[NB - 1] : v[2 % NB];
    t = (r & 64) ? b : a;
  }
  return __shfl_sync(0xffffffffu, t, r & 31);
}

// Shared memory (doubles): W[R*ldm] ring rows (entry (r, r-k) at (r % R)*ldm +
// k; ldm = bmax + 1, R a power of two: ring_rows), lcol and ccol [4][32 NB] the
// last columns of L and of the unscaled columns, by row, Yr
// [2*kBandAhead][kBandMaxRhs] right-hand sides on their way in.
//
// Warp 0 carries the pivot chain: with column j final it takes the pivot's
// reciprocal, scales the column, applies it to column j+1 (rows in registers,
// NB of them a lane; the raw column from the ring) and hands both on.  Warps
// 1-6 apply column j to columns j+2 and beyond, one FMA per entry, each thread
// up to K fixed entries (ti, tk) of the width-b trailing triangle in
// column-major order, so that column j+2, which the chain waits for, is every
// thread's first.  Warp 7 carries the right-hand sides (forward substitution,
// rows in registers as well), writes finished rows back and fetches new ones.
// Named barriers 1-2 (chain -> all, by column parity) and 3-4 (trailing ->
// chain).  One warp gets an FP64 operation every 64 cycles and the SM one every
// 19: a column of a 42-wide band (28 trailing operations, 7 on the chain) is
// bound by the unit at about 700 cycles, a narrow one by the chain at 550; with
// two block barriers a column and three trailing warps it took 1,860.  Every
// entry takes the same FMAs in the same order as before, bit for bit.
template <int K, int NB>
__global__ void __launch_bounds__(kBandThreads) k_band_factor(BandSystem S, int nrhs, double *x,
                                                              int ldx, int R) {
  extern __shared__ double sm[];
  const int c = blockIdx.x;
  if (c >= S.ncomp) return;
  const int e0 = S.cstart[c], n = S.cstart[c + 1] - e0, b = S.bw[c], ld = b + 1;
  const int ldm = S.bmax + 1, Rm = R - 1;
  constexpr int kWin = 32 * NB, kMask = kWin - 1;
  double *W = sm;
  double *lcol = W + (size_t)R * ldm, *ccol = lcol + 4 * kWin;
  double *Yr = ccol + 4 * kWin;
  __shared__ int bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double *B = S.band + S.boff[c];
  band_fill(S, e0, n, ld, B);
  const int n0 = min(n, R);
  for (int k = tid; k < n0 * ld; k += blockDim.x) W[(k / ld) * ldm + k % ld] = B[k];
  if (tid == 0) bad = 0;
  __syncthreads();
  constexpr int kAll = kBandThreads, kBack = kBandWorkers + 32;
  if (warp == 0) {
    double xc[NB];                // column j by rows, zero outside the band
    double d = n > 0 ? W[0] : 1.0;
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const int r = 1 + ((lane + 32 * u - 1) & kMask);
      xc[u] = r <= min(b, n - 1) ? W[(r & Rm) * ldm + r] : 0.0;
    }
    if (lane == 0 && n > 0 && pivot_fails(S, 0, d)) {
      bad = 1;
      S.flags[1] = e0;
      S.flags[0] = 3;
    }
#pragma unroll 1
    for (int j = 0; j < n; j++) {
      const double inv = chain_rcp(d);
      if (j >= 1) band_sync(3 + ((j - 1) & 1), kBack);
      // raw column j+1, rows j+1 .. min(j+1+b, n-1)
      int r[NB];
      double raw[NB];
      const int last = min(j + 1 + b, n - 1);
#pragma unroll
      for (int u = 0; u < NB; u++) {
        r[u] = j + 1 + ((lane + 32 * u - (j + 1)) & kMask);
        raw[u] = r[u] <= last ? W[(r[u] & Rm) * ldm + r[u] - (j + 1)] : 0.0;
      }
      const double ucc = window_row<NB>(xc, j + 1);
      double l[NB], xn[NB];
#pragma unroll
      for (int u = 0; u < NB; u++) {
        l[u] = xc[u] * inv;
        xn[u] = r[u] <= j + b ? fma(-l[u], ucc, raw[u]) : raw[u];
      }
      double *lc = lcol + (j & 3) * kWin, *cc = ccol + (j & 3) * kWin;
#pragma unroll
      for (int u = 0; u < NB; u++) {
        lc[r[u] & kMask] = l[u];
        cc[r[u] & kMask] = xc[u];
        if (r[u] <= min(j + b, n - 1)) W[(r[u] & Rm) * ldm + r[u] - j] = l[u];
        if (r[u] == j + 1 && j + 1 < n) W[((j + 1) & Rm) * ldm] = xn[u];
      }
      band_arrive(1 + (j & 1), kAll);
      d = window_row<NB>(xn, j + 1);
      if (lane == 0 && j + 1 < n && pivot_fails(S, j + 1, d) && !bad) {
        bad = 1;
        S.flags[1] = e0 + j + 1;
        S.flags[0] = 3;
      }
#pragma unroll
      for (int u = 0; u < NB; u++) xc[u] = r[u] == j + 1 ? 0.0 : xn[u];
    }
  } else if (warp <= kBandTrail) {
    // entries (ti, tk), 1 <= tk <= ti < b, of the window's triangle,
    // column-major: (ti << 16) | tk
    int ent[K];
    const int wid = tid - 32;
#pragma unroll
    for (int k = 0; k < K; k++) {
      int q = wid + kBandWorkers * k;
      ent[k] = -1;
      for (int tk = 1; tk < b; tk++) {
        if (q < b - tk) {
          ent[k] = ((tk + q) << 16) | tk;
          break;
        }
        q -= b - tk;
      }
    }
#pragma unroll 1
    for (int j = 0; j < n; j++) {
      band_sync(1 + (j & 1), kAll);
      const int m = min(b, n - 1 - j);
      const double *lc = lcol + (j & 3) * kWin, *cc = ccol + (j & 3) * kWin;
      // one pass of the loop is three loads, an FMA and a store; column j+2 is
      // in the first pass and released right behind it
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int e = ent[k];
        const int ti = e >> 16, tk = e & 0xffff;
        if (e >= 0 && ti < m) {
          const int row = j + 1 + ti;
          double *a = W + (row & Rm) * ldm + (ti - tk);
          *a = fma(-lc[row & kMask], cc[(j + 1 + tk) & kMask], *a);
        }
        if (k == 0 && j < n - 1) band_arrive(3 + (j & 1), kBack);
      }
    }
  } else {
    // right-hand sides: row r's value in register (r / 32) % NB of lane r % 32
    double y[NB][kBandMaxRhs];
#pragma unroll
    for (int u = 0; u < NB; u++)
#pragma unroll
      for (int q = 0; q < kBandMaxRhs; q++) {
        const int r = lane + 32 * u;
        y[u][q] = q < nrhs && r < n ? x[(long)q * ldx + e0 + r] : 0.0;
      }
#pragma unroll 1
    for (int j = 0; j < n; j++) {
      band_sync(1 + (j & 1), kAll);
      const double *lc = lcol + (j & 3) * kWin;
      const int m = min(b, n - 1 - j);
      double lv[NB];
      bool in[NB];
#pragma unroll
      for (int u = 0; u < NB; u++) {
        const int r = j + 1 + ((lane + 32 * u - (j + 1)) & kMask);
        in[u] = r <= j + m;
        lv[u] = in[u] ? lc[r & kMask] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < kBandMaxRhs; q++) {
        if (q >= nrhs) break;
        double col[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) col[u] = y[u][q];
        const double yj = window_row<NB>(col, j);
#pragma unroll
        for (int u = 0; u < NB; u++) {
          if (in[u]) y[u][q] = fma(-lv[u], yj, y[u][q]);
          // row j's slot takes row j + 32 NB, fetched through shared memory:
          // it arrives kBandAhead columns later, before its first use
          const double *yi = Yr + ((j - kBandAhead) & (2 * kBandAhead - 1)) * kBandMaxRhs + q;
          if (lane + 32 * u == ((j - kBandAhead) & kMask) && j >= kBandAhead)
            y[u][q] = *yi;
          if (lane + 32 * u == (j & kMask)) {
            x[(long)q * ldx + e0 + j] = y[u][q];
            if (j + kWin < n)
              cp_async8(Yr + (j & (2 * kBandAhead - 1)) * kBandMaxRhs + q,
                        x + (long)q * ldx + e0 + j + kWin);
          }
        }
      }
      // row j is final: back to the band; its ring row takes band row j+R,
      // which is complete kBandAhead columns later
      const bool refill = j + R < n;
      double *Wj = W + (j & Rm) * ldm;
      for (int t = lane; t < ld; t += 32) {
        B[(long)j * ld + t] = Wj[t];
        if (refill) cp_async8(Wj + t, B + (long)(j + R) * ld + t);
      }
      cp_async_commit();
      cp_async_wait<kBandAhead - 1>();
      __syncwarp();
    }
    cp_async_wait<0>();
  }
  __syncthreads();
  // the correctly rounded reciprocal pivots, and the diagonal scaling
  if (!bad) {
    for (int i = tid; i < n; i += blockDim.x) {
      const double inv = __drcp_rn(B[(long)i * ld]);
      S.invD[e0 + i] = inv;
      for (int r = 0; r < nrhs; r++) x[(long)r * ldx + e0 + i] *= inv;
    }
  }
}

// Backward substitution of one part per block: x_i = z_i once every row below
// has been applied, then z_r -= L(i, r) x_i for r = i-1 .. i-b (row i of the
// band, contiguous), over all right-hand sides in turn.  Warp 0 computes: the
// rows in reach sit in its registers (window_row), a step is a shuffle and an
// FMA a register, no branch, its operands in shared memory.  Warp 1 feeds it
// in batches of kBackRows steps, kBackStages of them in flight (cp.async): the
// band's rows, and the rows of z that come into reach; it takes the results
// back.  Named barriers 1-4: a batch is there, 5-8: its place is free.  z
// through shared memory with the fetching in the same warp took 550 cycles a
// row; the FMA's way to the shuffle and back is 120.
constexpr int kBackRows = 8, kBackStages = 4;

size_t back_smem(int bmax) {
  return (size_t)kBackStages * kBackRows * (bmax + 1 + 2) * sizeof(double);
}

template <int NB>
__global__ void __launch_bounds__(64) k_band_back(BandSystem S, int nrhs, double *x, int ldx) {
  extern __shared__ double sm[];
  constexpr int kWin = 32 * NB, kMask = kWin - 1;
  const int lane = threadIdx.x & 31, c = blockIdx.x, ldm = S.bmax + 1;
  double *rows = sm;                                              // [stage][step][ldm]
  double *zin = rows + (size_t)kBackStages * kBackRows * ldm;     // [stage][step]
  double *xout = zin + kBackStages * kBackRows;                   // [stage][step]
  const int e0 = S.cstart[c], n = S.cstart[c + 1] - e0, b = S.bw[c], ld = b + 1;
  const double *B = S.band + S.boff[c];
  const int per = (n + kBackRows - 1) / kBackRows, nb = per * nrhs;   // batches
  if (threadIdx.x < 32) {
    int k = 0;
    for (int q = 0; q < nrhs; q++) {
      const double *xr = x + (long)q * ldx + e0;
      double z[NB];                          // rows i .. i - 32 NB + 1
#pragma unroll
      for (int u = 0; u < NB; u++) {
        const int r = n - 1 - ((n - 1 - (lane + 32 * u)) & kMask);
        z[u] = r >= 0 ? xr[r] : 0.0;
      }
#pragma unroll 1
      for (int i0 = n - 1; i0 >= 0; i0 -= kBackRows, k++) {
        const int st = k & (kBackStages - 1);
        band_sync(1 + st, 64);
        const double *Ls = rows + (size_t)st * kBackRows * ldm, *zs = zin + st * kBackRows;
#pragma unroll
        for (int t = 0; t < kBackRows; t++) {
          const int i = i0 - t;
          if (i < 0) break;
          const double *Li = Ls + t * ldm;
          const double zi = zs[t];
          int kk[NB];
          double lv[NB];
#pragma unroll
          for (int u = 0; u < NB; u++) {
            kk[u] = (i - lane - 32 * u) & kMask;     // i minus the slot's row
            lv[u] = Li[min(kk[u], b)];
          }
          const double xi = window_row<NB>(z, i);
          const int reach = min(b, i);
#pragma unroll
          for (int u = 0; u < NB; u++) {
            if (kk[u] >= 1 && kk[u] <= reach) z[u] = fma(-lv[u], xi, z[u]);
            if (kk[u] == 0) z[u] = zi;               // row i's slot takes row i - 32 NB
          }
          if (lane == 0) xout[st * kBackRows + t] = xi;
        }
        __syncwarp();
        band_arrive(5 + st, 64);
      }
    }
    return;
  }
  // batch k: rows i0 .. i0 - kBackRows + 1 of right-hand side k / per
  auto take = [&](int k) {
    const int st = k & (kBackStages - 1), i0 = n - 1 - (k % per) * kBackRows;
    band_sync(5 + st, 64);
    if (lane < kBackRows && i0 - lane >= 0)
      x[(long)(k / per) * ldx + e0 + i0 - lane] = xout[st * kBackRows + lane];
  };
  for (int k = 0; k < nb + kBackStages; k++) {
    const int st = k & (kBackStages - 1);
    if (k >= kBackStages) take(k - kBackStages);
    if (k < nb) {
      const int i0 = n - 1 - (k % per) * kBackRows;
      for (int t = 0; t < kBackRows && i0 - t >= 0; t++)
        for (int e = lane; e < ld; e += 32)
          cp_async8(rows + ((size_t)st * kBackRows + t) * ldm + e, B + (long)(i0 - t) * ld + e);
      if (lane < kBackRows && i0 - lane - kWin >= 0)
        cp_async8(zin + st * kBackRows + lane, x + (long)(k / per) * ldx + e0 + i0 - lane - kWin);
    }
    cp_async_commit();
    // batch k - 2 has arrived
    cp_async_wait<2>();
    __syncwarp();
    if (k >= 2 && k - 2 < nb) band_arrive(1 + ((k - 2) & (kBackStages - 1)), 64);
  }
}

// Forward substitution and diagonal scaling on factors already in the band
// (solves after the factorisation): one warp per part, y_i = b_i - L(i,:) y
// reduced over the lanes.
__global__ void k_band_forward(BandSystem S, int nrhs, double *x, int ldx) {
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= S.ncomp) return;
  const int e0 = S.cstart[c], n = S.cstart[c + 1] - e0, b = S.bw[c], ld = b + 1;
  const double *B = S.band + S.boff[c];
  for (int q = 0; q < nrhs; q++) {
    double *xq = x + (long)q * ldx + e0;
    for (int i = 0; i < n; i++) {
      const int kmax = min(b, i);
      double s = 0.0;
      for (int k = 1 + lane; k <= kmax; k += 32) s += B[(long)i * ld + k] * xq[i - k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) xq[i] -= s;
      __syncwarp();
    }
    for (int i = lane; i < n; i += 32) xq[i] *= S.invD[e0 + i];
    __syncwarp();
  }
}

// The rows in use, kBandAhead fetched ahead, and two: the chain reads a fetched
// row two hand-offs after the warp that waited for it
int ring_rows(int bmax) {
  int R = 1;
  while (R < bmax + 1 + kBandAhead + 2) R <<= 1;
  return R;
}

// rows of a window in registers: the width, the pivot's row and kBandAhead
// rows for the loads of the next ones to arrive
int window_regs(int bmax) {
  const int rows = bmax + 1 + kBandAhead;
  return rows <= 32 ? 1 : rows <= 64 ? 2 : 4;
}

size_t factor_smem(int bmax) {
  const size_t ldm = bmax + 1, R = ring_rows(bmax);
  return (R * ldm + 8 * 32 * window_regs(bmax) + 2 * kBandAhead * kBandMaxRhs) * sizeof(double);
}

// trailing entries per worker for the widest band, rounded up to a kernel
// instance
int entries_per_worker(int bmax) {
  const int tri = bmax * (bmax - 1) / 2;
  const int k = (tri + kBandWorkers - 1) / kBandWorkers;
  for (int c : {1, 2, 3, 4, 5, 6, 8, 12, 16})
    if (k <= c) return c;
  return -1;
}

template <int K, int NB>
int launch_factor(const BandSystem &S, int nrhs, double *x, int ldx, cudaStream_t s) {
  const size_t smem = factor_smem(S.bmax);
  if (cudaFuncSetAttribute(k_band_factor<K, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return XG_ECUDA;
  k_band_factor<K, NB><<<S.ncomp, kBandThreads, smem, s>>>(S, nrhs, x, ldx, ring_rows(S.bmax));
  return cudaGetLastError() == cudaSuccess ? 0 : XG_ECUDA;
}

}  // namespace

int band_plan(int neq, const int *rowptr, const int *colidx, const std::vector<int> &cstart,
              std::vector<int> &bw, std::vector<long> &boff) {
  const int ncomp = (int)cstart.size() - 1;
  bw.assign(ncomp, 0);
  boff.assign(ncomp + 1, 0);
  for (int c = 0; c < ncomp; c++) {
    int w = 0;
    for (int i = cstart[c]; i < cstart[c + 1]; i++) {
      const int j = colidx[rowptr[i]];
      if (j < cstart[c]) return XG_EINVAL;        // coupled to another part
      w = std::max(w, i - j);
    }
    if (w > kBandMaxWidth) return XG_EINVAL;
    bw[c] = w;
    boff[c + 1] = boff[c] + (long)(cstart[c + 1] - cstart[c]) * (w + 1);
  }
  (void)neq;
  // the factorisation's ring of rows must fit in one block's shared memory,
  // and each worker's entries in its registers
  const int bmax = ncomp ? *std::max_element(bw.begin(), bw.end()) : 0;
  if (factor_smem(bmax) > 200 * 1024 || entries_per_worker(bmax) < 0) return XG_EINVAL;
  return 0;
}

int band_factor_async(const BandSystem &S, cudaStream_t s, int nrhs, double *x, int ldx) {
  if (S.ncomp == 0) return 0;
  if (nrhs < 0 || nrhs > kBandMaxRhs) return XG_EINVAL;
  if (cudaMemsetAsync(S.flags, 0, 4 * sizeof(int), s) != cudaSuccess) return XG_ECUDA;
  // widths up to 23 take one register of rows and at most two entries a
  // worker, up to 55 two and at most eight, the rest (up to 77) four
  switch (entries_per_worker(S.bmax)) {
    case 1: return launch_factor<1, 1>(S, nrhs, x, ldx, s);
    case 2: return window_regs(S.bmax) == 1 ? launch_factor<2, 1>(S, nrhs, x, ldx, s)
                                            : launch_factor<2, 2>(S, nrhs, x, ldx, s);
    case 3: return launch_factor<3, 2>(S, nrhs, x, ldx, s);
    case 4: return launch_factor<4, 2>(S, nrhs, x, ldx, s);
    case 5: return launch_factor<5, 2>(S, nrhs, x, ldx, s);
    case 6: return launch_factor<6, 2>(S, nrhs, x, ldx, s);
    case 8: return launch_factor<8, 2>(S, nrhs, x, ldx, s);
    case 12: return launch_factor<12, 4>(S, nrhs, x, ldx, s);
    case 16: return launch_factor<16, 4>(S, nrhs, x, ldx, s);
    default: return XG_EINVAL;
  }
}

int band_factor(const BandSystem &S, cudaStream_t s, int *bad_eq, int nrhs, double *x, int ldx) {
  if (S.ncomp == 0) return 0;
  const int r = band_factor_async(S, s, nrhs, x, ldx);
  if (r) return r;
  int hflags[4];
  if (cudaMemcpyAsync(hflags, S.flags, sizeof hflags, cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return XG_ECUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return XG_ECUDA;
  if (bad_eq) *bad_eq = hflags[0] == 3 ? hflags[1] : -1;
  return hflags[0] != 0 ? XG_ESOLVE : 0;
}

int band_solve(const BandSystem &S, int nrhs, double *x, int ldx, cudaStream_t s, bool forward) {
  if (S.ncomp == 0) return 0;
  if (forward) {
    const int warps = 4;
    k_band_forward<<<(S.ncomp + warps - 1) / warps, 32 * warps, 0, s>>>(S, nrhs, x, ldx);
  }
  const size_t smem = back_smem(S.bmax);
  switch (window_regs(S.bmax)) {
    case 1: k_band_back<1><<<S.ncomp, 64, smem, s>>>(S, nrhs, x, ldx); break;
    case 2: k_band_back<2><<<S.ncomp, 64, smem, s>>>(S, nrhs, x, ldx); break;
    default: k_band_back<4><<<S.ncomp, 64, smem, s>>>(S, nrhs, x, ldx); break;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : XG_ECUDA;
}

}  // namespace xg
