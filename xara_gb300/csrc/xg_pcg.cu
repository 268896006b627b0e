// xg_pcg.cu -- block-Jacobi preconditioned conjugate gradients: vectors,
// inner products and the preconditioner in FP64, the SpMV's products in
// float-float over a node-block copy of the matrix (FP64 warp per CSR row
// without one).
//
// The whole solve is one cooperative, persistent launch.  The inner products
// are reduced deterministically (fixed-order block partials, which every block
// sums in the same order), so the iterates are bit-identical run to run.
// k_pcg_nodes works on the node-block copy: slices of 32 node rows on warps
// spread over all SMs; blocks meet twice an iteration by publishing
// their partial sums and reading everybody's.  k_pcg serves the solves without
// a copy (grid-stride CSR rows, a counting grid barrier).  Every wait is
// bounded by the global timer: a block that waits longer than
// kBarrierTimeoutNs raises flags[0] and every block leaves the solve, so a
// fault can never hang the GPU.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <iterator>
#include <vector>

#include "xg_block_stream.h"
#include "xg_ff.h"
#include "xg_internal.h"
#include "xg_rcp.h"

namespace xg {

namespace {

constexpr int kPcgThreads = 512;
constexpr int kPcgMaxBlocks = 160;      // blocks a meeting can hold
constexpr unsigned long long kBarrierTimeoutNs = kCopyTimeoutNs;

// Sense-reversing grid barrier: bar[0] arrivals, bar[1] generation.
// Returns false (and sets flags[0]) on timeout or when another block did.
__device__ bool grid_barrier(unsigned int *bar, volatile int *flags) {
  __syncthreads();
  __shared__ int ok;
  if (threadIdx.x == 0) {
    ok = 1;
    volatile unsigned int *vgen = bar + 1;
    const unsigned int gen = *vgen;
    __threadfence();
    const unsigned int arrived = atomicAdd(bar, 1u);
    if (arrived == gridDim.x - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      const unsigned long long t0 = global_ns();
      while (*vgen == gen) {
        if (flags[0] != 0) { ok = 0; break; }
        if (global_ns() - t0 > kBarrierTimeoutNs) { flags[0] = 2; ok = 0; break; }
        __nanosleep(64);
      }
    }
    __threadfence();
    if (flags[0] != 0) ok = 0;
  }
  __syncthreads();
  return ok != 0;
}

__device__ double block_reduce(double v, double *smem) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) smem[w] = v;
  __syncthreads();
  double t = 0.0;
  if (w == 0) {
    t = (lane < (int)(blockDim.x >> 5)) ? smem[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// Power-of-two scale of p's split: p2 = p * 2^-s with s the exponent of a
// bound on max |p|, so that every entry of the split lies below 2 whatever
// the size of the residual (p shrinks with it over a solve; a fixed range
// would send the late iterations to FP64).  Entries more than 2^126 below
// the bound fall into the single-precision subnormals or to zero: a change
// of at most 2^-126 of max |p| per entry, below the split's own rounding.
__device__ __forceinline__ int split_exponent(double bound) {
  if (!(bound > 0.0) || !isfinite(bound)) return 0;
  const int e = (int)(((unsigned)__double2hiint(bound) >> 20) & 0x7ff) - 1023;
  return e < -1000 ? -1000 : (e > 1000 ? 1000 : e);
}
__device__ __forceinline__ double pow2(int e) {
  return __hiloint2double((int)((unsigned)(1023 + e) << 20), 0);
}

// Sum of partials[0..nb) in a fixed order, broadcast to the whole block.
__device__ double sum_partials(const double *partials, int nb, double *smem) {
  double s = 0.0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) s += partials[i];
  s = block_reduce(s, smem);
  if (threadIdx.x == 0) smem[32] = s;
  __syncthreads();
  const double r = smem[32];
  __syncthreads();
  return r;
}

__device__ __forceinline__ double spmv_row(const PcgSystem &S, int row, const double *x,
                                           int lane) {
  double s = 0.0;
  const int b = S.rowptr[row], e = S.rowptr[row + 1];
  for (int k = b + lane; k < e; k += 32) s += S.vals[k] * x[S.colidx[k]];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  return s;  // lane 0
}

// Row of (A x) from the CSR arrays in FP64, one thread.
__device__ __forceinline__ double csr_row64(const PcgSystem &S, int row, const double *x) {
  double s = 0.0;
  const int e = S.rowptr[row + 1];
#pragma unroll 4
  for (int k = S.rowptr[row]; k < e; k++) s = fma(S.vals[k], x[S.colidx[k]], s);
  return s;
}

// Order of the stored inverse diagonal blocks: the node-block order, or 6
// (each block padded to 6 x 6) for a system without a node-block copy.
__device__ __forceinline__ int binv_order(const PcgSystem &S) { return S.kb > 0 ? S.kb : 6; }

// Stride of a node's slots in p2: the block order, 3 rounded up to 4 so that
// a node's entries are one aligned 32-byte sector.
template <int KB>
struct NodeSlots {
  static constexpr int kStride = KB == 3 ? 4 : KB;
};

template <int KB>
__device__ __forceinline__ void load_p2_node(const float2 *p2, int j, float2 *xb) {
  constexpr int KS = NodeSlots<KB>::kStride;
  if constexpr (KS == 1) {
    xb[0] = p2[j];
  } else {
    const float4 *src = reinterpret_cast<const float4 *>(p2 + (long)j * KS);
#pragma unroll
    for (int t = 0; t < KS / 2; t++) {
      const float4 v = src[t];
      xb[2 * t] = make_float2(v.x, v.y);
      xb[2 * t + 1] = make_float2(v.z, v.w);
    }
  }
}

// f(row, (A x)[row]) for this warp's CSR rows, on lane 0.
template <typename F>
__device__ __forceinline__ void for_rows_Ax(const PcgSystem &S, const double *x, F f) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int gthreads = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (int row = gtid >> 5; row < S.n; row += gthreads >> 5) {
    const double ax = spmv_row(S, row, x, lane);
    if (lane == 0) f(row, ax);
  }
}

// Vector work is done per diagonal block (<= 6 equations of one node), so
// every equation is read and written by exactly one thread in a phase.
struct BlockRange { int b, m; };
__device__ __forceinline__ BlockRange block_range(const PcgSystem &S, int k) {
  BlockRange r;
  r.b = S.blk_start[k];
  r.m = S.blk_start[k + 1] - r.b;
  return r;
}

// z = Binv r on block k
__device__ __forceinline__ void precondition_block(const PcgSystem &S, int k, BlockRange br) {
  constexpr int MB = 6;
  const double *B = S.binv + (long)k * MB * MB;
  double rr[MB];
#pragma unroll
  for (int i = 0; i < MB; i++) rr[i] = i < br.m ? S.r[br.b + i] : 0.0;
#pragma unroll
  for (int i = 0; i < MB; i++) {
    if (i >= br.m) break;
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < MB; j++)
      if (j < br.m) t += B[MB * i + j] * rr[j];
    S.z[br.b + i] = t;
  }
}

// scalars: [3] iterations  [4] relres  [5] (b - A x)^2  [6] |b|
// partials: [0, 3 nb) the inner products' block sums.
__global__ void __launch_bounds__(kPcgThreads, 2)
    k_pcg(PcgSystem S, const double *b, double *x, double rtol, int maxit) {
  __shared__ double smem[40];
  volatile int *flags = S.flags;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int gthreads = gridDim.x * blockDim.x;
  const int nb = gridDim.x;
  double *part = S.partials;

  // r = b - A x ; (x is the initial guess)
  for_rows_Ax(S, x, [&](int row, double ax) { S.r[row] = b[row] - ax; });
  if (!grid_barrier(S.barrier, flags)) return;
  double lrz = 0.0, lbb = 0.0, lrr = 0.0;
  for (int k = gtid; k < S.nblk; k += gthreads) {
    const BlockRange br = block_range(S, k);
    precondition_block(S, k, br);
    for (int i = br.b; i < br.b + br.m; i++) {
      S.p[i] = S.z[i];
      lrz += S.r[i] * S.z[i];
      lbb += b[i] * b[i];
      lrr += S.r[i] * S.r[i];
    }
  }
  lrz = block_reduce(lrz, smem);
  if (threadIdx.x == 0) part[blockIdx.x] = lrz;
  lbb = block_reduce(lbb, smem);
  if (threadIdx.x == 0) part[nb + blockIdx.x] = lbb;
  lrr = block_reduce(lrr, smem);
  if (threadIdx.x == 0) part[2 * nb + blockIdx.x] = lrr;
  if (!grid_barrier(S.barrier, flags)) return;
  double rz = sum_partials(part, nb, smem);
  const double bb = sum_partials(part + nb, nb, smem);
  double rr = sum_partials(part + 2 * nb, nb, smem);
  const double bnorm = sqrt(bb);
  int it = 0;
  int status = 0;
  if (bnorm == 0.0 || sqrt(rr) <= rtol * bnorm) {
    status = 1;
  }
  while (status == 0 && it < maxit) {
    // q = A p ; pq = p.q
    if (!grid_barrier(S.barrier, flags)) return;   // partial sums consumed, p complete
    double lpq = 0.0;
    for_rows_Ax(S, S.p, [&](int row, double ap) {
      S.q[row] = ap;
      lpq += ap * S.p[row];
    });
    lpq = block_reduce(lpq, smem);
    if (threadIdx.x == 0) part[blockIdx.x] = lpq;
    if (!grid_barrier(S.barrier, flags)) return;
    const double pq = sum_partials(part, nb, smem);
    if (!(pq > 0.0)) { status = -1; break; }
    const double alpha = rz / pq;
    if (!grid_barrier(S.barrier, flags)) return;   // partial sums consumed, q complete
    lrz = 0.0; lrr = 0.0;
    for (int k = gtid; k < S.nblk; k += gthreads) {
      const BlockRange br = block_range(S, k);
      for (int i = br.b; i < br.b + br.m; i++) {
        x[i] += alpha * S.p[i];
        S.r[i] -= alpha * S.q[i];
      }
      precondition_block(S, k, br);
      for (int i = br.b; i < br.b + br.m; i++) {
        lrz += S.r[i] * S.z[i];
        lrr += S.r[i] * S.r[i];
      }
    }
    lrz = block_reduce(lrz, smem);
    if (threadIdx.x == 0) part[blockIdx.x] = lrz;
    lrr = block_reduce(lrr, smem);
    if (threadIdx.x == 0) part[nb + blockIdx.x] = lrr;
    if (!grid_barrier(S.barrier, flags)) return;
    const double rz_new = sum_partials(part, nb, smem);
    rr = sum_partials(part + nb, nb, smem);
    it++;
    if (sqrt(rr) <= rtol * bnorm) { status = 1; break; }
    const double beta = rz_new / rz;
    rz = rz_new;
    for (int k = gtid; k < S.nblk; k += gthreads) {
      const BlockRange br = block_range(S, k);
      for (int i = br.b; i < br.b + br.m; i++) S.p[i] = S.z[i] + beta * S.p[i];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S.scalars[3] = it;
    S.scalars[4] = bnorm > 0.0 ? sqrt(rr) / bnorm : 0.0;
    S.flags[1] = status;
  }
}

// ---------------------------------------------------------------------------
// the node-block copy's solve
// ---------------------------------------------------------------------------
constexpr unsigned long long kPcgUnset = 0xFFFFFFFFFFFFFFFFull;   // byte fill 0xFF

template <int KB>
struct NodeShared {
  static constexpr int kWarps = NodeShape<KB>::kWarps, kGroup = NodeShape<KB>::kGroup;
  static constexpr int kRing = NodeShape<KB>::kRing;
  BlockRecord<KB> rec[kWarps][kRing][kGroup];
  float2 y[kWarps][KB][32];             // a part's row sums; the parts' residuals as doubles
  double x[kWarps][KB][32];             // the solution (vectors in registers otherwise)
  unsigned long long full[kWarps][kRing + 1];
  double part[2][kWarps];               // the warps' sums
  unsigned top[kWarps];
  double out[5];
  unsigned max;
  int ok[2];                            // by epoch, set by the meeting before
};

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ void publish(double *p, double v) {
  if ((unsigned long long)__double_as_longlong(v) == kPcgUnset)
    v = __longlong_as_double(0x7FF8000000000000ll);   // keep a NaN a NaN
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// upper bound of |v| by its high word (a NaN or an infinity above all)
__device__ __forceinline__ unsigned mag_hi(double v) {
  return (unsigned)__double2hiint(v) & 0x7fffffffu;
}
__device__ __forceinline__ double mag_bound(unsigned hi) { return __hiloint2double((int)hi, -1); }

// Sum of the warp's values, N <= 7 a lane, on every lane.  Integer arithmetic on
// the significands: shifted to the largest one's place with two bits to spare
// (four for N = 1) and rounded there, added in three pieces by the warp's
// integer reductions (a piece's terms fit 32 bits), and rounded to a double
// once.  A value is off by at most 2^-55 (2^-57) of the largest, so the sum is
// as good as FP64 additions in any order.  Five butterfly steps of FP64 additions
// take 540 cycles (64 each, and 90 to hand a result to the shuffle), 1,725 when
// 16 warps share the SM's FP64 unit; this takes 310, and 425.  Values too close
// to the ends of the exponent range go the butterfly way.
template <int N>
__device__ __forceinline__ double warp_sum(const double (&v)[N]) {
  constexpr int kSpare = N == 1 ? 4 : 2;
  static_assert(N >= 1 && N <= 7, "the sum of 32 N terms has to fit 63 bits");
  unsigned top = 0u;
#pragma unroll
  for (int u = 0; u < N; u++) top = max(top, (unsigned)__double2hiint(v[u]) & 0x7fffffffu);
  top = __reduce_max_sync(0xffffffffu, top);
  const int E = (int)(top >> 20);
  if (E < 80 || E > 2030) {
    double t = 0.0;
    unsigned any = 0u;
#pragma unroll
    for (int u = 0; u < N; u++) {
      t += v[u];
      any |= ((unsigned)__double2hiint(v[u]) & 0x7fffffffu) | (unsigned)__double2loint(v[u]);
    }
    if (E == 0 && __reduce_or_sync(0xffffffffu, any) == 0u) return 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  }
  long long sum = 0;
#pragma unroll
  for (int u = 0; u < N; u++) {
    const unsigned hi = (unsigned)__double2hiint(v[u]), lo = (unsigned)__double2loint(v[u]);
    const int e = (int)((hi >> 20) & 0x7ffu), shift = E - e;
    if (e > 0 && shift < 58) {
      long long m = (long long)((((unsigned long long)((hi & 0xfffffu) | 0x100000u)) << 32 | lo)
                                << (kSpare + 1));
      m = ((m >> shift) + 1) >> 1;
      sum += (hi >> 31) ? -m : m;
    }
  }
  const unsigned s0 = __reduce_add_sync(0xffffffffu, (unsigned)sum & 0xfffffu);
  const unsigned s1 = __reduce_add_sync(0xffffffffu, (unsigned)(sum >> 20) & 0xfffffu);
  const int s2 = __reduce_add_sync(0xffffffffu, (int)(sum >> 40));
  const long long t = ((long long)s2 << 40) + ((long long)s1 << 20) + (long long)s0;
  if (t == 0) return 0.0;
  unsigned long long n = (unsigned long long)(t < 0 ? -t : t);
  const int lz = __clzll((long long)n);
  n <<= lz;                        // leading bit 63 = 2^(63 - lz) of 2^(E - 1075 - kSpare)
  const unsigned long long sig = ((n >> 1) + 0x200) >> 10;   // 53 bits, or 2^53 after rounding
  return __longlong_as_double((long long)((((unsigned long long)(E + 10 - kSpare - lz)) << 52) +
                                              sig |
                                          (t < 0 ? 0x8000000000000000ull : 0ull)));
}
__device__ __forceinline__ double warp_sum(double v) {
  const double a[1] = {v};
  return warp_sum(a);
}

// The rows of node rows with more than S.nb_cap blocks (a node tied to a
// whole face by a multi-point constraint couples to every node of that
// face) in chunks of at most kLongChunk CSR entries, four warps per chunk
// with a quarter of it each: g(quarter, partial, h(row)) on lane 0.  A warp per
// row would leave one warp thousands of entries; at 64 cycles an FP64
// operation even a whole chunk's 16 a lane are a thousand.
constexpr int kLongChunk = 512, kLongPart = kLongChunk / 4;
template <typename H, typename G>
__device__ __forceinline__ void long_row_chunks(const PcgSystem &S, const double *x, H h, G g) {
  // from the last warps of the last blocks on, which have fewer slices
  const int warps = blockDim.x >> 5, nwarps = gridDim.x * warps;
  const int lane = threadIdx.x & 31;
  const int first = (warps - 1 - (int)(threadIdx.x >> 5)) * gridDim.x + gridDim.x - 1 - blockIdx.x;
  for (int c = first; c < 4 * S.nchunks; c += nwarps) {
    const int row = __ldg(S.chunk_row + (c >> 2)), c0 = __ldg(S.chunk_beg + (c >> 2));
    const int b = c0 + kLongPart * (c & 3);
    const int e = min(min(b + kLongPart, c0 + kLongChunk), __ldg(S.rowptr + row + 1));
    const double hr = h(row);
    double v[kLongPart / 32], xv[kLongPart / 32];
#pragma unroll
    for (int u = 0; u < kLongPart / 32; u++) {
      const int k = b + lane + 32 * u;
      v[u] = k < e ? __ldg(S.vals + k) : 0.0;
      xv[u] = k < e ? x[__ldg(S.colidx + k)] : 0.0;
    }
    double t = 0.0;
#pragma unroll
    for (int u = 0; u < kLongPart / 32; u++) t += v[u] * xv[u];
    t = warp_sum(t);
    if (lane == 0) g(c, t, hr);
  }
}

// v 2^-scale as a float pair, the values split2 gives, in integer arithmetic
// off the FP64 unit (whose conversions would take it longer than the products)
__device__ __forceinline__ float2 split2_scaled(double v, int scale) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int be = (int)((hi >> 20) & 0x7ffu), fe = be - 1023 - scale;
  if (be == 0 || be == 2047 || fe < -70 || fe > 100) return split2(v * pow2(-scale));
  unsigned top = ((hi & 0xfffffu) << 3) | (lo >> 29);
  int rem = (int)(lo & 0x1fffffffu);
  if (rem >= 1 << 28) {
    top++;
    rem -= 1 << 29;
  }
  const float h = __uint_as_float(((unsigned)(fe + 127) << 23) + top);
  const float l = __int2float_rn(rem) * __uint_as_float((unsigned)(fe - 52 + 127) << 23);
  return (hi >> 31) ? make_float2(-h, -l) : make_float2(h, l);
}

// (sh, sl) += (h, l)
__device__ __forceinline__ void ff_add(float h, float l, float &sh, float &sl) {
  const float t = __fadd_rn(sh, h);
  const float bp = __fsub_rn(t, sh);
  const float err = __fadd_rn(__fsub_rn(sh, __fsub_rn(t, bp)), __fsub_rn(h, bp));
  sh = t;
  sl = __fadd_rn(sl, __fadd_rn(l, err));
}

// A grid-wide meeting that carries up to two sums and the largest of the
// threads' mx.  Every block publishes its partial sums in its own slot (four
// sets of slots by epoch, a slot unset again once every block must have read
// it: when the next meeting is over) and every block waits for all slots and
// sums them in the same order: one way through the L2 instead of an atomic
// count, its release and a read of the sums.  finish(q, sum) runs on lane 0 of
// warp q, behind the block's first barrier and before its second (values for
// all threads go into E.out).  What a thread of a block
// that releases wrote before is visible behind it to the blocks that acquire;
// of two meetings in a row one does both everywhere, which also carries the
// unset slots.  False on timeout or when another block failed.
template <int NV, int KB, typename F>
__device__ __forceinline__ bool meet(const PcgSystem &S, NodeShared<KB> &E, int &epoch, double v0,
                                     double v1, unsigned mx, volatile int *flags, F finish,
                                     bool release = true, bool acquire = true) {
  constexpr int kWarps = NodeShape<KB>::kWarps;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nb = gridDim.x;
  double *slots = S.partials + (size_t)(epoch & 3) * 3 * nb;
  double *old = S.partials + (size_t)((epoch + 3) & 3) * 3 * nb;
  if (NV >= 1) {
    v0 = warp_sum(v0);
    if (lane == 0) E.part[0][warp] = v0;
  }
  if (NV >= 2) {
    v1 = warp_sum(v1);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) {
      E.part[1][warp] = v1;
      E.top[warp] = mx;
    }
  }
  __syncthreads();
  if (tid == 0) E.ok[(epoch + 1) & 1] = 1;
  constexpr int kPolls = NV == 2 ? 3 : 1;      // polling warps: sum, sum, largest
  if (warp < kPolls) {
    double v = 0.0;
    if (NV >= 1 && warp < 2) v = warp_sum(lane < kWarps ? E.part[warp & 1][lane] : 0.0);
    else if (NV >= 1)
      v = __hiloint2double(0, (int)__reduce_max_sync(0xffffffffu, lane < kWarps ? E.top[lane] : 0u));
    if (lane == 0) {
      if (release) fence_gpu();
      publish(slots + warp * nb + blockIdx.x, v);
    }
    double a[kPcgMaxBlocks / 32];
    bool ok = true;
    unsigned long long t0 = 0;
    for (int tries = 1;; tries++) {
      bool ready = true;
#pragma unroll
      for (int u = 0; u < kPcgMaxBlocks / 32; u++) {
        const int i = lane + 32 * u;
        a[u] = 0.0;
        if (i < nb)
          asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];"
                       : "=d"(a[u])
                       : "l"(slots + warp * nb + i)
                       : "memory");
      }
#pragma unroll
      for (int u = 0; u < kPcgMaxBlocks / 32; u++)
        ready &= (unsigned long long)__double_as_longlong(a[u]) != kPcgUnset;
      if (__all_sync(0xffffffffu, ready)) break;
      if (tries % 64) continue;
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      const bool late = now - t0 > kBarrierTimeoutNs;
      if (late) flags[0] = 2;
      if (__any_sync(0xffffffffu, late || flags[0] != 0)) { ok = false; break; }
    }
    if (acquire) fence_gpu();
    if (!ok && lane == 0) E.ok[epoch & 1] = 0;
    if (NV >= 1 && warp < 2) {
      const double t = warp_sum(a);
      if (lane == 0) finish(warp, t);
    } else if (NV >= 1) {
      unsigned m = 0u;
#pragma unroll
      for (int u = 0; u < kPcgMaxBlocks / 32; u++) m = max(m, (unsigned)__double2loint(a[u]));
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) E.max = m;
    }
  }
  __syncthreads();
  const bool ok = E.ok[epoch & 1] != 0;
  // every block is past the meeting before this one
  if (tid < 3)
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(old + tid * nb + blockIdx.x),
                 "d"(__longlong_as_double((long long)kPcgUnset)) : "memory");
  epoch++;
  return ok;
}

// Node-block sliced ELL copy of the matrix, thread per node row: the
// equations of node i (its diagonal block, m <= KB of them) against the
// nodes j it couples to, each coupling a KB x KB block (zero-padded where a
// node has fewer free dofs).  Slice s holds node rows 32s .. 32s+31; block k
// of its rows is record nb_off[s]/32 + k (BlockRecord), so a warp's 32 node rows
// read each entry position with one coalesced access and one column index
// serves KB*KB values; rows with fewer blocks than the slice's longest have
// zeros there.  z is held split into (hi, lo) float pairs, node-major with
// NodeSlots<KB>::kStride slots per node (p2), so a block's KB entries of z are
// one aligned load.  Each row is summed in float-float (xg_ff.h), a part's
// groups of blocks alternately into two partial sums, the parts in order: a
// fixed order.

// Slice s of 32 node rows belongs to block s % gridDim.x, there to warp group
// (s / gridDim.x) % (kWarps / SP): SP warps share a slice's blocks in the SpMV,
// so that a system with fewer slices than warps still has every SM's rings and
// warps at work.  The SpMV's matrix comes through the warps' rings by bulk
// copies; its gathers of z run kAhead groups ahead.  A slice's vectors are kept
// one node a lane, by the group's first warp -- or an equation a lane, row a by
// warp a of the group, where there are as many warps as rows -- in registers
// when every group has at most one slice (kOne), else in memory.  Long nodes
// (more than nb_cap blocks) are left out there: their rows are summed in
// chunks, and a warp of block l % gridDim.x updates their vectors, an equation
// a lane.
//
// An iteration meets twice: with w = A z the products follow z,
//   p = z + beta p,  q = w + beta q = A p,  alpha = r.z / p.q,
// so that the blocks need not wait for each other's p between beta and the
// SpMV, and only z is published.  Its split's scale is taken from the largest
// entry of the z before; where the largest entry turns out to be more than
// 2^40 away from that, the iteration's SpMV runs on FP64 z.
//
// What bounds it: up to some 30,000 equations the two meetings' latency (an L2
// round trip to publish, one to read, a fence: 4 us each) and the few dependent
// steps between them; at 100,000 the issue of the float-float products and the
// rings' upkeep (300 instructions a group, a third of them products), the 79 MB
// of matrix staying in the L2; from 600,000 on the HBM stream.  Microseconds an
// iteration, with grid-stride rows, four counting grid barriers and butterflied
// FP64 sums before: 3,361 equations 47.6, now 13.0; 25,689: 50.5, 19.0; 101,185:
// 54.3, 27.5; 604,176: 118.7, 103.8 (4.6 TB/s).
template <int KB, int SP, bool kOne>
__global__ void __launch_bounds__(32 * NodeShape<KB>::kWarps, 1)
    k_pcg_nodes(PcgSystem S, const double *b, double *x, double rtol, int maxit) {
  extern __shared__ __align__(128) unsigned char dyn[];
  NodeShared<KB> &E = *reinterpret_cast<NodeShared<KB> *>(dyn);
  constexpr int KS = NodeSlots<KB>::kStride, KK = KB * KB;
  constexpr int kWarps = NodeShape<KB>::kWarps, kGroup = NodeShape<KB>::kGroup;
  constexpr int kAhead = NodeShape<KB>::kAhead;
  constexpr int kGroups = kWarps / SP;
  constexpr bool kRows = kOne && KB > 1 && SP >= KB;   // an equation a lane
  constexpr int NR = kRows ? 1 : KB;                   // equations a lane
  constexpr bool kB = kOne && NR * KB <= 9;            // inverse diagonal blocks in registers
  volatile int *flags = S.flags;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = warp / SP, part = warp % SP;
  const int a0 = kRows ? part : 0;
  const bool owner = kRows ? part < KB : part == 0;    // keeps vectors
  const int ns = (S.nblk + 31) / 32, first = blockIdx.x + gridDim.x * group;
  const int stride = gridDim.x * kGroups;
  int epoch = 0;

  if (tid < 2) E.ok[tid] = 1;
  if (lane < NodeShape<KB>::kRing) mbar_init(&E.full[warp][lane]);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  BlockStream<KB, SP, kOne> blocks{S, E.rec[warp], E.full[warp], lane, part, first, stride, ns};
  blocks.start();

  // node of a slice on this lane, -1 for none (past the end or a long node)
  auto node_of = [&](int s) {
    const int i = 32 * s + lane;
    return i < S.nblk && S.nb_len[i] <= S.nb_cap ? i : -1;
  };
  // The warp's long nodes: this lane's row of the node, whether there is one,
  // and its partial sums' range.  The first one's numbers stay in registers.
  struct Long {
    int node, row, m, beg, end;
    bool in;
    double B[KB];
  };
  const bool chunked = (int)(gridDim.x - 1 - blockIdx.x) < 4 * S.nchunks;   // in this block
  const bool longs = (int)blockIdx.x < S.nlongn;
  const int long0 = blockIdx.x + gridDim.x * ((2 * kWarps - 2 - warp) % kWarps);
  auto long_of = [&](int l) {
    Long L;
    L.node = S.long_node[l];
    L.row = S.blk_start[L.node];
    L.m = S.blk_start[L.node + 1] - L.row;
    L.in = lane < L.m;
    L.row += lane;
    const int i0 = S.long_row0[l] + (L.in ? lane : 0);
    L.beg = 4 * S.long_chunk0[i0];
    L.end = 4 * S.long_chunk0[i0 + 1];
#pragma unroll
    for (int c = 0; c < KB; c++)
      L.B[c] = L.in && c < L.m ? S.binv[(long)L.node * KK + lane * KB + c] : 0.0;
    return L;
  };
  Long mine_long;
  if (long0 < S.nlongn) mine_long = long_of(long0);
  auto for_long = [&](auto f) {
    if (long0 < S.nlongn) {
      f(mine_long);
      for (int l = long0 + gridDim.x * kWarps; l < S.nlongn; l += gridDim.x * kWarps) f(long_of(l));
    }
  };
  // (A v)[row] of a long node's rows from their chunks' partial sums
  auto long_sum = [&](const Long &L) {
    double w = 0.0;
#pragma unroll
    for (int a = 0; a < KB; a++) {
      if (a >= L.m) break;
      const int beg = __shfl_sync(0xffffffffu, L.beg, a), end = __shfl_sync(0xffffffffu, L.end, a);
      double t = 0.0;
#pragma unroll 4
      for (int c = beg + lane; c < end; c += 32) t += S.chunk_part[c];
      t = warp_sum(t);
      if (lane == a) w = t;
    }
    return w;
  };
  // z of a long node's row on this lane from the rows' r
  auto long_z = [&](const Long &L, double r) {
    double z = 0.0;
#pragma unroll
    for (int c = 0; c < KB; c++) z += L.B[c] * __shfl_sync(0xffffffffu, r, c);
    return z;
  };

  // this lane's node and its vectors (kOne)
  int mine = -1, mine0 = 0, minem = 0;
  bool mine_ff = false;
  double rk[NR], pk[NR], zk[NR], qk[NR], Bk[kB ? NR * KB : 1];
#pragma unroll
  for (int a = 0; a < NR; a++) rk[a] = pk[a] = zk[a] = qk[a] = 0.0;
  if (kOne && first < ns) {
    mine = node_of(first);
    if (mine >= 0) {
      mine0 = S.blk_start[mine];
      minem = S.blk_start[mine + 1] - mine0;
      mine_ff = S.blk_ff[mine] != 0;
    }
  }
  if (kB) {
#pragma unroll
    for (int t = 0; t < NR * KB; t++)
      Bk[t] = owner && mine >= 0 && a0 + t / KB < minem && t % KB < minem
                  ? S.binv[(long)mine * KK + KB * a0 + t] : 0.0;
  }
  // z = B r, the sums' terms
  auto precondition = [&](const double *B, int m, const double *r, const double *own,
                          double *z, double &lrz, double &lrr, unsigned &mz) {
#pragma unroll
    for (int a = 0; a < NR; a++) {
      double t = 0.0;
      if (a0 + a < m) {
#pragma unroll
        for (int c = 0; c < KB; c++)
          if (c < m) t += B[KB * a + c] * r[c];
        lrz += own[a] * t;
        lrr += own[a] * own[a];
        mz = max(mz, mag_hi(t));
      }
      z[a] = t;
    }
  };
  auto load = [&](const double *v, int r0, int m, double (&o)[NR]) {
#pragma unroll
    for (int a = 0; a < NR; a++) o[a] = a < m ? v[r0 + a] : 0.0;
  };
  auto publish_z = [&](int i, int row, int a, double z, int scale) {
    S.z[row] = z;
    S.p2[(long)i * KS + a] = split2_scaled(z, scale);
  };

  bool ok = true;
  int it = 0, status = 0;
  double rr = 0.0, bnorm = 0.0;
  do {
    // r = b - A x (x is the initial guess), in FP64 from the CSR arrays
    if (S.nchunks > 0) {
      long_row_chunks(S, x, [](int) { return 0.0; },
                      [&](int c, double t, double) { S.chunk_part[c] = t; });
      ok = meet<0>(S, E, epoch, 0.0, 0.0, 0u, flags, [](int, double) {});
      if (!ok) break;
    }
    double lrz = 0.0, lbb = 0.0, lrr = 0.0;
    unsigned mz = 0u;
    if (part == 0 || kOne)
      for (int s = first; s < ns; s += stride) {
        const int i = kOne ? mine : node_of(s);
        if (i < 0 || !owner) continue;
        const int r0 = S.blk_start[i], m = S.blk_start[i + 1] - r0;
        double r[KB], own[NR], z[NR];
#pragma unroll
        for (int a = 0; a < KB; a++) {
          r[a] = a < m ? b[r0 + a] - csr_row64(S, r0 + a, x) : 0.0;
          if (!kRows) own[a < NR ? a : 0] = r[a];
          else if (a == a0) own[0] = r[a];
        }
#pragma unroll
        for (int a = 0; a < NR; a++)
          if (a0 + a < m) lbb += b[r0 + a0 + a] * b[r0 + a0 + a];
        precondition(S.binv + (long)i * KK + KB * a0, m, r, own, z, lrz, lrr, mz);
#pragma unroll
        for (int a = 0; a < NR; a++) {
          if (a0 + a >= m) continue;
          if (kOne) {
            E.x[warp][a][lane] = x[r0 + a0 + a];
            rk[a] = own[a];
            zk[a] = z[a];
          } else {
            S.r[r0 + a] = own[a];
            S.p[r0 + a] = S.q[r0 + a] = 0.0;
          }
          S.z[r0 + a0 + a] = z[a];
        }
      }
    for_long([&](const Long &L) {
      const double bv = L.in ? b[L.row] : 0.0, w = long_sum(L), r = bv - w;
      const double z = long_z(L, r);
      if (L.in) {
        S.r[L.row] = r;
        S.z[L.row] = z;
        S.p[L.row] = S.q[L.row] = 0.0;
        lbb += bv * bv;
        lrz += r * z;
        lrr += r * r;
        mz = max(mz, mag_hi(z));
      }
    });
    ok = meet<2>(S, E, epoch, lrz, lrr, mz, flags, [&](int q, double t) { E.out[q] = t; });
    if (!ok) break;
    double rz = E.out[0];
    rr = E.out[1];
    bool all64 = !isfinite(mag_bound(E.max));       // FP64 SpMV from here on
    int scale = split_exponent(mag_bound(E.max));   // p2 = z * 2^-scale
    int next = scale;
    if (part == 0 || kOne)
      for (int s = first; s < ns; s += stride) {
        const int i = kOne ? mine : node_of(s);
        if (i < 0 || !owner) continue;
        const int r0 = S.blk_start[i], m = S.blk_start[i + 1] - r0;
#pragma unroll
        for (int a = 0; a < NR; a++)
          if (a0 + a < m) publish_z(i, r0 + a0 + a, a0 + a, S.z[r0 + a0 + a], scale);
      }
    for_long([&](const Long &L) {
      if (L.in) publish_z(L.node, L.row, lane, S.z[L.row], scale);
    });
    ok = meet<1>(S, E, epoch, lbb, 0.0, 0u, flags, [&](int, double t) { E.out[0] = t; });
    if (!ok) break;
    bnorm = sqrt(E.out[0]);
    // r.r against the tolerance: the squares decide except within rounding of it
    const double tol = rtol * bnorm, tol2 = tol * tol;
    const bool squares = tol2 > 1e-250 && tol2 < 1e250;
    auto converged = [&](double t) {
      if (squares) {
        if (t > tol2 * (1.0 + 1e-14)) return false;
        if (t < tol2 * (1.0 - 1e-14)) return true;
      }
      return sqrt(t) <= tol;
    };
    double beta = 0.0;
    if (bnorm == 0.0 || converged(rr)) status = 1;
    if (tid == 0) E.out[2] = chain_reciprocal(rz);
    while (status == 0 && it < maxit) {
      // w = A z, p = z + beta p, q = w + beta q ; pq = p.q
      double lpq = 0.0;
      const bool ff = !all64 && abs(next - scale) <= 40;
      const double up = pow2(scale);
      if (kOne) {
#pragma unroll
        for (int a = 0; a < NR; a++) pk[a] = zk[a] + beta * pk[a];
      }
      for (int s = first; s < ns; s += stride) {
        const int i = kOne ? mine : node_of(s);
        const bool fast = ff && (kOne ? mine_ff : i >= 0 && S.blk_ff[i] != 0);
        const int width = kOne && kGroup == 1 ? 0 : blocks.width(s);
        const int groups = kOne ? blocks.total : blocks.groups(width);
        float h0[KB], l0[KB], h1[KB], l1[KB];
#pragma unroll
        for (int a = 0; a < KB; a++) h0[a] = l0[a] = h1[a] = l1[a] = 0.f;
        // z of the columns of group g
        auto gather = [&](int g, float2 (&o)[kGroup][KS]) {
          if (g >= groups) return;
          const BlockRecord<KB> *r = blocks.get(ok);
#pragma unroll
          for (int u = 0; u < kGroup; u++)
            if (kGroup == 1 || kGroup * (part + SP * g) + u < width)
              load_p2_node<KB>(S.p2, r[u].col[lane], o[u]);
        };
        auto products = [&](int g, const float2 (&zz)[kGroup][KS], float (&h)[KB], float (&l)[KB]) {
          const BlockRecord<KB> *r = blocks.rec[blocks.oldest];
#pragma unroll
          for (int u = 0; u < kGroup; u++) {
            if (kGroup > 1 && kGroup * (part + SP * g) + u >= width) break;
#pragma unroll
            for (int a = 0; a < KB; a++)
#pragma unroll
              for (int c = 0; c < KB; c++) ff_madd(r[u].v[a * KB + c][lane], zz[u][c], h[a], l[a]);
          }
          blocks.release(ok);
        };
        float2 zg[kAhead][kGroup][KS];
#pragma unroll
        for (int u = 0; u < kAhead; u++) gather(u, zg[u]);
        for (int g = 0; g < groups; g += kAhead) {
#pragma unroll
          for (int u = 0; u < kAhead; u++) {
            if (g + u >= groups) break;
            if (u & 1) products(g + u, zg[u], h1, l1);
            else products(g + u, zg[u], h0, l0);
            gather(g + u + kAhead, zg[u]);
          }
        }
#pragma unroll
        for (int a = 0; a < KB; a++) ff_add(h1[a], l1[a], h0[a], l0[a]);
        if (SP > 1) {
          if (kRows || part > 0) {
#pragma unroll
            for (int a = 0; a < KB; a++) E.y[warp][a][lane] = make_float2(h0[a], l0[a]);
          }
          asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(32 * SP) : "memory");
          if (kRows && owner) {
            const float2 v = E.y[warp - part][a0][lane];
            h0[0] = v.x;
            l0[0] = v.y;
          }
          if (owner) {
#pragma unroll
            for (int h = 1; h < SP; h++)
#pragma unroll
              for (int a = 0; a < NR; a++) {
                const float2 v = E.y[warp - part + h][a0 + a][lane];
                ff_add(v.x, v.y, h0[a], l0[a]);
              }
          }
        }
        if (owner && i >= 0) {
          const int r0 = kOne ? mine0 : S.blk_start[i];
          const int m = kOne ? minem : S.blk_start[i + 1] - r0;
          double z[NR], p[NR], q[NR];
          if (!kOne) {
            load(S.z, r0, m, z);
            load(S.p, r0, m, p);
            load(S.q, r0, m, q);
          }
#pragma unroll
          for (int a = 0; a < NR; a++) {
            if (a0 + a >= m) continue;
            const int row = r0 + a0 + a;
            const double w = fast ? ((double)h0[a] + (double)l0[a]) * up : csr_row64(S, row, S.z);
            if (kOne) {
              qk[a] = w + beta * qk[a];
              lpq += pk[a] * qk[a];
            } else {
              S.p[row] = p[a] = z[a] + beta * p[a];
              S.q[row] = q[a] = w + beta * q[a];
              lpq += p[a] * q[a];
            }
          }
        }
      }
      if (S.nchunks > 0) {
        // the long nodes' p and q stay as they are until the meeting is over
        long_row_chunks(S, S.z, [&](int row) { return S.z[row] + beta * S.p[row]; },
                        [&](int c, double t, double p) {
                          S.chunk_part[c] = t;
                          lpq += t * p;
                        });
        for_long([&](const Long &L) {
          if (L.in) lpq += beta * S.q[L.row] * (S.z[L.row] + beta * S.p[L.row]);
        });
      }
      if (!ok) {         // a copy that did not come
        flags[0] = 2;
        E.ok[epoch & 1] = 0;
      }
      // alpha = rz / p.q
      ok = meet<1>(S, E, epoch, lpq, 0.0, 0u, flags, [&](int, double t) {
             E.out[0] = t;
             E.out[1] = reciprocal_out_of_range(t) ? rz / t : rz * chain_reciprocal(t);
           }, chunked, longs);
      if (!ok) break;
      if (!(E.out[0] > 0.0)) { status = -1; break; }
      const double alpha = E.out[1];
      scale = next;
      lrz = 0.0;
      lrr = 0.0;
      mz = 0u;
      if (kRows) {
        // the group's residuals, row by warp
        double *res = reinterpret_cast<double *>(&E.y[warp - part][0][0]);
        if (owner) {
          E.x[warp][0][lane] += alpha * pk[0];
          rk[0] -= alpha * qk[0];
          res[32 * part + lane] = rk[0];
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(32 * SP) : "memory");
        if (owner && mine >= 0) {
          double r[KB];
#pragma unroll
          for (int c = 0; c < KB; c++) r[c] = res[32 * c + lane];
          precondition(kB ? Bk : S.binv + (long)mine * KK + KB * a0, minem, r, rk, zk, lrz, lrr, mz);
          if (a0 < minem) publish_z(mine, mine0 + a0, a0, zk[0], scale);
        }
      } else if (owner) {
        for (int s = first; s < ns; s += stride) {
          const int i = kOne ? mine : node_of(s);
          if (i < 0) continue;
          const int r0 = kOne ? mine0 : S.blk_start[i];
          const int m = kOne ? minem : S.blk_start[i + 1] - r0;
          double r[NR], z[NR], xv[NR], p[NR], q[NR];
          if (!kOne) {
            load(x, r0, m, xv);
            load(S.r, r0, m, r);
            load(S.p, r0, m, p);
            load(S.q, r0, m, q);
          }
#pragma unroll
          for (int a = 0; a < NR; a++) {
            if (a >= m) continue;
            if (kOne) {
              E.x[warp][a][lane] += alpha * pk[a];
              r[a] = rk[a] -= alpha * qk[a];
            } else {
              x[r0 + a] = xv[a] + alpha * p[a];
              S.r[r0 + a] = r[a] -= alpha * q[a];
            }
          }
          precondition(kB ? Bk : S.binv + (long)i * KK, m, r, r, z, lrz, lrr, mz);
#pragma unroll
          for (int a = 0; a < NR; a++)
            if (a < m) {
              if (kOne) zk[a] = z[a];
              publish_z(i, r0 + a, a, z[a], scale);
            }
        }
      }
      for_long([&](const Long &L) {
        double zv = 0.0, pv = 0.0, qv = 0.0, rv = 0.0, xv = 0.0;
        if (L.in) {
          zv = S.z[L.row];
          pv = S.p[L.row];
          qv = S.q[L.row];
          rv = S.r[L.row];
          xv = x[L.row];
        }
        const double w = long_sum(L), p = zv + beta * pv, q = w + beta * qv, r = rv - alpha * q;
        const double z = long_z(L, L.in ? r : 0.0);
        if (L.in) {
          S.p[L.row] = p;
          S.q[L.row] = q;
          S.r[L.row] = r;
          x[L.row] = xv + alpha * p;
          publish_z(L.node, L.row, lane, z, scale);
          lrz += r * z;
          lrr += r * r;
          mz = max(mz, mag_hi(z));
        }
      });
      const double rz_inv = E.out[2];
      ok = meet<2>(S, E, epoch, lrz, lrr, mz, flags, [&](int q, double t) {
        E.out[q] = t;
        if (q == 0 && reciprocal_out_of_range(rz)) E.out[4] = t / rz;
        if (q == 1) E.out[3] = converged(t) ? 1.0 : 0.0;
      });
      if (!ok) break;
      rr = E.out[1];
      it++;
      if (E.out[3] != 0.0) { status = 1; break; }
      beta = reciprocal_out_of_range(rz) ? E.out[4] : E.out[0] * rz_inv;
      rz = E.out[0];
      all64 |= !isfinite(mag_bound(E.max));
      next = split_exponent(mag_bound(E.max));
      if (warp == kWarps - 1 && lane == 0) E.out[2] = chain_reciprocal(rz);
    }
  } while (false);
  blocks.drain();
  if (!ok) return;
  if (kOne && owner && mine >= 0)
#pragma unroll
    for (int a = 0; a < NR; a++)
      if (a0 + a < minem) x[mine0 + a0 + a] = E.x[warp][a][lane];
  if (blockIdx.x == 0 && tid == 0) {
    S.scalars[3] = it;
    S.scalars[4] = bnorm > 0.0 ? sqrt(rr) / bnorm : 0.0;
    S.scalars[6] = bnorm;
    S.flags[1] = status;
  }
}

// scalars[5] = |b - A x|^2 in FP64 from the CSR arrays, a warp per row, the
// blocks' sums added in their order by the last block (flags[2] counts them).
//
// k_pcg_nodes' r follows by recurrence, and with it the products' errors, which add
// up: after some thousands of iterations on a system of jumping coefficients (1 to
// 1e3) b - A x was 7e-12 of b where r was 1e-12 (5e-12 with q = A p formed in every
// iteration).  pcg_solve looks at the true one once r has converged and
// starts again from x where it is not there yet.  What bounds it: the matrix's
// stream; of 101,185 equations 166 us where a solve takes 13,000.
constexpr double kResidualSlack = 1.05;
constexpr int kResidualThreads = 256;
__global__ void __launch_bounds__(kResidualThreads) k_pcg_residual(PcgSystem S, const double *b,
                                                                   const double *x) {
  __shared__ double smem[40];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warps = gridDim.x * (kResidualThreads / 32);
  double rr = 0.0;
  for (int row = blockIdx.x * (kResidualThreads / 32) + (threadIdx.x >> 5); row < S.n; row += warps) {
    double t = 0.0;
    const int e = S.rowptr[row + 1];
    for (int k = S.rowptr[row] + lane; k < e; k += 256) {     // eight loads in flight
      double v[8], xv[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        v[u] = k + 32 * u < e ? S.vals[k + 32 * u] : 0.0;
        xv[u] = k + 32 * u < e ? x[S.colidx[k + 32 * u]] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (32 * u < e - k + lane) t = fma(v[u], xv[u], t);
    }
    t = warp_sum(t);
    const double r = b[row] - t;
    if (lane == 0) rr += r * r;
  }
  rr = block_reduce(rr, smem);
  if (threadIdx.x == 0) {
    S.partials[blockIdx.x] = rr;
    __threadfence();
    last = atomicAdd(S.flags + 2, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  rr = sum_partials(S.partials, gridDim.x, smem);
  if (threadIdx.x == 0) S.scalars[5] = rr;
}

// Diagonal blocks of the CSR matrix, inverted by Gauss-Jordan with partial
// pivoting (blocks are at most 6 x 6: the free dofs of one node).
__global__ void k_factor_blocks(PcgSystem S) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= S.nblk) return;
  const int b = S.blk_start[k], m = S.blk_start[k + 1] - b;
  double A[6][12];
  for (int i = 0; i < m; i++) {
    for (int j = 0; j < 2 * m; j++) A[i][j] = (j == m + i) ? 1.0 : 0.0;
    const int row = b + i;
    for (int q = S.rowptr[row]; q < S.rowptr[row + 1]; q++) {
      const int c = S.colidx[q];
      if (c >= b && c < b + m) A[i][c - b] = S.vals[q];
    }
  }
  bool singular = false;
  for (int c = 0; c < m; c++) {
    int piv = c;
    double best = fabs(A[c][c]);
    for (int i = c + 1; i < m; i++)
      if (fabs(A[i][c]) > best) { best = fabs(A[i][c]); piv = i; }
    if (best == 0.0) { singular = true; break; }
    if (piv != c)
      for (int j = 0; j < 2 * m; j++) { double t = A[c][j]; A[c][j] = A[piv][j]; A[piv][j] = t; }
    const double inv = 1.0 / A[c][c];
    for (int j = 0; j < 2 * m; j++) A[c][j] *= inv;
    for (int i = 0; i < m; i++) {
      if (i == c) continue;
      const double f = A[i][c];
      if (f != 0.0)
        for (int j = 0; j < 2 * m; j++) A[i][j] -= f * A[c][j];
    }
  }
  const int bo = binv_order(S);
  double *B = S.binv + (long)k * bo * bo;
  for (int i = 0; i < bo * bo; i++) B[i] = 0.0;
  if (singular) {
    // fall back to the point-Jacobi inverse of whatever diagonal exists
    for (int i = 0; i < m; i++) {
      double d = 0.0;
      const int row = b + i;
      for (int q = S.rowptr[row]; q < S.rowptr[row + 1]; q++)
        if (S.colidx[q] == row) d = S.vals[q];
      B[bo * i + i] = d != 0.0 ? 1.0 / d : 1.0;
    }
    return;
  }
  for (int i = 0; i < m; i++)
    for (int j = 0; j < m; j++) B[bo * i + j] = A[i][m + j];
}

// CSR values into the node-block copy, split into (hi, lo), thread per node
// row (once per matrix); blk_ff records whether every value of the node's
// rows lies in the split's range.  Slots no CSR entry maps to stay zero.
template <int KB>
__global__ void k_pack_blocks(PcgSystem S) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.nblk) return;
  BlockRecord<KB> *rec = reinterpret_cast<BlockRecord<KB> *>(S.nb_vals);
  bool ok = true;
  if (S.nb_len[i] <= S.nb_cap) {
    for (int r = S.blk_start[i]; r < S.blk_start[i + 1]; r++)
      for (int q = S.rowptr[r]; q < S.rowptr[r + 1]; q++) {
        const double v = S.vals[q];
        const unsigned at = (unsigned)S.nb_pos[q];
        ok = ok && ff_range(v);
        (&rec[at / (32 * KB * KB)].v[0][0])[at % (32 * KB * KB)] = split2(v);
      }
    const long base = S.nb_off[i >> 5];
    for (int k = 0; k < S.nb_len[i]; k++)
      rec[(base >> 5) + k].col[i & 31] = S.nb_cols[base + 32L * k + (i & 31)];
  }
  S.blk_ff[i] = ok ? 1 : 0;
}

// co-resident blocks of the CSR solve; blocks of the node solve (one per SM): of
// the current device (its occupancy, a slow query, asked once)
int sm_count(int dev) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}
int csr_blocks() {
  static std::atomic<int> known[64];
  int dev = 0;
  cudaGetDevice(&dev);
  int per = dev < 64 ? known[dev].load() : 0;
  if (per == 0) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pcg, kPcgThreads, 0);
    per = std::max(per, 1);
    if (dev < 64) known[dev].store(per);
  }
  return sm_count(dev) * per;
}
int node_blocks() {
  int dev = 0;
  cudaGetDevice(&dev);
  return std::min(sm_count(dev), kPcgMaxBlocks);
}

struct NodeKernel {
  const void *f;
  int threads, smem;
};
template <int KB, int SP, bool kOne>
NodeKernel node_kernel_ready() {
  const void *f = (const void *)k_pcg_nodes<KB, SP, kOne>;
  // the attribute belongs to the current device
  const bool ok = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(NodeShared<KB>)) == cudaSuccess;
  return {ok ? f : nullptr, 32 * NodeShape<KB>::kWarps, (int)sizeof(NodeShared<KB>)};
}
// Warps per slice: as many, up to eight, as leave every slice a warp group of
// its own; vectors in registers as long as that holds.  (More warps on a slice
// only shorten its chain of groups while there are idle ones: on 3,361 equations
// eight took 21.0 us an iteration where four took 24.7.)
template <int KB>
NodeKernel node_kernel(long slices, long blocks) {
  const long warps = blocks * NodeShape<KB>::kWarps;
  if constexpr (NodeShape<KB>::kWarps >= 8)
    if (8 * slices <= warps) return node_kernel_ready<KB, 8, true>();
  if (4 * slices <= warps) return node_kernel_ready<KB, 4, true>();
  if (2 * slices <= warps) return node_kernel_ready<KB, 2, true>();
  if (slices <= warps) return node_kernel_ready<KB, 1, true>();
  return node_kernel_ready<KB, 1, false>();
}

}  // namespace

int pcg_max_blocks() { return std::max(csr_blocks(), node_blocks()); }
size_t pcg_partial_doubles() { return std::max<size_t>(3 * (size_t)csr_blocks() + 8, 12 * (size_t)node_blocks()); }

int block_ell_layout(int n, const int *rowptr, const int *colidx, int nblk, const int *blk_start,
                     int cap, BlockEll &h) {
  h = BlockEll{};
  int maxm = 0;
  for (int i = 0; i < nblk; i++) maxm = std::max(maxm, blk_start[i + 1] - blk_start[i]);
  if (nblk == 0 || maxm < 1 || maxm > 6) return 0;
  const int kb = maxm == 1 ? 1 : maxm == 2 ? 2 : maxm == 3 ? 3 : 6;
  std::vector<int> node_of(n);
  for (int i = 0; i < nblk; i++)
    for (int r = blk_start[i]; r < blk_start[i + 1]; r++) node_of[r] = i;
  // block columns of every node row: the union over its rows (sorted)
  std::vector<long> lptr(nblk + 1, 0);
  std::vector<int> lst, row_l, merged;
  std::vector<int> all;
  all.reserve((size_t)rowptr[n] / (kb * kb) + nblk);
  for (int i = 0; i < nblk; i++) {
    lst.clear();
    for (int r = blk_start[i]; r < blk_start[i + 1]; r++) {
      row_l.clear();
      for (int q = rowptr[r]; q < rowptr[r + 1]; q++) {
        const int j = node_of[colidx[q]];
        if (row_l.empty() || row_l.back() != j) row_l.push_back(j);
      }
      if (r == blk_start[i]) {
        lst.swap(row_l);
      } else if (row_l != lst) {
        merged.clear();
        std::set_union(lst.begin(), lst.end(), row_l.begin(), row_l.end(),
                       std::back_inserter(merged));
        lst.swap(merged);
      }
    }
    all.insert(all.end(), lst.begin(), lst.end());
    lptr[i + 1] = (long)all.size();
  }
  const int ns = (nblk + 31) / 32;
  h.off.assign((size_t)ns + 1, 0);
  h.len.assign(nblk, 0);
  h.chunk_row.clear();
  h.chunk_beg.clear();
  h.long_chunk0.assign(1, 0);
  h.long_node.clear();
  h.long_row0.clear();
  for (int s = 0; s < ns; s++) {
    int w = 0;
    for (int i = 32 * s; i < std::min(nblk, 32 * s + 32); i++) {
      const int len = (int)(lptr[i + 1] - lptr[i]);
      h.len[i] = len;
      if (len <= cap) {
        w = std::max(w, len);
        continue;
      }
      h.long_node.push_back(i);
      h.long_row0.push_back((int)h.long_chunk0.size() - 1);
      for (int r = blk_start[i]; r < blk_start[i + 1]; r++) {
        for (int q = rowptr[r]; q < rowptr[r + 1]; q += kLongChunk) {
          h.chunk_row.push_back(r);
          h.chunk_beg.push_back(q);
        }
        h.long_chunk0.push_back((int)h.chunk_row.size());
      }
    }
    h.off[s + 1] = h.off[s] + 32L * w;
  }
  if (h.off.back() * kb * kb >= (long)INT32_MAX) return 0;   // positions as 32-bit ints
  h.cols.assign((size_t)h.off.back(), 0);
  h.pos.assign((size_t)rowptr[n], -1);
  for (int i = 0; i < nblk; i++) {
    const int len = h.len[i];
    if (len > cap) continue;
    const long base = h.off[i / 32];
    const int lane = i % 32;
    const int *L = all.data() + lptr[i];
    for (int k = 0; k < len; k++) h.cols[(size_t)base + 32L * k + lane] = L[k];
    for (int r = blk_start[i]; r < blk_start[i + 1]; r++) {
      const int a = r - blk_start[i];
      int k = 0;
      for (int q = rowptr[r]; q < rowptr[r + 1]; q++) {
        const int j = node_of[colidx[q]];
        while (L[k] != j) k++;
        const int b = colidx[q] - blk_start[j];
        h.pos[q] = (int)(base * kb * kb + ((long)(k * kb + a) * kb + b) * 32 + lane);
      }
    }
  }
  h.kb = kb;
  return kb;
}

size_t block_ell_pairs(const BlockEll &h) {
  return (size_t)h.off.back() * (h.kb * h.kb) + (size_t)h.off.back() / 2;
}

size_t block_ell_bytes(const BlockEll &h, int nblk) {
  if (h.kb == 0) return 0;
  const int ks = h.kb == 3 ? 4 : h.kb;
  return (size_t)h.off.back() * sizeof(int) + block_ell_pairs(h) * sizeof(float2) +
         h.pos.size() * sizeof(int) + h.off.size() * sizeof(long) +
         (size_t)nblk * (sizeof(int) + 1 + ks * sizeof(float2));
}

int pcg_factor_blocks(const PcgSystem &S, cudaStream_t s) {
  if (S.nblk == 0) return 0;
  k_factor_blocks<<<(S.nblk + 127) / 128, 128, 0, s>>>(S);
  if (cudaGetLastError() != cudaSuccess) return XG_ECUDA;
  if (S.nb_vals && S.kb > 0) {
    const int nb = (S.nblk + 127) / 128;
    if (S.kb == 1) k_pack_blocks<1><<<nb, 128, 0, s>>>(S);
    else if (S.kb == 2) k_pack_blocks<2><<<nb, 128, 0, s>>>(S);
    else if (S.kb == 3) k_pack_blocks<3><<<nb, 128, 0, s>>>(S);
    else k_pack_blocks<6><<<nb, 128, 0, s>>>(S);
    if (cudaGetLastError() != cudaSuccess) return XG_ECUDA;
  }
  return 0;
}

// Blocks of a solve.  Without the copy about four rows per warp: SpMV rows are
// latency-bound chains (row pointer, column index, vector entry), so mid-size
// systems want many warps; the grid barrier's cost grows slowly with the block
// count.  With it a block per SM; small systems fewer, down to a slice of 32 nodes a
// block (the meetings read every block's slot).
int pcg_grid(int n, int nblk, int kb, int rows_per_block, int most) {
  const long rows = kb == 0 ? n : (nblk + 31) / 32;
  const long per = kb == 0 ? (rows_per_block > 0 ? rows_per_block : 64)
                           : std::max(rows_per_block / 32, 1);
  return (int)std::min<long>(std::max<long>((rows + per - 1) / per, 1), most);
}

// One launch from the x at hand, and with the copy the true residual behind it.
static int pcg_cycle(const PcgSystem &S, const double *b, double *x, double rtol, int maxit,
                     cudaStream_t s, int rows_per_block, int (&flags)[4], double (&scalars)[8]) {
  const int kb = (S.nb_vals && S.kb > 0) ? S.kb : 0;
  if (cudaMemsetAsync(S.flags, 0, 4 * sizeof(int), s) != cudaSuccess) return XG_ECUDA;
  PcgSystem Sv = S;
  void *args[] = {(void *)&Sv, (void *)&b, (void *)&x, (void *)&rtol, (void *)&maxit};
  if (kb == 0) {
    const int nb = pcg_grid(S.n, S.nblk, 0, rows_per_block, csr_blocks());
    if (cudaMemsetAsync(S.barrier, 0, 2 * sizeof(unsigned int), s) != cudaSuccess) return XG_ECUDA;
    if (cudaLaunchCooperativeKernel((const void *)k_pcg, dim3(nb), dim3(kPcgThreads), args, 0, s) !=
        cudaSuccess)
      return XG_ECUDA;
  } else {
    const long slices = (S.nblk + 31) / 32;
    const int nb = pcg_grid(S.n, S.nblk, kb, rows_per_block, node_blocks());
    const NodeKernel k = kb == 1 ? node_kernel<1>(slices, nb) : kb == 2 ? node_kernel<2>(slices, nb)
                       : kb == 3 ? node_kernel<3>(slices, nb) : node_kernel<6>(slices, nb);
    if (!k.f) return XG_ECUDA;
    if (cudaMemsetAsync(S.partials, 0xFF, 12 * (size_t)nb * sizeof(double), s) != cudaSuccess)
      return XG_ECUDA;
    if (cudaLaunchCooperativeKernel(k.f, dim3(nb), dim3(k.threads), args, k.smem, s) != cudaSuccess)
      return XG_ECUDA;
    const int rows = kResidualThreads / 32;
    const int rb = (int)std::min<long>(((long)S.n + rows - 1) / rows, 12 * node_blocks());
    k_pcg_residual<<<rb, kResidualThreads, 0, s>>>(S, b, x);
    if (cudaGetLastError() != cudaSuccess) return XG_ECUDA;
  }
  if (cudaMemcpyAsync(flags, S.flags, sizeof flags, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaMemcpyAsync(scalars, S.scalars, sizeof scalars, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return XG_ECUDA;
  return 0;
}

int pcg_solve(const PcgSystem &S, const double *b, double *x, double rtol, int maxit,
              int *iters, double *relres, cudaStream_t s, int rows_per_block) {
  if (iters) *iters = 0;
  if (relres) *relres = 0.0;
  if (S.n == 0) return 0;
  const bool copy = S.nb_vals && S.kb > 0;
  int done = 0;
  double before = INFINITY;                  // the true residual of the cycle before
  for (;;) {
    int flags[4];
    double sc[8];
    if (int e = pcg_cycle(S, b, x, rtol, maxit - done, s, rows_per_block, flags, sc)) return e;
    const bool again = done > 0, converged = flags[1] == 1;
    done += (int)sc[3];
    if (iters) *iters = done;
    if (relres && (converged || !again)) *relres = sc[4];
    if (flags[0] != 0) return XG_ESOLVE;     // barrier timeout
    // breakdown or maxit; behind a cycle that had converged x is still its answer,
    // bettered
    if (!converged) return again ? 0 : XG_ESOLVE;
    // the recursive residual is there: start again from x while the true one is
    // not and a cycle at least halves it
    if (!copy || (int)sc[3] == 0) return 0;
    const double r = sqrt(sc[5]);
    if (!(r > kResidualSlack * rtol * sc[6]) || !(r < 0.5 * before) || done >= maxit) return 0;
    before = r;
  }
}

}  // namespace xg
