// xg_profile.cu -- the `system ProfileSPD` path on the device: LDL' of the
// symmetric tangent without pivoting, then forward / diagonal / backward
// substitution (ProfileSPDLinDirectSolver::solve, system_of_eqn/
// linearSOE/profileSPD/ProfileSPDLinDirectSolver.cpp:100-256).
//
// Storage: the lower triangle of the envelope (row i holds columns
// first(i)..i, first(i) = the first column of row i in the CSR pattern) in
// dense 32 x 32 FP64 tiles.  Tile row I keeps the tiles of columns J =
// I-W..I (W = the widest envelope in tiles), so tile (I, J) lives at offset
// (I*(W+1) + I-J) * 1024, row-major inside the tile; tiles left of the
// envelope (J < ftile[I]) stay zero and are skipped.  Right-looking LDL':
// for every tile column J,
//   A  the diagonal tile is factored (pivots d, unit lower L_JJ);
//   B  every tile below it becomes P_IJ = A_IJ L_JJ^-T and L_IJ = P_IJ D^-1;
//   C  every trailing tile pair loses P_IJ L_KJ'.
// Pivot checks follow the reference: the first pivot must be positive, later
// ones only non-zero and above minDiagTol in magnitude.
//
// Why the tile products run on the tensor cores.  The FP64 unit retires one
// warp instruction per 19 cycles and SM, and one warp no more than one per
// 64 cycles, so a 32^3 product costs 9.4 us on an SM: phase C alone would
// take 10 us of every column of a 10 x 10 x 20 frame (165 products over 152
// SMs).  C is therefore computed as sums of exact products: each operand row
// is scaled by a power of two and written as nine 9-bit digits (81 bits below
// the row's largest entry, where a double has 53), held as halves; the 45
// digit products whose weight reaches the result run as m16n8k16 tensor-core
// products whose float accumulators hold integers of at most 2^24 and so are
// exact; the nine weights are added as 64-bit integers and rounded to a
// double once.  The dropped products lie near 2^-77 of the product of the
// rows' largest entries; the columns of both operands are scaled by powers of
// two of sqrt(|d_k|) first, so that a row's entries (translations and
// rotations) are of one size.  Nine digits, not seven: the entries of a
// stiffness factor fall off by many orders along a row and FP64 keeps each to
// its own 53 bits; with seven (63 bits, products cut at 2^-59) the solution
// of the 10 x 10 x 20 frame lost three digits to the FP64 product, with nine
// none.  What the fixed point cannot hold are products far below their rows'
// sizes; those are taken in FP64 (weak_products).  (The idea of error-free digit products: K. Ozaki, T. Ogita, S. Oishi
// and S. M. Rump, Numer. Algorithms 59, 2012.)
//
// Who runs what.  One persistent cooperative launch, a block per SM.  What the
// next tile column waits for runs as a stream, in FP64 with the operands of the
// plain order (an explicit inverse of L_JJ would let the panels be products, but
// costs two digits: energy norm error 7e-13 against 4e-15 on a 64 x 16 quad
// block).  Tile J's elimination (block `diag` J mod 3) publishes every column of
// L_JJ as it is formed.  A tile row I belongs to two row blocks, 16 rows each,
// from its first column to its last: column by column they
// solve (I, J) and take P_IJ L_J+1,J' off tile (I, J+1), which they keep in
// registers, and row J+1's publish their columns of P and L for that and for the
// next diag block, which takes them off tile J+1.  So the next diagonal tile and
// every row's next panel are ready two hand-offs after the last pivot.  With the
// panels and those products from the list each row took solve, digits, product
// and three flags a column, 14.8 us however fast the eliminations (9) were.  A
// tile column takes 12.5 us now on a 64 x 16 quad block (63 of them, 15.4 before)
// and 13.7 on a 10 x 10 x 20 frame (454, 15.4): the elimination and 3 us from its
// last column to the next one's first, of which the two hand-offs are half.
// The other blocks take the other panels, the other tile pairs and the
// substitutions' matrices from a list in look-ahead order; their ninth warp draws the next task and waits for its operands
// (bounded by the global timer) while the eight others compute.  Every
// dependency sits earlier in the list or in the stream, and the digits live
// in a ring of kRing tile columns (a column's slots are refilled when its
// last pair has been applied).
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "xg_internal.h"
#include "xg_rcp.h"

namespace xg {

namespace {

constexpr int kT = 32;                 // tile edge
constexpr int kTT = kT * kT;
constexpr int kComputeThreads = 256;   // the eight computing warps of a block
constexpr int kFactorThreads = kComputeThreads + 32;

// digits of a tile operand: [kDigits][row][column] halves, then the rows'
// exponents
constexpr int kDigits = 9, kLowDigits = 5;   // of them in the lower word
constexpr int kDigitBytes = kDigits * kTT * 2;
constexpr int kOpBytes = kDigitBytes + kT * 4;
// ring slot of a panel tile: P, then L
constexpr int kSlotBytes = 2 * kOpBytes;
constexpr int kRing = 8;
constexpr int kDiagBlocks = 3;
// the stream's blocks: four warps that poll, four for the row blocks' digits
constexpr int kPollThreads = 128, kDigitThreads = 128;
constexpr int kBlockThreads = kComputeThreads + kPollThreads + kDigitThreads;
constexpr int kBadExp = 1 << 28;       // the exponent of a row with an infinity or a NaN
constexpr int kZeroExp = -(1 << 27);   // of a row without a digit
constexpr int kWeakBits = 24;          // below its rows' sizes by these a product is taken in FP64

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ double *tile_at(const ProfileSystem &S, int I, int o) {
  return S.L + ((size_t)I * (S.W + 1) + o) * kTT;
}

// Before a factorisation, in one launch: every row's envelope tiles zeroed and
// filled with the CSR values (a warp per row; rows past n get a unit pivot so
// the padded system solves to zero there), the counters cleared, the published
// columns and sweep values unset.
__global__ void k_prof_prepare(ProfileSystem S, size_t ncount, size_t nsweep) {
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t gthreads = (size_t)gridDim.x * blockDim.x;
  const double none = __longlong_as_double((long long)0xFFFFFFFFFFFFFFFFull);
  for (size_t k = gtid; k < ncount; k += gthreads) S.flags[k] = 0;
  for (size_t k = gtid; k < 5 * (size_t)S.nt * kTT; k += gthreads) S.lstream[k] = none;
  for (size_t k = gtid; k < nsweep; k += gthreads) S.sweep[k] = none;
  const int lane = threadIdx.x & 31;
  for (int i = (int)(gtid >> 5); i < S.nt * kT; i += (int)(gthreads >> 5)) {
    const int I = i / kT, r = i % kT;
    double *row = tile_at(S, I, 0) + r * kT;
    const bool pad = i >= S.n;
    for (int o = 0; o <= I - S.ftile[I]; o++)
      row[(size_t)o * kTT + lane] = pad && o == 0 && lane == r ? 1.0 : 0.0;
    __syncwarp();
    if (pad) continue;
    for (int k = S.rowptr[i] + lane; k < S.rowptr[i + 1]; k += 32) {
      const int j = S.colidx[k];
      if (j <= i) row[(size_t)(I - j / kT) * kTT + (j % kT)] = S.vals[k];
    }
  }
}

__device__ __forceinline__ int slot_of(const ProfileSystem &S, int I, int o) {
  return I * (S.W + 1) + o;
}
__device__ __forceinline__ unsigned char *dig_slot(const ProfileSystem &S, int J, int o) {
  return S.dig + ((size_t)(J % kRing) * S.W + (o - 1)) * kSlotBytes;   // o >= 1
}

__device__ __forceinline__ void named_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int count) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// The status words, and how long a wait may last.
struct Waits {
  volatile int *p;
  unsigned long long ns;
  __device__ __forceinline__ volatile int &operator[](int k) const { return p[k]; }
};

// Wait until *p >= target (one thread); false on a raised error flag or after
// the limit (flags[0] = 2).
__device__ __noinline__ bool wait_slow(const int *p, int target, Waits flags) {
  const volatile int *vp = p;
  const unsigned long long t0 = global_ns();
  for (;;) {
    for (int k = 0; k < 32; k++)
      if (*vp >= target) return true;
    if (flags[0] != 0) return false;
    if (global_ns() - t0 > flags.ns) {
      flags[0] = 2;
      return false;
    }
  }
}
__device__ __forceinline__ bool wait_geq(const int *p, int target, Waits flags) {
  return *(const volatile int *)p >= target || wait_slow(p, target, flags);
}

// The same with the order of the loads behind it (half the time of a fence).
__device__ __forceinline__ bool wait_acquire(const int *p, int target, Waits flags) {
  for (int k = 0;; k++) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if (v >= target) return true;
    if (k == 0) continue;
    if (!wait_slow(p, target, flags)) return false;
  }
}

// Published values: a scratch vector is filled with kUnset beforehand (a NaN
// pattern that no arithmetic result is stored as) and a consumer polls
// exactly the values it reads, so a value and its arrival are one word.
constexpr unsigned long long kUnset = 0xFFFFFFFFFFFFFFFFull;   // byte fill 0xFF

__device__ __forceinline__ double ld_relaxed(const double *p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ bool unset(double v) {
  return (unsigned long long)__double_as_longlong(v) == kUnset;
}

// *p once its producer has published it; 0 after a failed wait (flags[0]
// is then nonzero and the host reports the solve as failed).  await_slow is
// for the sweeps, where 64 blocks of threads poll and a look at the flag and
// the clock between two loads keeps them from crowding the L2 (981 against
// 1,108 us a backward sweep of 454 tile rows); await_column for the few warps
// that follow the factorisation's stream.
__device__ __forceinline__ double await_slow(const double *p, Waits flags) {
  const unsigned long long t0 = global_ns();
  for (;;) {
    const double v = ld_relaxed(p);
    if (!unset(v)) return v;
    if (flags[0] != 0) return 0.0;
    if (global_ns() - t0 > flags.ns) {
      flags[0] = 2;
      return 0.0;
    }
  }
}
__device__ __forceinline__ double await_column(const double *p, Waits flags) {
  const unsigned long long t0 = global_ns();
  for (;;) {
#pragma unroll 1
    for (int k = 0; k < 32; k++) {
      const double v = ld_relaxed(p);
      if (!unset(v)) return v;
    }
    if (flags[0] != 0) return 0.0;
    if (global_ns() - t0 > flags.ns) {
      flags[0] = 2;
      return 0.0;
    }
  }
}

// p[0], p[8], p[16], p[24] (the four loads in flight together)
__device__ __forceinline__ void await4(const double *p, double v[4], Waits flags) {
#pragma unroll
  for (int m = 0; m < 4; m++) v[m] = ld_relaxed(p + 8 * m);
#pragma unroll
  for (int m = 0; m < 4; m++)
    if (unset(v[m])) v[m] = await_slow(p + 8 * m, flags);
}

__device__ __forceinline__ void publish(double *p, double v) {
  if (unset(v)) v = __longlong_as_double(0x7FF8000000000000ll);   // keep a NaN a NaN
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// the computing and the polling warps
__device__ __forceinline__ void bsync() { named_sync(11, kComputeThreads + kPollThreads); }
// the eight computing warps
__device__ __forceinline__ void csync() { named_sync(9, kComputeThreads); }

// floor(log2(|v|) / 2): the power of two that brings sqrt(|v|) near 1
__device__ __forceinline__ int half_exp(double v) {
  const int be = (__double2hiint(v) >> 20) & 0x7ff;
  return (be == 0 || be == 0x7ff) ? 0 : (be - 1023) >> 1;
}

// Four consecutive entries of row r (columns 4q .. 4q+3, the eight threads
// of a row adjacent lanes of a warp), scaled by 2^-cs, as digits of |v|, v =
// x 2^(79-E), |x 2^-cs| < 2^E over the row, in two words of four and five
// digits: |v| plus 256 in every digit place has unsigned 9-bit fields, each
// 256 above its signed digit; a field in a half's mantissa under the exponent
// of 1024 is 1024 + field, 1280 less is the digit, and v's sign goes onto
// every digit.
__device__ __forceinline__ void slice_row4(const double (&x)[4], const int (&cs)[4], int r, int q,
                                           unsigned char *dst) {
  int e[4], em = -(1 << 20);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int be = (__double2hiint(x[i]) >> 20) & 0x7ff;
    e[i] = be == 0 ? -(1 << 20) : be == 0x7ff ? kBadExp : be - cs[i];
    em = max(em, e[i]);
  }
  em = max(em, __shfl_xor_sync(0xffffffffu, em, 1));
  em = max(em, __shfl_xor_sync(0xffffffffu, em, 2));
  em = max(em, __shfl_xor_sync(0xffffffffu, em, 4));
  const bool bad = em >= kBadExp - (1 << 16);
  constexpr int kLowBits = 9 * kLowDigits;
  constexpr unsigned long long kLowMask = (1ull << kLowBits) - 1;
  constexpr unsigned long long kBiasLow = 0x1008040201ull << 8, kBiasHigh = 0x8040201ull << 8;
  unsigned long long uh[4], ul[4];
  unsigned sg[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int hi = __double2hiint(x[i]), lo = __double2loint(x[i]);
    unsigned long long m = ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)lo;
    int sh = 26 - (em - e[i]);
    if (bad || sh <= -54 || e[i] <= -(1 << 19)) m = 0;
    if (sh < 0) {
      sh = max(sh, -63);
      m = (m + (1ull << (-sh - 1))) >> -sh;
      sh = 0;
    }
    ul[i] = ((m << sh) & kLowMask) + kBiasLow;
    uh[i] = (m >> (kLowBits - sh)) + kBiasHigh + (ul[i] >> kLowBits);
    sg[i] = ((unsigned)hi >> 16) & 0x8000u;
  }
  const size_t at = (size_t)(r * kT + 4 * q) * 2;
  const __half2 k1280 = __halves2half2(__ushort_as_half(0x6500), __ushort_as_half(0x6500));
#pragma unroll
  for (int d = 0; d < kDigits; d++) {
    constexpr int kHigh = kDigits - kLowDigits;
    const int s = 9 * ((d < kHigh ? kHigh : kDigits) - 1 - d);
    unsigned f[4];
#pragma unroll
    for (int i = 0; i < 4; i++) f[i] = (unsigned)((d < kHigh ? uh[i] : ul[i]) >> s) & 511u;
    unsigned w0 = f[0] | (f[1] << 16) | 0x64006400u, w1 = f[2] | (f[3] << 16) | 0x64006400u;
    const __half2 h0 = __hsub2(*reinterpret_cast<__half2 *>(&w0), k1280);
    const __half2 h1 = __hsub2(*reinterpret_cast<__half2 *>(&w1), k1280);
    w0 = *reinterpret_cast<const unsigned *>(&h0) ^ (sg[0] | (sg[1] << 16));
    w1 = *reinterpret_cast<const unsigned *>(&h1) ^ (sg[2] | (sg[3] << 16));
    *reinterpret_cast<uint2 *>(dst + d * kTT * 2 + at) = make_uint2(w0, w1);
  }
  if (q == 0)
    *reinterpret_cast<int *>(dst + kDigitBytes + 4 * r) =
        bad ? kBadExp : em <= -(1 << 16) ? kZeroExp : em - 1022;
}

__device__ __forceinline__ void mma16816(float (&c)[4], unsigned a0, unsigned a1, unsigned a2,
                                         unsigned a3, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// (hi 2^36 + lo) 2^sc rounded to a double (to nearest, ties up); |hi| < 2^62,
// |lo| < 2^63
__device__ __forceinline__ double fixed_to_double(long long hi, long long lo, int sc) {
  if (sc >= kBadExp / 2) return __longlong_as_double(0x7ff8000000000000ll);
  hi += lo >> 36;
  unsigned long long rem = (unsigned long long)lo & 0xfffffffffull;
  const bool neg = hi < 0;
  if (neg) {
    hi = rem ? ~hi : -hi;
    rem = (0x1000000000ull - rem) & 0xfffffffffull;
  }
  const int k = min(__clzll(hi), 36);
  const unsigned long long m = ((unsigned long long)hi << k) | (rem >> (36 - k));
  if (m == 0) return 0.0;
  const int lz = __clzll((long long)m);
  const unsigned long long n = m << lz;
  const int be = 1023 + 63 - lz + sc + 36 - k;
  unsigned long long bits = ((unsigned long long)(be - 1) << 52) + (n >> 11) + ((n >> 10) & 1);
  if (be <= 0) bits = 0;
  if (be >= 2047) bits = 0x7ff0000000000000ull;
  if (neg) bits |= 0x8000000000000000ull;
  return __longlong_as_double((long long)bits);
}

// Rows m0..m0+15 against rows n0..n0+7 of two operands: out = sums over the
// 32 columns, in the m16n8 accumulator layout (rows m0 + lane/4 and 8 more,
// columns n0 + 2 (lane % 4) and the next).  A lane takes columns 8 (lane %
// 4) .. +7 of its rows as its share of the contraction, the same for both
// operands, so a digit of a row is one 16-byte load (the operands are
// written during this launch: read through the L2).  Returns which of the four
// lie kWeakBits below the product of their rows' sizes (bit k: out[k]).
__device__ __forceinline__ uint4 frag(const unsigned char *op, int d, int row, int t) {
  return __ldcg(reinterpret_cast<const uint4 *>(op) + (d * kT + row) * 4 + t);
}
__device__ __forceinline__ int row_exp(const unsigned char *op, int row) {
  return __ldcg(reinterpret_cast<const int *>(op + kDigitBytes) + row);
}
__device__ __forceinline__ unsigned tile_product(const unsigned char *A, const unsigned char *B,
                                                 int m0, int n0, int lane, double (&out)[4]) {
  const int g = lane >> 2, t = lane & 3;
  uint4 a0[kDigits], a1[kDigits], b[kDigits];
#pragma unroll
  for (int d = 0; d < kDigits; d++) {
    a0[d] = frag(A, d, m0 + g, t);
    a1[d] = frag(A, d, m0 + 8 + g, t);
    b[d] = frag(B, d, n0 + g, t);
  }
  const int ea0 = row_exp(A, m0 + g), ea1 = row_exp(A, m0 + 8 + g);
  const int eb0 = row_exp(B, n0 + 2 * t), eb1 = row_exp(B, n0 + 2 * t + 1);
  float acc[kDigits][4];
#pragma unroll
  for (int u = 0; u < kDigits; u++)
#pragma unroll
    for (int k = 0; k < 4; k++) acc[u][k] = 0.f;
#pragma unroll
  for (int i = 0; i < kDigits; i++) {
#pragma unroll
    for (int j = 0; j < kDigits - i; j++)
      mma16816(acc[i + j], a0[i].x, a1[i].x, a0[i].y, a1[i].y, b[j].x, b[j].y);
#pragma unroll
    for (int j = 0; j < kDigits - i; j++)
      mma16816(acc[i + j], a0[i].z, a1[i].z, a0[i].w, a1[i].w, b[j].z, b[j].w);
  }
  unsigned weak = 0u;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    // weights 2^36 .. 1 of two words; the value is (hi 2^36 + lo) 2^(Ea+Eb-86)
    long long hi = 0, lo = 0;
#pragma unroll
    for (int u = 0; u < kDigits; u++) {
      const long long v = __float2int_rn(acc[u][k]);
      if (u < kDigits - 4) hi += v << (9 * (kDigits - 5 - u));
      else lo += v << (9 * (kDigits - 1 - u));
    }
    const int e = (k < 2 ? ea0 : ea1) + ((k & 1) ? eb1 : eb0);
    out[k] = fixed_to_double(hi, lo, e - 86);
    // (a row without digits or with a NaN has no size)
    if (e > kZeroExp / 2 && e < kBadExp / 2 &&
        ((__double2hiint(out[k]) >> 20) & 0x7ff) <= max(e + 1023 - kWeakBits, 0))
      weak |= 1u << k;
  }
  return weak;
}

struct FactorSmem {
  double A[kT][kT + 1];          // the tile at hand, by rows
  double W[kT][kT + 1];          // columns: a panel's P, a diagonal tile's unscaled columns
  double L[kT][kT + 1];          // and their L
  double inv[kT];                // reciprocal pivots of the panel's column
  double Lc[2][kT];              // the published column being applied
  int4 task[2];
  int fail;
};
// more than half an SM's shared memory: one block per SM
constexpr int kFactorSmem = 120 * 1024;
static_assert(sizeof(FactorSmem) <= kFactorSmem, "");

__device__ __forceinline__ void load4(const double *g, double (&x)[4]) {
  const double2 a = __ldcg(reinterpret_cast<const double2 *>(g));
  const double2 b = __ldcg(reinterpret_cast<const double2 *>(g) + 1);
  x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}

// LDL' of the diagonal tile in sm.A, as a two-stage pipeline, its columns of
// L published to st ([column][row], the reciprocal pivot on the diagonal) as
// they are formed; sm.L keeps them by columns (the pivot on the diagonal),
// sm.W the unscaled columns.  Warp 0 carries the pivot chain: with column c
// final it takes the pivot's reciprocal (xg_rcp.h), scales the column,
// applies it to column c+1 (one FMA per row) and, in the shadow of that FMA,
// writes column c out for warps 1-6, which apply it to columns c+3 and beyond
// (one FMA per entry, each thread holding up to three fixed entries).  The
// raw column c+1 with column c-1 applied, and its factor, are formed in the
// shadow of the reciprocal, so the trailing warps have two columns' time.
// An FP64 result reaches another FP64 operation after 64 cycles and any other
// unit after 90; a divergent branch on the chain costs 50-100 cycles, so it
// has none: every lane writes, also the rows above the diagonal that nobody
// reads, and the reciprocal's range is looked at behind the FMA.  520 cycles
// a column; 815 with the column written out under branches before the FMA and
// the reciprocal in FP64.  Hand-offs: named barriers 1-2 (chain -> trailing,
// by column parity) and 3-4 (trailing -> chain).  The FMAs and their operands
// are those of the plain right-looking order.
constexpr int kPipeCount = 7 * 32;      // the chain warp and six trailing warps
struct TrailEntries { int rw[3], sc[3]; };
// this thread's entries (r, s), 3 <= s <= r < 32, column-major order
__device__ __forceinline__ TrailEntries trail_entries(int warp, int lane) {
  TrailEntries t;
#pragma unroll
  for (int u = 0; u < 3; u++) {
    int e = (warp - 1) * 32 + lane + u * 192;
    t.rw[u] = t.sc[u] = -1;
    if (warp < 1 || warp > 6) continue;
    for (int k = 3; k < kT; k++) {
      if (e < kT - k) { t.rw[u] = k + e; t.sc[u] = k; break; }
      e -= kT - k;
    }
  }
  return t;
}
__device__ void eliminate_tile(FactorSmem &sm, int warp, int lane, const TrailEntries &te,
                               double *st) {
  if (warp == 0) {
    double x = sm.A[lane][0], lp = 0.0, up = 0.0;
#pragma unroll 1
    for (int c = 0; c < kT; c++) {
      const double d = __shfl_sync(0xffffffffu, x, c);
      double raw = 0.0, ucc = 0.0;
      if (c < kT - 1) {
        if (c >= 2) named_sync(3 + (c & 1), kPipeCount);
        raw = sm.A[lane][c + 1];
        ucc = __shfl_sync(0xffffffffu, x, c + 1);
        const double up1 = __shfl_sync(0xffffffffu, up, c + 1);
        if (c >= 1) raw = fma(-lp, up1, raw);
      }
      double inv = wide_reciprocal(d);
      double l = x * inv;
      double xn = fma(-l, ucc, raw);
      if (reciprocal_out_of_range(d)) {
        inv = __drcp_rn(d);
        l = x * inv;
        xn = fma(-l, ucc, raw);
      }
      sm.L[c][lane] = lane == c ? x : l;
      sm.W[c][lane] = x;
      if (c <= kT - 4) named_arrive(1 + (c & 1), kPipeCount);
      publish(st + c * kT + lane, lane == c ? inv : l);
      lp = l;
      up = x;
      x = xn;
    }
  } else if (warp <= 6) {
    double m[3];
#pragma unroll
    for (int u = 0; u < 3; u++) m[u] = te.rw[u] >= 0 ? sm.A[te.rw[u]][te.sc[u]] : 0.0;
    for (int c = 0; c < kT - 3; c++) {
      named_sync(1 + (c & 1), kPipeCount);
#pragma unroll
      for (int u = 0; u < 3; u++) {
        if (te.sc[u] >= c + 3) {
          m[u] = fma(-sm.L[c][te.rw[u]], sm.W[c][te.sc[u]], m[u]);
          if (te.sc[u] == c + 3) sm.A[te.rw[u]][c + 3] = m[u];
        }
      }
      named_arrive(3 + (c & 1), kPipeCount);
    }
  }
}

// Row r of a solved panel (I = J+o, J), row rs of the columns W of P and L in
// shared memory: L to the tile, P and L as digits to the ring slot; the eight
// threads q of a row adjacent.
template <int N>
__device__ __forceinline__ void panel_store(const ProfileSystem &S, const double (*W)[N],
                                            const double (*L)[N], const double *inv, int r, int rs,
                                            int q, int o, int J) {
  double p[4], l[4];
  int t[4], nt[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    p[i] = W[4 * q + i][rs];
    l[i] = L[4 * q + i][rs];
    nt[i] = half_exp(inv[4 * q + i]);
    t[i] = -nt[i];
  }
  double2 *tile = reinterpret_cast<double2 *>(tile_at(S, J + o, o) + r * kT + 4 * q);
  tile[0] = make_double2(l[0], l[1]);
  tile[1] = make_double2(l[2], l[3]);
  unsigned char *slot = dig_slot(S, J, o);
  slice_row4(p, t, r, q, slot);
  slice_row4(l, nt, r, q, slot + kOpBytes);
}

// Phase B on tile (I, J): P L_JJ' = A, L = P D^-1, column by column as L_JJ
// is published.  Lane = row; warp w of the eight computing ones holds columns
// w, w+8, w+16, w+24 in registers, so that a column's FMAs fill whole warps
// (496 in all: 9,400 cycles of the FP64 unit, below the elimination's own
// time); the warp whose column is final hands it to the others through shared
// memory.  The ninth warp polls the published columns (panel_poll), a column
// ahead of the others; one barrier a column.  Afterwards L goes
// to the tile and both, as digits, to the ring slot.
__device__ void panel_poll(const ProfileSystem &S, FactorSmem &sm, int J, int lane,
                           Waits flags) {
  const double *st = S.lstream + (size_t)J * kTT;
  double v = ld_relaxed(st + lane);
  for (int c = 0; c < kT; c++) {
    if (lane >= c) {
      if (unset(v)) v = await_column(st + c * kT + lane, flags);
      sm.Lc[c & 1][lane] = v;
      if (lane > c) v = ld_relaxed(st + (c + 1) * kT + lane);
    }
    __syncwarp();
    named_sync(10, kFactorThreads);
  }
}
__device__ void panel_task(const ProfileSystem &S, FactorSmem &sm, int I, int J, int tid) {
  const int r = tid >> 3, q = tid & 7, o = I - J, w = tid >> 5, lane = tid & 31;
  double *tile = tile_at(S, I, o) + r * kT + 4 * q;
  double x[4];
  load4(tile, x);
#pragma unroll
  for (int i = 0; i < 4; i++) sm.A[r][4 * q + i] = x[i];
  csync();
#pragma unroll
  for (int j = 0; j < 4; j++) x[j] = sm.A[lane][8 * j + w];
  if (w == 0) sm.W[0][lane] = x[0];
#pragma unroll
  for (int jc = 0; jc < 4; jc++) {
    for (int c8 = 0; c8 < 8; c8++) {
      const int c = 8 * jc + c8;
      named_sync(10, kFactorThreads);
      const double wc = sm.W[c][lane];
      const double *lc = sm.Lc[c & 1];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int s = 8 * j + w;
        if (j >= jc && s > c) {
          x[j] = fma(-wc, lc[s], x[j]);
          if (s == c + 1) sm.W[s][lane] = x[j];
        }
      }
      if (w == c8) {      // column c is this warp's: scale it
        const double inv = lc[c], v = x[jc] * inv;
        sm.L[c][lane] = v;
        if (lane == 0) sm.inv[c] = inv;
      }
    }
  }
  csync();
  panel_store(S, sm.W, sm.L, sm.inv, r, r, q, o, J);
}

// The entries of out that weak marks, summed again in FP64 from L and the pivots:
// eight entries at a time, four lanes each with eight columns: 18 operations of 64
// cycles for a warp where a lane by itself takes 64.  In a 10 x 10 x 20 frame 8 %
// of the warps have a mark; its load step takes 34.0 ms with them, 33.5 without and
// 35.2 with the products lane by lane.
__device__ void weak_products(const ProfileSystem &S, int J, int a, int b, int m0, int n0, int lane,
                              unsigned weak, double (&out)[4]) {
  const int group = lane >> 2, t = lane & 3;
  const double d = __drcp_rn(ld_relaxed(S.lstream + (size_t)J * kTT + lane * (kT + 1)));
#pragma unroll
  for (int u = 0; u < 4; u++) {
    unsigned marks = __ballot_sync(0xffffffffu, (weak >> u) & 1u);
    while (marks) {
      unsigned rest = marks, at = marks;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        if (k == group) at = rest;
        rest &= rest - 1;
      }
      const bool any = at != 0u;                 // this group's entry: the lane it belongs to
      const int of = any ? __ffs(at) - 1 : 0;
      const double2 *x = reinterpret_cast<const double2 *>(
          tile_at(S, J + a, a) + (m0 + (of >> 2) + 8 * (u >> 1)) * kT + 8 * t);
      const double2 *y = reinterpret_cast<const double2 *>(
          tile_at(S, J + b, b) + (n0 + 2 * (of & 3) + (u & 1)) * kT + 8 * t);
      double2 xv[4], yv[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        xv[k] = __ldcg(x + k);
        yv[k] = __ldcg(y + k);
      }
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        s = fma(xv[k].x * __shfl_sync(0xffffffffu, d, 8 * t + 2 * k), yv[k].x, s);
        s = fma(xv[k].y * __shfl_sync(0xffffffffu, d, 8 * t + 2 * k + 1), yv[k].y, s);
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      const int rank = __popc(marks & ((1u << lane) - 1u));
      const double v = __shfl_sync(0xffffffffu, s, 4 * (rank & 7));
      if ((marks >> lane & 1u) && rank < 8) out[u] = v;
      marks = rest;
    }
  }
}

// Phase C on pair (I = J+a, K = J+b), b <= a: A_IK -= P_IJ L_KJ'.  On a
// diagonal tile the blocks above the diagonal are left out.  An entry far below
// its rows' sizes -- two rows whose large entries do not meet, as of parts that
// a weak coupling joins -- is where the digits' fixed point holds fewer bits than
// a double (their error, 2^-77 of the sizes, is a rounding of an entry 2^-24
// below them, and all of one at 2^-77): it is summed again in FP64 from L and
// the pivots, so that small entries keep their own 53 bits.
__device__ void pair_task(const ProfileSystem &S, int J, int a, int b, int tid) {
  const int w = tid >> 5, lane = tid & 31, m0 = (w >> 2) * 16, n0 = (w & 3) * 8;
  if (a == b && n0 >= m0 + 16) return;
  const int g = lane >> 2, t = lane & 3;
  double2 *c0 = reinterpret_cast<double2 *>(tile_at(S, J + a, a - b) + (m0 + g) * kT + n0 + 2 * t);
  double2 *c1 = c0 + 4 * kT;
  const double2 v0 = __ldcg(c0), v1 = __ldcg(c1);
  double out[4];
  const unsigned weak = tile_product(dig_slot(S, J, a), dig_slot(S, J, b) + kOpBytes, m0, n0, lane, out);
  if (__any_sync(0xffffffffu, weak != 0u)) weak_products(S, J, a, b, m0, n0, lane, weak, out);
  *c0 = make_double2(v0.x - out[0], v0.y - out[1]);
  *c1 = make_double2(v1.x - out[2], v1.y - out[3]);
}

// W_J = L_JJ^-T for the substitutions: rows r of W solve w L_JJ' = e_r, four
// rows a warp side by side (a row's step is a shuffle and one FMA, some 180
// cycles of latency of which 64 are the FP64 unit's; one after another the four
// took 6 us; a one-tile factorisation with its set-up launch 39.2 us, now 37.2)
__device__ void inverse_task(const ProfileSystem &S, FactorSmem &sm, int J, int tid) {
  const int w = tid >> 5, lane = tid & 31;
  const double *Ljj = tile_at(S, J, 0);
  for (int k = tid; k < kTT; k += kComputeThreads) sm.A[k >> 5][k & 31] = __ldcg(Ljj + k);
  csync();
  double x[4];
#pragma unroll
  for (int j = 0; j < 4; j++) x[j] = lane == w + 8 * j ? 1.0 : 0.0;
  for (int c = w; c < kT - 1; c++) {
    const double l = sm.A[lane][c];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (c < w + 8 * j) continue;
      const double wc = __shfl_sync(0xffffffffu, x[j], c);
      if (lane > c) x[j] = fma(-wc, l, x[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; j++) S.Winv[(size_t)J * kTT + (w + 8 * j) * kT + lane] = x[j];
}

// For the substitutions, off the chain, with W_J = L_JJ^-T: pass 0
// F_J = W' L_J,J-1, 1 G_J = W L_J+1,J', 2 E_J = W' L_J,J-2, 3 H_J = W
// L_J+2,J' (zero where the tile is outside the envelope), a task each; then
// Q_J = E_J - F_J F_J-1 and R_J = H_J - G_J G_J+1.  With them a sweep row
// depends on the row two back: y_J = c3_J - F_J c_J-1 - Q_J y_J-2, c_J =
// c3_J - E_J y_J-2 (c3_J: W' times the right-hand side less rows J-3 and
// older), and the same backwards with G, H, R.
__device__ __forceinline__ bool coupling_tile(const ProfileSystem &S, int J, int pass, int *I,
                                              int *o) {
  const bool lower = (pass & 1) == 0;      // W' times a tile of row J
  *o = pass < 2 ? 1 : 2;
  *I = lower ? J : J + *o;
  return lower ? (J >= *o && S.ftile[J] <= J - *o) : (J + *o < S.nt && S.ftile[J + *o] <= J);
}
__device__ void coupling_task(const ProfileSystem &S, FactorSmem &sm, int J, int pass, int tid) {
  int I, o;
  const bool has = coupling_tile(S, J, pass, &I, &o), lower = (pass & 1) == 0;
  const size_t off = (size_t)J * kTT;
  double *out = (pass == 0 ? S.F : pass == 1 ? S.G : pass == 2 ? S.E : S.H) + off;
  if (!has) {
    for (int k = tid; k < kTT; k += kComputeThreads) out[k] = 0.0;
    return;
  }
  const double *T = tile_at(S, I, o);
  for (int k = tid; k < kTT; k += kComputeThreads) {
    sm.A[k >> 5][k & 31] = __ldcg(S.Winv + off + k);
    sm.W[k >> 5][k & 31] = __ldcg(T + k);
  }
  csync();
  for (int k = tid; k < kTT; k += kComputeThreads) {
    const int i = k >> 5, c = k & 31;
    double a0 = 0.0, a1 = 0.0;
    if (lower) {
      for (int q = 0; q < kT; q += 2) {
        a0 = fma(sm.A[q][i], sm.W[q][c], a0);
        a1 = fma(sm.A[q + 1][i], sm.W[q + 1][c], a1);
      }
    } else {
      for (int q = 0; q < kT; q += 2) {
        a0 = fma(sm.A[i][q], sm.W[c][q], a0);
        a1 = fma(sm.A[i][q + 1], sm.W[c][q + 1], a1);
      }
    }
    out[k] = a0 + a1;
  }
}
// which 0: Q_J, 1: R_J
__device__ void second_coupling_task(const ProfileSystem &S, FactorSmem &sm, int J, int which,
                                     int tid) {
  const size_t off = (size_t)J * kTT;
  const double *C0 = (which == 0 ? S.E : S.H) + off;
  double *out = (which == 0 ? S.Q : S.R) + off;
  if (which == 0 ? J == 0 : J == S.nt - 1) {
    for (int k = tid; k < kTT; k += kComputeThreads) out[k] = __ldcg(C0 + k);
    return;
  }
  const double *A = (which == 0 ? S.F : S.G) + off;
  const double *B = which == 0 ? A - kTT : A + kTT;
  for (int k = tid; k < kTT; k += kComputeThreads) {
    sm.A[k >> 5][k & 31] = __ldcg(A + k);
    sm.W[k >> 5][k & 31] = __ldcg(B + k);
  }
  csync();
  for (int k = tid; k < kTT; k += kComputeThreads) {
    const int i = k >> 5, c = k & 31;
    double a0 = 0.0, a1 = 0.0;
    for (int q = 0; q < kT; q += 2) {
      a0 = fma(sm.A[i][q], sm.W[q][c], a0);
      a1 = fma(sm.A[i][q + 1], sm.W[q + 1][c], a1);
    }
    out[k] = __ldcg(C0 + k) - (a0 + a1);
  }
}

// Dependencies of a list task (type, I, K, J): every update of its tile from
// earlier columns (the count of columns J' < J both tile rows reach), and the
// diagonal / panel tiles it reads.
// how often tile (I, J) is reported done: a panel of the row blocks by eight
// warps
__device__ __forceinline__ int done_count(const ProfileSystem &S, int I, int J) {
  return I > J && J >= S.own_first[I] ? 2 * kDigitThreads / 32 : 1;
}
__device__ __forceinline__ bool wait_done(const ProfileSystem &S, int I, int J,
                                          Waits flags) {
  return wait_geq(S.done + slot_of(S, I, I - J), done_count(S, I, J), flags);
}
enum { kPanel = 1, kPair = 2, kInverse = 5, kCouple = 6, kForward = 7, kCouple2 = 8 };
__device__ bool wait_task(const ProfileSystem &S, int4 t, Waits flags) {
  const int type = t.x, I = t.y, K = t.z, J = t.w;
  if (type == kPanel)     // the columns of L_JJ are polled inside the task
    return (J < kRing || wait_geq(S.colcnt + J - kRing, S.npairs[J - kRing], flags)) &&
           wait_geq(S.upd + slot_of(S, I, I - J), J - max(S.ftile[I], S.ftile[J]), flags);
  if (type == kPair)
    return wait_done(S, I, J, flags) && wait_done(S, K, J, flags) &&
           wait_geq(S.upd + slot_of(S, I, I - K), J - max(S.ftile[I], S.ftile[K]), flags);
  if (type == kInverse) return wait_done(S, J, J, flags);
  if (type == kCouple) {
    int Ic, o;
    if (!wait_geq(S.cplw + J, 1, flags)) return false;
    return !coupling_tile(S, J, K, &Ic, &o) || wait_done(S, Ic, Ic - o, flags);
  }
  if (type == kCouple2) {
    const int O = K == 0 ? J - 1 : J + 1;    // the neighbour's F or G
    return wait_geq(S.cpl + J, 4, flags) && (O < 0 || O >= S.nt || wait_geq(S.cpl + O, 4, flags));
  }
  // row J's forward step: its coupling matrices and the panel tiles of the
  // row further left (the y values of the rows before it are polled inside
  // the step)
  if (!wait_geq(S.cplq + J, 1, flags)) return false;
  const int ohi = min(S.W, J - S.ftile[J]);
  for (int o = 3; o <= ohi; o++)
    if (!wait_done(S, J, J - o, flags)) return false;
  return true;
}

// Pipelined substitutions on kPipeBlocks co-resident blocks (cooperative
// launch): block b owns the tile rows J = b, b + P, ... .  Forward, in
// increasing J: c3_J = L_JJ^-1 (b_J minus the contributions of rows J-3 and
// older), then with the factorisation's coupling matrices
//   y_J = c3_J - F_J c_J-1 - Q_J y_J-2,   c_J = c3_J - E_J y_J-2,
// so a row waits for the row two back (and for c_J-1, which its owner
// publishes as soon as y_J-3 is known): the two interleaved chains halve
// the serial length.  Backward, in decreasing J, the same with
// c3'_J = L_JJ^-T (D_J^-1 y_J minus the transposed contributions of rows J+3
// and beyond):  x_J = c3'_J - G_J c'_J+1 - R_J x_J+2,  c'_J = c3'_J -
// H_J x_J+2.  There are no row flags: every solved value is published to a
// scratch vector filled with kUnset beforehand (a NaN pattern that no
// arithmetic result is stored as), and a consumer thread polls exactly the
// values it reads.  Waits are bounded by the global timer.
constexpr int kPipeBlocks = 64;
constexpr int kPipeThreads = 256;
// right-hand side q, zero past the last equation
__device__ __forceinline__ double rhs_at(const ProfileSystem &S, int q, int i) {
  return i < S.n ? __ldcg(S.b[q] + i) : 0.0;
}

// Forward substitution of tile row J for the right-hand sides given to the
// factorisation (S.fwd_nrhs of them), as a task of the factorisation itself:
// the right-hand sides are known before the tangent is factored (the
// unbalance and the reference load of a Newton iteration), so row J's step
// runs as soon as its coupling matrices are written, a few columns behind
// the factorisation's front, instead of after it.  The step is the pipelined
// sweep's (k_prof_solve_pipe) for one row: c3_J = L_JJ^-1 (b_J minus rows
// J-3 and older), y_J = c3_J - F_J c_J-1 - Q_J y_J-2, c_J = c3_J - E_J
// y_J-2, published to the sweep's scratch (y, c) for the rows after it and
// for the backward sweep.
__device__ bool forward_row(const ProfileSystem &S, int J, double (*rb)[kT],
                            Waits flags) {
  const int tid = threadIdx.x;
  const int r = tid >> 3, g = tid & 7;
  const int nrhs = S.fwd_nrhs, ls = S.nt * kT;
  double *ys = S.sweep, *cs = ys + (size_t)nrhs * ls;
  auto group_sum = [](double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
  };
  auto row_of = [&](const double *M, double (&mv)[4]) {
#pragma unroll
    for (int m = 0; m < 4; m++) mv[m] = __ldcg(M + r * kT + g + 8 * m);
  };
  auto row_times = [&](const double (&mv)[4], const double *p) {
    double v[4];
    await4(p + g, v, flags);
    double t = 0.0;
#pragma unroll
    for (int m = 0; m < 4; m++) t = fma(mv[m], v[m], t);
    return group_sum(t);
  };
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const int ohi = min(S.W, J - S.ftile[J]);
  for (int o = ohi; o >= 3; o--) {
    const double *Lt = tile_at(S, J, o) + r * kT + g;
    const double l0 = __ldcg(Lt), l1 = __ldcg(Lt + 8), l2 = __ldcg(Lt + 16), l3 = __ldcg(Lt + 24);
    for (int q = 0; q < nrhs; q++) {
      double y[4];
      await4(ys + (size_t)q * ls + (J - o) * kT + g, y, flags);
      acc[q] += l0 * y[0] + l1 * y[1] + l2 * y[2] + l3 * y[3];
    }
  }
  for (int q = 0; q < nrhs; q++) {
    const double v = group_sum(acc[q]);
    if (g == 0) rb[q][r] = rhs_at(S, q, J * kT + r) - v;
  }
  const double *Wt = S.Winv + (size_t)J * kTT;
  double wv[4];
#pragma unroll
  for (int m = 0; m < 4; m++) wv[m] = __ldcg(Wt + (g + 8 * m) * kT + r);
  const size_t off = (size_t)J * kTT;
  double fv[4], qv[4], ev[4];
  row_of(S.F + off, fv);
  row_of(S.Q + off, qv);
  row_of(S.E + off, ev);
  csync();
  const bool hasF = J >= 1 && S.ftile[J] <= J - 1;
  for (int q = 0; q < nrhs; q++) {
    double c3 = 0.0;
#pragma unroll
    for (int m = 0; m < 4; m++) c3 = fma(wv[m], rb[q][g + 8 * m], c3);
    c3 = group_sum(c3);
    const size_t vq = (size_t)q * ls;
    double t2 = 0.0, t3 = 0.0;
    if (J >= 2) t3 = row_times(ev, ys + vq + (J - 2) * kT);
    if (g == 0) publish(cs + vq + J * kT + r, c3 - t3);
    if (J >= 2) t2 = row_times(qv, ys + vq + (J - 2) * kT);
    const double t1 = hasF ? row_times(fv, cs + vq + (J - 1) * kT) : 0.0;
    if (g == 0) publish(ys + vq + J * kT + r, (c3 - t1) - t2);
  }
  return flags[0] == 0;
}

// Diagonal tiles J = first, first + kDiagBlocks, ...: the tile, updated by
// the columns before J-2, loses panels (J, J-2) and (J, J-1) column by column as
// they are published, then it is factored.  The packed lower triangle sits in
// registers meanwhile (rows 31-s and s-1 in the lanes of slot s, 17 slots on
// eight warps); four warps poll, a column in four each, since a look at a published
// value takes longer than a column.
constexpr int kSlots = 17;
__device__ void diag_block(const ProfileSystem &S, FactorSmem &sm, int first, Waits flags) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid >> 3, q = tid & 7;
  const TrailEntries te = trail_entries(warp, lane);
  if (tid == kComputeThreads) sm.fail = 0;
  for (int J = first; J < S.nt; J += kDiagBlocks) {
    const bool fed = J > 0 && S.ftile[J] < J;
    const bool fed2 = J > 1 && S.ftile[J] < J - 1;
    const double *tile = tile_at(S, J, 0);
    if (fed) {
      if (warp >= 8) {
        const int k = warp - 8;
        for (int back = fed2 ? 2 : 1; back >= 1; back--) {
          const double *wl = (back == 2 ? S.w2stream : S.wlstream) + (size_t)(J - back) * 2 * kTT + lane;
          double a = ld_relaxed(wl + k * 2 * kT), b = ld_relaxed(wl + k * 2 * kT + kT);
          for (int c = k; c < kT; c += 4) {
            // L is published after P: once it is there, P is a load away
            if (unset(b)) {
              b = await_column(wl + c * 2 * kT + kT, flags);
              if (unset(a)) a = ld_relaxed(wl + c * 2 * kT);
            }
            if (unset(a)) a = await_column(wl + c * 2 * kT, flags);
            sm.W[c][lane] = a;
            sm.L[c][lane] = b;
            if (back == 1 && c == 0 && lane == 0 &&
                !wait_acquire(S.upd + slot_of(S, J, 0), max(J - 2 - S.ftile[J], 0), flags))
              sm.fail = 1;
            if (c + 4 < kT) {
              a = ld_relaxed(wl + (c + 4) * 2 * kT);
              b = ld_relaxed(wl + (c + 4) * 2 * kT + kT);
            }
            __syncwarp();
            named_sync(12 + k, kFactorThreads);
          }
        }
      } else {
        int rw[3], kk[3];
        double m[3], acc[3];
#pragma unroll
        for (int u = 0; u < 3; u++) {
          const int s = warp + 8 * u;
          rw[u] = -1;
          kk[u] = 0;
          if (s < kSlots) {
            if (lane < kT - s) { rw[u] = kT - 1 - s; kk[u] = lane; }
            else if (s < kSlots - 1) { rw[u] = s - 1; kk[u] = lane - (kT - s); }
          }
          m[u] = acc[u] = 0.0;
        }
        // the tile itself comes in when its other updates have (they are late
        // ones); the products are summed on their own and taken off once, as the
        // tile pairs' are: one rounding at the size of the tile's entry
        for (int k = fed2 ? 0 : kT; k < 2 * kT; k++) {
          const int c = k & (kT - 1);
          named_sync(12 + (c & 3), kFactorThreads);
#pragma unroll
          for (int u = 0; u < 3; u++)
            if (rw[u] >= 0) acc[u] = fma(sm.W[c][rw[u]], sm.L[c][kk[u]], acc[u]);
          if (k == kT) {
#pragma unroll
            for (int u = 0; u < 3; u++)
              if (rw[u] >= 0) m[u] = __ldcg(tile + rw[u] * kT + kk[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < 3; u++)
          if (rw[u] >= 0) sm.A[rw[u]][kk[u]] = m[u] - acc[u];
      }
    } else if (tid < kComputeThreads) {
      for (int k = tid; k < kTT; k += kComputeThreads) sm.A[k >> 5][k & 31] = __ldcg(tile + k);
    }
    bsync();
    if (sm.fail) return;
    if (warp < 8) eliminate_tile(sm, warp, lane, te, S.lstream + (size_t)J * kTT);
    bsync();
    if (tid < kT) {
      const int eq = J * kT + tid;
      const double d = sm.L[tid][tid];
      S.invD[eq] = __drcp_rn(d);
      S.piv[eq] = d;
      // ProfileSPDLinDirectSolver.cpp:134-138 (first pivot), :189-199; the
      // first failing pivot of the tile is reported
      const bool bad = eq < S.n && ((eq == 0) ? !(d > 0.0)
                                              : (d == 0.0 || fabs(d) <= S.min_diag_tol));
      const unsigned which = __ballot_sync(0xffffffffu, bad);
      if (which && tid == 0) {
        if (atomicCAS((int *)flags.p, 0, 4) == 0) {
          flags[1] = J * kT + __ffs(which) - 1;
          __threadfence();
          flags[0] = 3;
        }
        sm.fail = 1;
      }
    }
    if (tid < kComputeThreads) {
      double v[4];
#pragma unroll
      for (int i = 0; i < 4; i++) v[i] = 4 * q + i > r ? 0.0 : sm.L[4 * q + i][r];
      double2 *g = reinterpret_cast<double2 *>(tile_at(S, J, 0) + r * kT + 4 * q);
      g[0] = make_double2(v[0], v[1]);
      g[1] = make_double2(v[2], v[3]);
    }
    bsync();
    if (sm.fail) return;
    if (tid == 0) {
      __threadfence();
      atomicExch(S.done + slot_of(S, J, 0), 1);
    }
  }
}

// Rows 16 half .. 16 half + 15 of the tile rows I of a slot: for every column J
// from S.own_first[I] to I-1 the solve of (I, J), P L_JJ' = A and L = P D^-1, and, kLag
// columns behind it, the update of tile (I, J+1) with the published columns of
// L_J+1,J; the next solve starts from these registers.
//
// Warp 0 carries the chain of the panel's columns (lane = row): it takes the two
// newest columns off column t, publishes it and scales it.  Warps 1-7 apply a
// column to those three and more behind it and to tile (I, J+1), a row and a
// column parity a lane, column pairs w-1, w+6, w+13; so a column is not as long as
// their turns at the FP64 unit (33 warp operations at first, 17 at last, 475
// cycles on average) and the chain's latency together: 690 cycles with all eight
// warps in step, where the elimination takes 540.  Four warps poll the two streams,
// a column in four each: a look at a published value takes some 900 cycles (eight
// slots, so that a warp fills the next one while its last is read).  Four more
// write the finished panel and its digits while the others are at the next.
// Barriers: 1-4 a column is polled (to the chain), 5-7 the chain has it (to the
// others), 8-10 the others have applied it, 12-13 a panel's buffer is full, 14-15
// it is free.
constexpr int kLag = 4;                // a multiple of the four polling warps
struct RowSmem {
  double W[2][kT][17], L[2][kT][17];   // P and L by columns, two panels
  double R[kT][17];                    // columns with all but the two newest applied
  double inv[2][kT];
  double Lc[8][kT], Ln[8][kT];         // the streams' columns being applied
  int fail;
};
static_assert(sizeof(RowSmem) <= kFactorSmem, "");
__device__ void row_digits(const ProfileSystem &S, RowSmem &sm, int slot, int half,
                           Waits flags) {
  const int tid = threadIdx.x - kComputeThreads - kPollThreads, lane = tid & 31;
  int n = 0;
  for (int I = S.slot_row[slot]; I < S.nt; I = S.next_row[I])
    for (int J = S.own_first[I]; J < I; J++, n++) {
      const int buf = n & 1;
      named_sync(12 + buf, 32 + kDigitThreads);
      if (sm.fail) return;
      // the ring slot's last user has gone (a failed wait raises flags[0])
      if (lane == 0 && J >= kRing) {
        wait_geq(S.colcnt + J - kRing, S.npairs[J - kRing], flags);
        __threadfence();
      }
      __syncwarp();
      panel_store(S, sm.W[buf], sm.L[buf], sm.inv[buf], 16 * half + (tid >> 3), tid >> 3, tid & 7,
                  I - J, J);
      __syncwarp();
      if (lane == 0) {
        __threadfence();
        atomicAdd(S.done + slot_of(S, I, I - J), 1);
      }
      named_arrive(14 + buf, 32 + kDigitThreads);
    }
}

__device__ void row_block(const ProfileSystem &S, RowSmem &sm, int slot, int half,
                          Waits flags) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  if (tid == 0) sm.fail = 0;
  __syncthreads();
  if (w >= 12) {
    row_digits(S, sm, slot, half, flags);
    return;
  }
  const int r16 = lane & 15, h = lane >> 4;
  const bool trail = w >= 1 && w < 8;
  const int s0 = 2 * (w - 1) + h;          // columns s0, s0 + 14, s0 + 28
  const bool third = s0 + 28 < kT;
  auto first_columns = [&](const double (&x)[3]) {      // columns 0-2 for the chain
    if (s0 < 3) sm.R[s0][r16] = x[0];
  };
  int n = 0, front = 0;
  for (int I = S.slot_row[slot]; I < S.nt; I = S.next_row[I]) {
    const int J0 = S.own_first[I];
    if (tid == kComputeThreads) {
      // the eliminations up to the row's first column but one, one after another: the
      // slot may be idle for as long as those take, its wait's limit is for each
      while (front < J0 - 1 && wait_done(S, front, front, flags)) front++;
      front = I - 1;      // when this row's last panel is solved
      if (!wait_geq(S.upd + slot_of(S, I, I - J0), J0 - max(S.ftile[I], S.ftile[J0]), flags))
        sm.fail = 1;
      __threadfence();
    }
    bsync();
    double x[3] = {0.0, 0.0, 0.0};
    if (trail) {
      if (!sm.fail) {
        const double *t = tile_at(S, I, I - J0) + (16 * half + r16) * kT + s0;
        x[0] = __ldcg(t);
        x[1] = __ldcg(t + 14);
        if (third) x[2] = __ldcg(t + 28);
      }
      first_columns(x);
    }
    bsync();
    for (int J = J0; J < I; J++, n++) {
      const int buf = n & 1;
      if (sm.fail) {       // let the digit warps see it
        if (w == 0) named_arrive(12 + buf, 32 + kDigitThreads);
        return;
      }
      const bool more = J + 1 < I, upd = more && S.ftile[J + 1] <= J;
      const int steps = upd ? kT + kLag : kT;
      double(*W)[17] = sm.W[buf], (*L)[17] = sm.L[buf];
      if (w >= 8) {
        const int k = w - 8;
        const double *st = S.lstream + (size_t)J * kTT + lane;
        const double *ll = S.wlstream + ((size_t)J * 2 * kTT + kT) + lane;
        double v = ld_relaxed(st + k * kT), b = 0.0;
        for (int t = k; t < steps; t += 4) {
          if (t < kT) {
            if (lane >= t) {
              if (unset(v)) v = await_column(st + t * kT, flags);
              sm.Lc[t & 7][lane] = v;
            }
            if (t + 4 < kT && lane >= t + 4) v = ld_relaxed(st + (t + 4) * kT);
          }
          if (upd) {
            const int c = t - kLag;
            if (c >= 0) {
              if (unset(b)) b = await_column(ll + c * 2 * kT, flags);
              sm.Ln[t & 7][lane] = b;
            }
            if (c + 4 < kT) b = ld_relaxed(ll + (c + 4) * 2 * kT);
          }
          // tile (I, J+1) with the updates of the columns before J
          if (t == steps - 8 && more && lane == 0 &&
              !wait_acquire(S.upd + slot_of(S, I, I - J - 1),
                            max(J - max(S.ftile[I], S.ftile[J + 1]), 0), flags))
            sm.fail = 1;
          __syncwarp();
          named_sync(1 + k, 64);
        }
        if (!more && k == 0 && flags[0] != 0 && lane == 0) sm.fail = 1;
      } else if (w == 0) {
        double *wl = J + 2 < I || h != 0 ? nullptr
                                         : (J + 1 == I ? S.wlstream : S.w2stream) +
                                               (size_t)J * 2 * kTT + 16 * half + r16;
        if (n >= 2) named_sync(14 + buf, 32 + kDigitThreads);
        double p1 = 0.0, p2 = 0.0;           // columns t-1, t-2
        int m3 = 0;                          // t mod 3
        for (int t = 0; t < steps; t++) {
          if (t >= 3) named_sync(8 + m3, kComputeThreads);
          double p = 0.0;
          if (t < kT) {
            p = sm.R[t][r16];
            if (t >= 2) p = fma(-p2, sm.Lc[(t - 2) & 7][t], p);
            if (t >= 1) p = fma(-p1, sm.Lc[(t - 1) & 7][t], p);
            W[t][r16] = p;
            if (wl) publish(wl + t * 2 * kT, p);
          }
          named_sync(1 + (t & 3), 64);
          if (t < kT) {
            const double inv = sm.Lc[t & 7][t], v = p * inv;
            L[t][r16] = v;
            if (lane == 0) sm.inv[buf][t] = inv;
            if (wl) publish(wl + t * 2 * kT + kT, v);
          }
          named_arrive(5 + m3, kComputeThreads);
          p2 = p1;
          p1 = p;
          m3 = m3 == 2 ? 0 : m3 + 1;
        }
        named_arrive(12 + buf, 32 + kDigitThreads);
      } else {
        double acc[3] = {0.0, 0.0, 0.0}, xn[3] = {0.0, 0.0, 0.0};
        int m3 = 0;
        for (int c = 0; c < steps; c++) {
          named_sync(5 + m3, kComputeThreads);
          if (c < kT - 3) {
            const double wc = W[c][r16];
            const double *lc = sm.Lc[c & 7];
#pragma unroll
            for (int u = 0; u < 3; u++) {
              const int s = s0 + 14 * u;
              if (s >= c + 3 && s < kT) {
                x[u] = fma(-wc, lc[s], x[u]);
                if (s == c + 3) sm.R[s][r16] = x[u];
              }
            }
          }
          if (c < steps - 3) named_arrive(8 + m3, kComputeThreads);
          if (upd && c >= kLag) {
            const double pc = W[c - kLag][r16];
            const double *ln = sm.Ln[c & 7];
            acc[0] = fma(pc, ln[s0], acc[0]);
            acc[1] = fma(pc, ln[s0 + 14], acc[1]);
            if (third) acc[2] = fma(pc, ln[s0 + 28], acc[2]);
          }
          if (c == steps - 8 && more) {
            const double *g = tile_at(S, I, I - J - 1) + (16 * half + r16) * kT + s0;
            xn[0] = __ldcg(g);
            xn[1] = __ldcg(g + 14);
            if (third) xn[2] = __ldcg(g + 28);
          }
          m3 = m3 == 2 ? 0 : m3 + 1;
        }
#pragma unroll
        for (int u = 0; u < 3; u++) x[u] = xn[u] - acc[u];
        first_columns(x);
      }
      bsync();
    }
  }
}

// The other blocks: tasks from the list.  Warp 8 draws the next task and
// waits for its operands while warps 0-7 run the present one (barriers 7-8:
// a task is ready, 5-6: its slot is free again); during a panel, which lasts
// as long as its column's elimination, it polls the column instead.
__device__ void worker_block(const ProfileSystem &S, FactorSmem &sm, Waits flags) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 8) {
    int pending = 0;
    bool last_long = false;
    for (int it = 0;; it++) {
      const int s = it & 1;
      while (pending == 2 || (pending && last_long)) {
        named_sync(5 + ((it - pending) & 1), kFactorThreads);
        pending--;
      }
      int type = -1;
      if (lane == 0) {
        const int k = atomicAdd(S.next_task, 1);
        int4 tk = make_int4(-1, 0, 0, 0);
        if (k < S.ntasks && flags[0] == 0) {
          tk = S.tasks[k];
          if (!wait_task(S, tk, flags)) tk.x = -1;
        }
        sm.task[s] = tk;
        type = tk.x;
        __threadfence();
      }
      type = __shfl_sync(0xffffffffu, type, 0);
      __syncwarp();
      named_arrive(7 + s, kFactorThreads);
      if (type < 0) return;
      if (type == kPanel) panel_poll(S, sm, sm.task[s].w, lane, flags);
      last_long = type == kPanel;
      pending++;
    }
  }
  for (int it = 0;; it++) {
    const int s = it & 1;
    named_sync(7 + s, kFactorThreads);
    const int4 t = sm.task[s];
    if (t.x < 0) return;
    if (t.x == kPanel) panel_task(S, sm, t.y, t.w, tid);
    else if (t.x == kPair) pair_task(S, t.w, t.y - t.w, t.z - t.w, tid);
    else if (t.x == kInverse) inverse_task(S, sm, t.w, tid);
    else if (t.x == kCouple) coupling_task(S, sm, t.w, t.z, tid);
    else if (t.x == kCouple2) second_coupling_task(S, sm, t.w, t.z, tid);
    else forward_row(S, t.w, reinterpret_cast<double (*)[kT]>(&sm.A[0][0]), flags);
    csync();
    if (tid == 0) {
      __threadfence();
      if (t.x == kPanel) {
        atomicExch(S.done + slot_of(S, t.y, t.y - t.w), 1);
      } else if (t.x == kPair) {
        atomicAdd(S.upd + slot_of(S, t.y, t.y - t.z), 1);
        atomicAdd(S.colcnt + t.w, 1);
      } else if (t.x == kInverse) {
        atomicExch(S.cplw + t.w, 1);
      } else if (t.x == kCouple) {
        atomicAdd(S.cpl + t.w, 1);
      } else if (t.x == kCouple2 && t.z == 0) {
        atomicExch(S.cplq + t.w, 1);
      }
    }
    __syncwarp();
    named_arrive(5 + s, kFactorThreads);
  }
}

__global__ void __launch_bounds__(kBlockThreads, 1) k_prof_factor(ProfileSystem S) {
  extern __shared__ __align__(16) unsigned char dyn[];
  FactorSmem &sm = *reinterpret_cast<FactorSmem *>(dyn);
  __shared__ int ticket;
  const Waits flags{S.flags, S.wait_ns};
  if (threadIdx.x == 0) ticket = atomicAdd(S.next_task + 1, 1);
  __syncthreads();
  const int t = ticket, row = t - kDiagBlocks;
  if (row >= 0 && row < 2 * S.nslots) {
    row_block(S, *reinterpret_cast<RowSmem *>(dyn), row >> 1, row & 1, flags);
    return;
  }
  if (t < kDiagBlocks) {
    if (threadIdx.x < kComputeThreads + kPollThreads) diag_block(S, sm, t, flags);
  } else if (threadIdx.x < kFactorThreads) {
    worker_block(S, sm, flags);
  }
}

__global__ void __launch_bounds__(kPipeThreads) k_prof_solve_pipe(ProfileSystem S, int nrhs,
                                                                  double *ys, double *cs,
                                                                  double *xs, double *ds,
                                                                  int backward_only) {
  __shared__ double rv[2][4][kT];
  const Waits flags{S.flags, S.wait_ns};
  if (flags[0] != 0) return;                    // the factorisation failed
  const int tid = threadIdx.x;
  const int r = tid >> 3, g = tid & 7;          // tile row, column group (4 columns)
  const int nt = S.nt, W = S.W, P = gridDim.x, ls = nt * kT;
  // reduce over the eight column groups of a row (lanes r*8 .. r*8+7)
  auto group_sum = [](double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
  };
  // this thread's four entries of row r of a 32 x 32 matrix (loaded ahead
  // of the waits), and their product with the vector published at p
  auto row_of = [&](const double *M, double (&mv)[4]) {
#pragma unroll
    for (int m = 0; m < 4; m++) mv[m] = __ldcg(M + r * kT + g + 8 * m);
  };
  auto row_times = [&](const double (&mv)[4], const double *p) {
    double v[4];
    await4(p + g, v, flags);
    double t = 0.0;
#pragma unroll
    for (int m = 0; m < 4; m++) t = fma(mv[m], v[m], t);
    return group_sum(t);
  };
  int it = 0;                                   // rv is double-buffered by iteration
  // ---------------- forward (done by the factorisation when backward_only)
  for (int J = blockIdx.x; J < nt && !backward_only; J += P, it++) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const int ohi = min(W, J - S.ftile[J]);
    for (int o = ohi; o >= 3; o--) {
      const double *Lt = tile_at(S, J, o) + r * kT + g;
      const double l0 = __ldcg(Lt), l1 = __ldcg(Lt + 8), l2 = __ldcg(Lt + 16), l3 = __ldcg(Lt + 24);
      for (int q = 0; q < nrhs; q++) {
        double y[4];
        await4(ys + (size_t)q * ls + (J - o) * kT + g, y, flags);
        acc[q] += l0 * y[0] + l1 * y[1] + l2 * y[2] + l3 * y[3];
      }
    }
    double(*rb)[kT] = rv[it & 1];
    for (int q = 0; q < nrhs; q++) {
      const double v = group_sum(acc[q]);
      if (g == 0) rb[q][r] = rhs_at(S, q, J * kT + r) - v;
    }
    const double *Wt = S.Winv + (size_t)J * kTT;
    double wv[4];
#pragma unroll
    for (int m = 0; m < 4; m++) wv[m] = __ldcg(Wt + (g + 8 * m) * kT + r);
    const size_t off = (size_t)J * kTT;
    double fv[4], qv[4], ev[4];
    row_of(S.F + off, fv);
    row_of(S.Q + off, qv);
    row_of(S.E + off, ev);
    __syncthreads();
    const bool hasF = J >= 1 && S.ftile[J] <= J - 1;
    for (int q = 0; q < nrhs; q++) {
      double c3 = 0.0;
#pragma unroll
      for (int m = 0; m < 4; m++) c3 = fma(wv[m], rb[q][g + 8 * m], c3);
      c3 = group_sum(c3);
      const size_t vq = (size_t)q * ls;
      // c_J first: it needs only y_J-2, and row J+1 waits for it
      double t2 = 0.0, t3 = 0.0;
      if (J >= 2) t3 = row_times(ev, ys + vq + (J - 2) * kT);
      if (g == 0) publish(cs + vq + J * kT + r, c3 - t3);
      if (J >= 2) t2 = row_times(qv, ys + vq + (J - 2) * kT);
      const double t1 = hasF ? row_times(fv, cs + vq + (J - 1) * kT) : 0.0;
      if (g == 0) publish(ys + vq + J * kT + r, (c3 - t1) - t2);
    }
  }
  // ---------------- backward
  const int jlast = blockIdx.x + ((nt - 1 - (int)blockIdx.x) / P) * P;
  for (int J = jlast; J >= 0; J -= P, it++) {
    if (J >= nt) continue;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const int ohi = min(W, nt - 1 - J);
    // column c = r of the result; rows g, g+8, g+16, g+24 of tile (J+o, J)
    for (int o = ohi; o >= 3; o--) {
      if (S.ftile[J + o] > J) continue;
      const double *Lt = tile_at(S, J + o, o) + r;
      const double l0 = __ldcg(Lt + g * kT), l1 = __ldcg(Lt + (g + 8) * kT);
      const double l2 = __ldcg(Lt + (g + 16) * kT), l3 = __ldcg(Lt + (g + 24) * kT);
      for (int q = 0; q < nrhs; q++) {
        double xv[4];
        await4(xs + (size_t)q * ls + (J + o) * kT + g, xv, flags);
        acc[q] += l0 * xv[0] + l1 * xv[1] + l2 * xv[2] + l3 * xv[3];
      }
    }
    double(*rb)[kT] = rv[it & 1];
    for (int q = 0; q < nrhs; q++) {
      const double v = group_sum(acc[q]);
      // z_J = D^-1 y_J (ProfileSPD divides by the pivots before the back
      // sweep); y_J[r] was published by this same thread in the forward sweep
      if (g == 0)
        rb[q][r] = ld_relaxed(ys + (size_t)q * ls + J * kT + r) * S.invD[J * kT + r] - v;
    }
    const double *Wt = S.Winv + (size_t)J * kTT;
    double wv[4];
#pragma unroll
    for (int m = 0; m < 4; m++) wv[m] = __ldcg(Wt + r * kT + g + 8 * m);
    const size_t off = (size_t)J * kTT;
    double gv[4], rv4[4], hv[4];
    row_of(S.G + off, gv);
    row_of(S.R + off, rv4);
    row_of(S.H + off, hv);
    __syncthreads();
    const bool hasG = J + 1 < nt && S.ftile[J + 1] <= J;
    for (int q = 0; q < nrhs; q++) {
      double c3 = 0.0;
#pragma unroll
      for (int m = 0; m < 4; m++) c3 = fma(wv[m], rb[q][g + 8 * m], c3);
      c3 = group_sum(c3);
      const size_t vq = (size_t)q * ls;
      // c'_J first: it needs only x_J+2, and row J-1 waits for it
      double t2 = 0.0, t3 = 0.0;
      if (J + 2 < nt) t3 = row_times(hv, xs + vq + (J + 2) * kT);
      if (g == 0) publish(ds + vq + J * kT + r, c3 - t3);
      if (J + 2 < nt) t2 = row_times(rv4, xs + vq + (J + 2) * kT);
      const double t1 = hasG ? row_times(gv, ds + vq + (J + 1) * kT) : 0.0;
      if (g == 0) {
        const double xj = (c3 - t1) - t2;
        publish(xs + vq + J * kT + r, xj);
        if (J * kT + r < S.n) S.x[q][J * kT + r] = xj;
      }
    }
  }
}

}  // namespace

int profile_plan(int n, const int *rowptr, const int *colidx, std::vector<int> &ftile, int &nt,
                 int &W) {
  nt = (n + kT - 1) / kT;
  ftile.assign(nt > 0 ? nt : 1, 0);
  W = 0;
  for (int I = 0; I < nt; I++) {
    int f = I;
    for (int i = I * kT; i < n && i < (I + 1) * kT; i++) {
      const int j = colidx[rowptr[i]];   // first column of row i (sorted)
      if (j / kT < f) f = j / kT;
    }
    ftile[I] = f;
    if (I - f > W) W = I - f;
  }
  return 0;
}

// Which tile rows the row blocks keep, and from which column: a row from its first
// column to its last takes a slot of two blocks.  All rows where 28 slots are
// enough: a row that takes its panels and products from the list needs 14.8 us a
// column, and the elimination waits for the slowest (one long row behind a
// constraint held up a 64 x 16 quad block for 150 us).  Beyond that only the two rows
// next to the diagonal are kept: the tile pairs of the list, some 2.7 us each on the
// blocks that are left, then take longer a column than the rows'.  With all rows
// kept and with two, us a tile column: 36 below the diagonal tile 14.1 and 15.9, 42
// 15.2 and 16.4, 49 18.3 and 17.3, 74 148 and 25.2 -- so on 152 SMs the two meet
// near 45, and the line, which no envelope was measured beyond when it was drawn,
// lies on the safe side of it.
// first[I] >= I: no column; rows of a slot in the order of their first columns.
// A device of fewer SMs than 152 gets its share of the slots, so that blocks for the
// list are left; two rows next to the diagonal take two slots whatever the system.
constexpr int kMaxSlots = 28;
int profile_rows(int nt, const std::vector<int> &ftile, int sms, std::vector<int> &first,
                 std::vector<int> &next, std::vector<int> &slot_row) {
  const int most = std::min(kMaxSlots, (sms - kDiagBlocks) * kMaxSlots / (152 - kDiagBlocks));
  for (int reach : {nt, 2}) {
    first.resize(nt);
    next.assign(nt, nt);
    slot_row.clear();
    std::vector<int> order, last;      // last row of each slot
    for (int I = 0; I < nt; I++) {
      first[I] = std::max(ftile[I], I - reach);
      if (first[I] < I) order.push_back(I);
    }
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return first[a] < first[b]; });
    for (int I : order) {
      size_t k = 0;
      while (k < last.size() && last[k] > first[I]) k++;
      if (k == last.size()) {
        last.push_back(I);
        slot_row.push_back(I);
      } else {
        next[last[k]] = I;
        last[k] = I;
      }
    }
    if ((int)slot_row.size() <= most) break;
  }
  return kDiagBlocks + 2 * (int)slot_row.size() + 1;
}

// The dataflow order of the list's tasks (type, I, K, J): the stream's blocks
// run the diagonal tiles, the row blocks' panels, column J's updates of the next
// two diagonal tiles and those rows' updates of tile column J+1 by column J.  Column J: the
// updates of column J-1 that reach column J+1 (the next diagonal tile's last but
// one first), the other panels, column J's other updates of column J+1, the rest
// of column J-1's trailing update, and the coupling matrices and forward step two
// columns back.  npairs: tile pairs of each column in the list.
void profile_tasks(int nt, int W, const std::vector<int> &ftile, const std::vector<int> &first,
                   std::vector<int> &tasks, std::vector<int> &npairs) {
  tasks.clear();
  npairs.assign(std::max(nt, 1), 0);
  auto emit = [&](int type, int I, int K, int J) {
    tasks.push_back(type); tasks.push_back(I); tasks.push_back(K); tasks.push_back(J);
    if (type == kPair) npairs[J]++;
  };
  // the updates of column J whose target column is J+b for b in [blo, bhi]; not
  // the stream's: (J+1, J+1), (J+2, J+2) and the row blocks' of column J+1
  auto updates = [&](int J, int blo, int bhi) {
    if (J < 0) return;
    const int omax = std::min(W, nt - 1 - J);
    for (int b = blo; b <= std::min(bhi, omax); b++) {
      if (ftile[J + b] > J) continue;
      for (int a = b; a <= omax; a++) {
        if (ftile[J + a] > J || (a == b && b <= 2)) continue;
        if (b == 1 && first[J + a] <= J) continue;
        emit(kPair, J + a, J + b, J);
      }
    }
  };
  auto couple = [&](int J) {
    if (J < 0) return;
    emit(kInverse, J, J, J);
    for (int p = 0; p < 4; p++) emit(kCouple, J, p, J);
    emit(kCouple2, J, 0, J);
    if (J >= 1) emit(kCouple2, J - 1, 1, J - 1);
    if (J == nt - 1) emit(kCouple2, J, 1, J);
    emit(kForward, J, J, J);
  };
  for (int J = 0; J < nt; J++) {
    updates(J - 1, 2, 2);
    const int omax = std::min(W, nt - 1 - J);
    for (int o = 1; o <= omax; o++)
      if (ftile[J + o] <= J && first[J + o] > J) emit(kPanel, J + o, J + o, J);
    updates(J, 1, 1);
    updates(J - 1, 3, W);
    couple(J - 2);
  }
  for (int J = std::max(nt - 2, 0); J < nt; J++) couple(J);
}

size_t profile_tile_doubles(int nt, int W) { return (size_t)nt * (W + 1) * kTT; }
size_t profile_digit_bytes(int W) { return (size_t)kRing * W * kSlotBytes; }
int profile_tile_edge() { return kT; }

int profile_device(int *sms) {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess &&
                 cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
                 cudaFuncSetAttribute(k_prof_factor, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kFactorSmem) == cudaSuccess
             ? 0 : XG_ECUDA;
}

int profile_factor(const ProfileSystem &S, cudaStream_t s) {
  if (S.n == 0) return 0;
  if (S.fwd_nrhs < 1 || S.fwd_nrhs > 4) return XG_EINVAL;
  // the sweeps' values: forward ones published inside the factorisation,
  // backward ones by the solve behind it
  const size_t nsweep = 4 * (size_t)S.fwd_nrhs * S.nt * kT;
  const long nprep = std::min<long>(8 * (long)S.sms, (long)S.nt * kT / 8);
  k_prof_prepare<<<(int)std::max<long>(nprep, 1), 256, 0, s>>>(S, S.counter_bytes / sizeof(int),
                                                               nsweep);
  if (cudaGetLastError() != cudaSuccess) return XG_ECUDA;
  // all blocks co-resident: the stream waits for list tasks and they for it
  const int nb = (int)std::min<long>(S.sms, kDiagBlocks + 2 * S.nslots + (long)S.ntasks);
  ProfileSystem Sv = S;
  void *args[] = {(void *)&Sv};
  return cudaLaunchCooperativeKernel((void *)k_prof_factor, dim3(nb), dim3(kBlockThreads), args,
                                     kFactorSmem, s) == cudaSuccess
             ? 0 : XG_ECUDA;
}

int profile_status(const ProfileSystem &S, cudaStream_t s, int *bad_eq) {
  if (bad_eq) *bad_eq = -1;
  if (S.n == 0) return 0;
  int hflags[4];
  if (cudaMemcpyAsync(hflags, S.flags, sizeof hflags, cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return XG_ECUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return XG_ECUDA;
  if (bad_eq && hflags[0] == 3) *bad_eq = hflags[1];
  return hflags[0] != 0 ? XG_ESOLVE : 0;   // a pivot check failed, or a wait timed out
}

int profile_solve(const ProfileSystem &S, int nrhs, cudaStream_t s, bool backward_only) {
  if (S.n == 0) return 0;
  if (nrhs < 1 || nrhs > 4) return XG_EINVAL;
  const size_t ls = (size_t)S.nt * kT;
  double *ys = S.sweep, *cs = ys + (size_t)nrhs * ls, *xs = cs + (size_t)nrhs * ls;
  double *ds = xs + (size_t)nrhs * ls;
  // the sweeps' published values start unset (behind a factorisation that ran
  // the forward sweep they are)
  if (!backward_only) {
    if (cudaMemsetAsync(ys, 0xFF, 4 * (size_t)nrhs * ls * sizeof(double), s) != cudaSuccess)
      return XG_ECUDA;
    if (cudaMemsetAsync(S.flags, 0, 4 * sizeof(int), s) != cudaSuccess) return XG_ECUDA;
  }
  ProfileSystem Sv = S;
  int bonly = backward_only ? 1 : 0;
  void *args[] = {(void *)&Sv, (void *)&nrhs, (void *)&ys, (void *)&cs,
                  (void *)&xs, (void *)&ds,   (void *)&bonly};
  return cudaLaunchCooperativeKernel((void *)k_prof_solve_pipe, dim3(std::min(kPipeBlocks, S.nt)),
                                     dim3(kPipeThreads), args, 0, s) == cudaSuccess
             ? 0 : XG_ECUDA;
}

}  // namespace xg
