// xg_block_stream.h -- the node-block matrix on its way through a warp's ring of
// shared-memory stages (k_pcg_nodes, xg_pcg.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "xg_internal.h"

namespace xg {

namespace {

constexpr unsigned long long kCopyTimeoutNs = 2000000000ull;  // 2 s

// By block order: warps a block, blocks a ring stage, stages a warp, stages
// whose columns' z is gathered ahead.  A stage is one bulk copy (3,072, 2,304, 2,432
// and 9,344 bytes), the rings 180 to 192 KiB of an SM's shared memory.
template <int KB> struct NodeShape;
template <> struct NodeShape<1> { static constexpr int kWarps = 16, kGroup = 8, kRing = 4, kAhead = 2; };
template <> struct NodeShape<2> { static constexpr int kWarps = 16, kGroup = 2, kRing = 5, kAhead = 4; };
template <> struct NodeShape<3> { static constexpr int kWarps = 16, kGroup = 1, kRing = 5, kAhead = 4; };
template <> struct NodeShape<6> { static constexpr int kWarps = 4, kGroup = 1, kRing = 5, kAhead = 4; };

// A block of a slice: entry (a, b) of the 32 rows' blocks side by side, and the
// column nodes.  The node-block copy is an array of these, in the slices' order.
template <int KB>
struct BlockRecord {
  float2 v[KB * KB][32];
  int col[32];
};

// The bulk copies and their barriers (a host build brings its own).
#ifdef __CUDACC__
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *b) {
  asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes,
                                          unsigned long long *b) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(b))
      : "memory");
}
// Whether the phase is over (it may look for a short while).
__device__ __forceinline__ bool mbar_try(unsigned long long *b, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return done != 0;
}
#endif

// A warp's share of the matrix, streamed through its ring: its slices one after
// another, of each the groups of kGroup blocks part, part + SP, ..., and from
// the start again for the next SpMV, so that a ring's worth of the next
// iteration's blocks is there when its z is.  A share no longer than the ring
// is loaded once.  Lane 0 issues.
//
// A copy that has not come within the limit ends the stream (ok, the warp's own):
// what lies in its stage is no record (its columns would send the gathers
// anywhere), so the stage's columns become node 0, and no wait follows; no stage is
// filled again, and drain() waits for the copies still in flight, all within one
// limit more.
template <int KB, int SP, bool kOne>
struct BlockStream {
  static constexpr int kGroup = NodeShape<KB>::kGroup, kRing = NodeShape<KB>::kRing;
  using Record = BlockRecord<KB>;
  const PcgSystem &S;
  Record (*rec)[kGroup];        // the warp's ring
  unsigned long long *full;     // a barrier a stage, then where lane 0 lost a copy
  int lane, part, first, stride, ns;
  int total, len;               // groups of the share, stages in use
  bool ring;                    // more groups than stages
  int oldest, next;             // stages of the oldest group and the one to wait for next,
  unsigned phase;               // and the latter's barrier's phase
  int left, is, wide;           // groups left to issue of the slice in turn, the slice, its
  const Record *src;            // blocks left, and the next group

  __device__ __forceinline__ int width(int s) const {
    return (int)((__ldg(S.nb_off + s + 1) - __ldg(S.nb_off + s)) >> 5);
  }
  __device__ __forceinline__ int groups(int w) const {
    const int g = (w + kGroup - 1) / kGroup;
    return g > part ? (g - part + SP - 1) / SP : 0;
  }
  __device__ __forceinline__ void next_slice(int s) {
    for (is = s;; is += stride) {
      if (is >= ns) is = first;
      wide = width(is);
      left = groups(wide);
      if (left > 0) break;
    }
    wide -= kGroup * part;
    src = reinterpret_cast<const Record *>(S.nb_vals) + (__ldg(S.nb_off + is) >> 5) + kGroup * part;
  }
  __device__ void start() {
    total = 0;
    for (int s = first; s < ns; s += stride) total += groups(width(s));
    len = min(total, kRing);
    ring = total > kRing;
    if (lane == 0) full[kRing] = 0;
    __syncwarp();
    oldest = next = 0;
    phase = 0u;
    if (total > 0) {
      next_slice(first);
      for (int k = 0; k < len; k++) issue(k, true);
    }
  }
  __device__ __forceinline__ void issue(int k, bool ok) {
    if (lane == 0 && ok) {
      const unsigned bytes =
          (unsigned)sizeof(Record) * (kGroup == 1 ? 1u : (unsigned)min(kGroup, wide));
      mbar_expect(full + k, bytes);
      bulk_load(rec[k], src, bytes, full + k);
    }
    src += SP * kGroup;
    wide -= SP * kGroup;
    if (--left == 0) {
      if (kOne) {      // the same slice from its start
        src -= (long)SP * kGroup * total;
        wide += SP * kGroup * total;
        left = total;
      } else {
        next_slice(is + stride);
      }
    }
  }
  // the next group, once it has come
  __device__ __forceinline__ const Record *get(bool &ok) {
    ok &= wait(ok);
    const Record *r = rec[next];
    advance();
    return r;
  }
  __device__ __forceinline__ void advance() {
    if (++next == len) {
      next = 0;
      phase ^= (unsigned)ring;
    }
  }
  // the warp is done with the oldest group
  __device__ __forceinline__ void release(bool ok) {
    __syncwarp();
    if (ring) issue(oldest, ok);
    if (++oldest == len) oldest = 0;
  }
  __device__ __forceinline__ bool wait(bool ok) {
    unsigned long long t0 = 0;
    for (int tries = 0;; tries++) {
      if (mbar_try(full + next, phase)) return true;
      if (ok) {
        if ((tries & 63) != 63) continue;
        const unsigned long long now = global_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 <= kCopyTimeoutNs) continue;
        if (lane == 0)
          full[kRing] = 1u | (unsigned)next << 8 | (unsigned)oldest << 16 | phase << 24;
      }
      for (int u = 0; u < kGroup; u++) rec[next][u].col[lane] = 0;
      return false;
    }
  }
  // the copies in flight have come: nothing may land after the block is gone
  __device__ void drain() {
    if (lane != 0 || len == 0) return;
    if (full[kRing] != 0) {          // as lane 0 stood when it lost one
      const unsigned at = (unsigned)full[kRing];
      next = at >> 8 & 255u;
      oldest = at >> 16 & 255u;
      phase = at >> 24 & 1u;
    }
    // (a ring's groups taken and not yet released have come)
    const unsigned long long end = global_ns() + kCopyTimeoutNs;
    for (int k = ring ? (next - oldest + len) % len : 0; k < len; k++) {
      for (int t = 0; !mbar_try(full + next, phase); t++)
        if ((t & 63) == 63 && global_ns() > end) break;
      advance();
    }
  }
};

}  // namespace
}  // namespace xg
