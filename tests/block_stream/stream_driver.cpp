// Host driver for tests/test_block_stream.py: runs xg::BlockStream on one lane
// with bulk copies that arrive when they are waited for -- or never -- and
// counts what must not happen.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <random>
#include <vector>

#undef __noinline__
#define __noinline__

namespace {
struct Barrier {
  int armed = 0, done = 0;      // copies started, copies arrived
  bool lost = false;
  void *dst = nullptr;
  const void *src = nullptr;
  unsigned bytes = 0;
};
std::map<unsigned long long *, Barrier> g_bar;
int g_copy, g_lose, g_looks, g_bad;
bool g_failed;
unsigned long long g_now;

template <typename T> T __ldg(const T *p) { return *p; }
void __syncwarp() {}
using std::min;
unsigned long long global_ns() {                   // 1 ms a look
  g_looks++;
  return g_now += 1000000;
}
void mbar_expect(unsigned long long *b, unsigned bytes) {
  Barrier &B = g_bar[b];
  if (B.armed != B.done || g_failed) g_bad |= 1;   // filled again while a copy is on its way
  B.armed++;
  B.bytes = bytes;
}
void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *b) {
  Barrier &B = g_bar[b];
  if (B.bytes != bytes) g_bad |= 2;
  B.dst = dst;
  B.src = src;
  B.lost = g_copy++ == g_lose;
}
bool mbar_try(unsigned long long *b, unsigned parity) {
  Barrier &B = g_bar[b];
  if (B.armed != B.done && !B.lost) {
    std::memcpy(B.dst, B.src, B.bytes);
    B.done++;
  }
  return B.done > 0 && ((B.done - 1) & 1) == (int)parity;
}
}  // namespace

#include "../../xara_gb300/csrc/xg_block_stream.h"

template <int KB, int SP, bool kOne>
static int run(int ns, int stride, int passes, int lose, unsigned seed) {
  using Stream = xg::BlockStream<KB, SP, kOne>;
  using Record = typename Stream::Record;
  constexpr int kGroup = Stream::kGroup, kRing = Stream::kRing, kAhead = xg::NodeShape<KB>::kAhead;
  std::mt19937 rng(seed);
  std::vector<long> off(ns + 1, 0);
  for (int s = 0; s < ns; s++) off[s + 1] = off[s] + 32 * (long)(rng() % 23);
  const long nrec = off[ns] / 32;
  std::vector<Record> recs(nrec + 1);
  for (long k = 0; k < nrec; k++) recs[k].col[0] = (int)k;
  xg::PcgSystem S{};
  S.nb_off = off.data();
  S.nb_vals = reinterpret_cast<float2 *>(recs.data());
  int errors = 0;
  for (int part = 0; part < SP; part++) {
    std::vector<Record> ring((size_t)kRing * kGroup);
    for (auto &r : ring) r.col[0] = 1 << 30;           // no record
    unsigned long long full[8];
    g_bar.clear();
    g_copy = g_looks = g_bad = 0;
    g_lose = lose;
    g_failed = false;
    const int last = kOne ? 1 : ns;
    Stream B{S, reinterpret_cast<Record(*)[kGroup]>(ring.data()), full, 0, part, 0, kOne ? ns : stride,
             last};
    B.start();
    bool ok = true;
    for (int it = 0; it < passes; it++)
      for (int s = 0; s < last; s += kOne ? ns : stride) {
        const int width = B.width(s), groups = kOne ? B.total : B.groups(width);
        auto gather = [&](int g) {
          if (g >= groups) return;
          const Record *r = B.get(ok);
          g_failed = !ok;
          for (int u = 0; u < kGroup; u++) {
            const int k = kGroup * (part + SP * g) + u;
            if (k >= width) continue;
            const int col = r[u].col[0];               // a record's or, of a lost one, node 0
            errors += ok ? col != (int)(off[s] / 32) + k : col < 0 || col > nrec;
          }
        };
        for (int u = 0; u < kAhead; u++) gather(u);
        for (int g = 0; g < groups; g += kAhead)
          for (int u = 0; u < kAhead && g + u < groups; u++) {
            B.release(ok);
            gather(g + u + kAhead);
          }
      }
    if (lose < 0 && !ok) errors++;
    B.drain();
    for (auto &b : g_bar)
      if (b.second.armed != b.second.done && !b.second.lost) errors++;   // still on its way
    // two limits of 2,000 looks at most, and the start's and the drain's own
    errors += g_bad + (g_looks > 2 * 2000 + 8 + kRing);
  }
  return errors;
}

extern "C" int stream_errors(int kb, int sp, int one, int ns, int stride, int passes, int lose,
                             unsigned seed) {
#define CASE(K, P)                                                                  \
  if (kb == K && sp == P)                                                           \
    return one ? run<K, P, true>(ns, stride, passes, lose, seed)                    \
               : run<K, P, false>(ns, stride, passes, lose, seed)
  CASE(1, 1); CASE(1, 8); CASE(2, 1); CASE(2, 4); CASE(3, 1); CASE(3, 2); CASE(3, 8);
  CASE(6, 1); CASE(6, 4);
  return -1;
}
