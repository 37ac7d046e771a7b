// The parallel block index's plan (gzfp_index_plan.h) over many streams, and
// over devices with less memory than it asks for: the workspace stays within
// its limit, its parts do not overlap, its batches cover the stream, and with
// ever less memory there are ever shorter batches, down to a few segments.
#include <math.h>
#include <stdio.h>

#include <algorithm>
#include <random>
#include <vector>

#include "gzfp_index_plan.h"

using namespace gzfp;

static int fails = 0;
#define CHECK(c, ...)                                 \
  do {                                                \
    if (!(c) && fails++ < 20) {                       \
      printf("line %d: %s: ", __LINE__, #c);          \
      printf(__VA_ARGS__);                            \
      printf("\n");                                   \
    }                                                 \
  } while (0)

static void check(const IndexPlan& p, uint64_t span) {
  CHECK(p.bytes <= kIndexWorkspace, "%zu", p.bytes);
  CHECK(p.seg_bits > p.win && p.seg_bits <= 32768 && (p.seg_bits & (p.seg_bits - 1)) == 0, "%u",
        p.seg_bits);
  CHECK(p.nseg * p.seg_bits >= span && (p.nseg - 1) * p.seg_bits < span, "%llu",
        (unsigned long long)span);
  CHECK(p.per >= 1 && p.per <= p.nseg && (uint64_t)p.per * p.seg_bits <= kIndexBatchBits, "%u", p.per);
  CHECK((uint64_t)p.n1 * p.fan >= p.per && (uint64_t)p.n2 * p.fan >= p.n1 && p.n1 <= 65535, "%u", p.n1);
  // parts as the kernels use them: begin, bytes
  const size_t maps = (size_t)p.win + 1, nodes = (size_t)p.per + p.n1 + p.n2;
  std::vector<std::pair<size_t, size_t>> part = {
      {p.state, sizeof(IndexState)}, {p.counters, 8}, {p.table, (size_t)p.per * p.seg_bits * 2},
      {p.first, (size_t)p.per * (p.win + 1) * 4 + 4},  // every window bit, and block 0's again
      {p.exits, p.per * maps * 4}, {p.hops1, p.n1 * maps * 8}, {p.hops2, p.n2 * maps * 8},
      {p.entry, nodes * 4}, {p.base, nodes * 8}, {p.bytes, 0}};
  std::sort(part.begin(), part.end());
  for (size_t i = 0; i + 1 < part.size(); i++) {
    CHECK(part[i].first % 256 == 0, "%zu", part[i].first);
    CHECK(part[i].first + part[i].second <= part[i + 1].first, "%zu + %zu", part[i].first,
          part[i].second);
  }
}

int main() {
  std::mt19937_64 rng(1);
  auto upto = [&](double lo, double hi) {  // spread over the logarithm
    const double u = (double)(rng() >> 11) / 9007199254740992.0;
    return (uint64_t)(lo * pow(hi / lo, u));
  };
  for (int i = 0; i < 20000; i++) {
    const uint32_t win = (uint32_t)upto(9, 4200);
    const uint64_t nblocks = upto(33, 4e9), avg = upto(1, 2.0 * win);
    const uint64_t span = nblocks * avg + upto(1, 64);
    IndexPlan p = index_plan(span, nblocks, win, i & 1);
    check(p, span);
    // all of a batch's segments, where one is enough, else most of a limit
    CHECK(p.per == p.nseg || (uint64_t)p.per * p.seg_bits > kIndexBatchBits / 2 ||
              p.bytes > kIndexWorkspace / 2,
          "%u %zu", p.per, p.bytes);
    const size_t room = (size_t)upto(1 << 16, 2.0 * kIndexWorkspace);
    size_t asked = ~(size_t)0;
    int calls = 0;
    const uint32_t per0 = p.per;
    const int r = index_reserve(p, [&](size_t bytes) {
      CHECK(bytes < asked || asked == 0, "%zu", bytes);
      asked = bytes;
      calls++;
      return bytes > room ? 1 : 0;
    });
    check(p, span);
    CHECK(asked == p.bytes && calls <= 12, "%d", calls);
    if (r == 0)
      CHECK(p.bytes <= room && (calls > 1 || p.per == per0), "%zu", p.bytes);
    else
      CHECK(r == 1 && p.per <= kIndexLeastSegments, "%d %u", r, p.per);
    // another failure is not tried again
    IndexPlan q = index_plan(span, nblocks, win, i & 1);
    calls = 0;
    CHECK(index_reserve(q, [&](size_t) { return calls++, 2; }) == 2 && calls == 1, "%d", calls);
  }
  if (!fails) printf("ok\n");
  return fails != 0;
}
