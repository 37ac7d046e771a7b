// The words that the index's CTAs stage and the bits that their parses read,
// on the CPU: the kernels' per-thread bodies over a reader that knows the
// staged words and counts the reads outside them.
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "gzfp_index_plan.h"

using namespace gzfp;

namespace {

// A CTA's staged words: `words` from word w0 of the stream on, bit 0 of the
// buffer being bit `origin` of the job.
struct Staged {
  const uint64_t* in;
  uint64_t n, w0;
  uint32_t words, origin;
  unsigned long long* outside;
  const IndexTables* t = index_tables_host();
  uint64_t word(uint64_t i) const {
    if (i >= words) (*outside)++;
    return w0 + i < n ? in[w0 + i] : 0;
  }
  uint32_t half(uint64_t i) const { return (uint32_t)(word(i >> 1) >> (32 * (i & 1))); }
  uint32_t peek32(uint32_t p) const {
    const uint32_t b = p - origin;
    return fshr(half(b >> 5), half((b >> 5) + 1), b & 31);
  }
};

struct Stream {
  const uint64_t* in;
  uint64_t n;
  uint64_t load(uint64_t i) const { return i < n ? in[i] : 0; }
};

// Counts: reads outside the staged words; lengths unlike the serial walk's;
// blocks parsed.
struct Counts {
  unsigned long long outside, wrong, parsed;
};

template <int D, typename T>
void run(const General& mode, const uint64_t* in, uint64_t n, uint64_t nblocks, uint32_t win,
         uint32_t field_lo, uint32_t field_hi, int sms, Counts& c) {
  IndexJob j{};
  j.in = in;
  j.nwords = n;
  j.mode = mode;
  j.lo = 5;  // as behind a header
  const uint64_t span = n * 64 - j.lo, avg = span / nblocks + 1;
  j.win = win;
  const IndexPlan plan = index_plan(span, nblocks, win, true);
  j.seg_bits = plan.seg_bits;
  j.nseg = (uint32_t)plan.nseg;  // one batch
  const Stream words{in, n};

  const IndexStage g = index_parse_stage(j, sms);
  const IndexRange range = index_range<D, T>(mode, field_lo, field_hi);
  const uint32_t sh = (uint32_t)(j.lo & 63);
  for (uint64_t at0 = 0; at0 < (uint64_t)j.nseg * j.seg_bits; at0 += g.bits) {
    const Staged r{in, n, (j.lo + at0) >> 6, g.words, (uint32_t)at0 - sh, &c.outside};
    const uint32_t size = (uint32_t)std::min<uint64_t>(g.bits, (uint64_t)j.nseg * j.seg_bits - at0);
    for (uint32_t q = 0; q < size / 32; q++) {
      const uint32_t i = q + (sh >> 5);
      uint32_t m = index_heads<T>(r.half(i), r.half(i + 1), r.half(i + 2), sh & 31, range);
      for (; m; m &= m - 1) {
        const uint32_t p = (uint32_t)at0 + q * 32 + ctz32(m);
        BlockParse<D, T, Staged> parse;
        bool done = parse.begin(p, block_head<D, T>(r.peek32(p), mode));
        while (!done) done = parse.step(r);
        c.parsed++;
        BitReader<Stream> whole(words, j.lo + p);
        c.wrong += parse.used(mode) != block_bits<D, T>(whole, mode);
      }
    }
  }

  const IndexPlaces s = index_sample_stage<T>(span, avg, win, sms);
  const IndexRange open = index_open<D, T>(mode);
  for (uint64_t k = 0; k < s.places; k++) {
    const Staged r{in, n, (j.lo >> 6) + k * (span / 64 / s.places), s.words, 0, &c.outside};
    IndexSampler<D, T, Staged> walk;
    for (uint32_t p = 0; p < s.bits; p++) {
      if (!(r.peek32(p) & 1)) continue;
      walk.start(p, s.limit);
      while (walk.tick(mode, open, r)) {
      }
    }
  }
}

}  // namespace

// The stream's parses and samples as a device of `sms` SMs makes them; win:
// the longest block.
extern "C" void ib_run(int type, int dims, unsigned minbits, unsigned maxbits, unsigned maxprec,
                       int minexp, const uint64_t* in, size_t nwords, unsigned long long nblocks,
                       unsigned win, unsigned field_lo, unsigned field_hi, int sms,
                       unsigned long long* counts) {
  const General mode{minbits, maxbits, maxprec, minexp};
  Counts c{0, 0, 0};
  auto go = [&](auto t) {
    typedef decltype(t) T;
    if (dims == 1) run<1, T>(mode, in, nwords, nblocks, win, field_lo, field_hi, sms, c);
    if (dims == 2) run<2, T>(mode, in, nwords, nblocks, win, field_lo, field_hi, sms, c);
    if (dims == 3) run<3, T>(mode, in, nwords, nblocks, win, field_lo, field_hi, sms, c);
  };
  if (type == 3) go(0.0f);
  if (type == 4) go(0.0);
  counts[0] = c.outside;
  counts[1] = c.wrong;
  counts[2] = c.parsed;
}
