// gzfp_index_chain.cuh -- the block starts of a general-mode stream, found
// in parallel: the per-thread bodies of the index kernels (gzfp_index.cuh,
// gzfp_index_link.cu).  Host+device: the CPU tests run the same bodies.
//
// A block's length is known only by parsing it, so the starts form a chain
// p -> p + length(p) from block 0.  But a length can be parsed at any bit,
// and the header says where it is worth it: of the bits of a floating-point
// stream, half are 1 and so could be a block's first, and of these one in a
// few hundred is followed by an exponent like the field's (8 or 11 bits).  So:
//  1. sample: a few hundred places of the stream are searched for chains of
//     blocks with steady exponents; the exponents found give a range;
//  2. every bit that looks like a header with an exponent in the range is
//     parsed, all at once, and its length written to table[bit] (1-5 times
//     as many parses as there are blocks);
//  3. the stream is cut into segments of seg_bits bits, which the true chain
//     enters somewhere in their first `win` bits (the longest block).  Per
//     header found there: the bit where its chain enters the next segment,
//     and the blocks on the way (index_exit); these maps are composed over
//     groups of segments and groups of groups (index_compose);
//  4. the true chain is followed over the top groups, then down again to
//     every segment's entry (index_descend), and one thread per segment
//     writes its block starts (index_emit).
// An entry of the table is a fact about the stream, whatever it was parsed
// for, and step 4 follows lengths from block 0 on, so the starts written are
// the true ones.  A block whose exponent is out of the range shows as a
// missing entry; the caller then widens the range by it and repeats.
// Where there are no headers (integers), or exponents too far apart, chains
// are instead walked from every bit of the windows to their segment's end
// (IndexLane), a walk ending where another has been: chains from wrong bits
// merge with others, after a few hundred blocks in all.
#pragma once

#include <stddef.h>

#include "gzfp_index_parse.cuh"

namespace gzfp {

constexpr uint32_t kIndexNone = 0xffffffffu;  // no exit, no entry

struct IndexJob {
  const uint64_t* in;
  uint64_t nwords;
  General mode;
  uint64_t lo;         // stream bit of segment 0
  uint32_t nseg;       // segments
  uint32_t seg_bits;   // bits per segment, a power of two, > the longest block
  uint32_t win;        // window: the longest block, < seg_bits
  uint32_t fan;        // segments per group, groups per top group
  uint32_t zeros;      // a 0 bit is a whole block (floating point, minbits <= 1)
  uint64_t nblocks;
  uint16_t* table;     // per bit: the length of a block there, 0 unknown
};

// The true chain's state between batches of segments, its outcome, and the
// exponents seen.
struct IndexState {
  unsigned long long pos, count;  // next block's bit, blocks before it
  unsigned long long end;         // bit after the last block
  unsigned long long head;        // broken: the 64 bits at the missing block
  unsigned int done;              // the last block's start is written
  unsigned int broken;            // a block's length is missing
  unsigned int field_lo, field_hi;  // exponent fields (lo > hi: none seen)
};

// The chain is complete or broken: nothing is left to do for the batches that
// follow (only the link kernels' last two change it, so that a batch's other
// kernels all see it alike).
GZ_HD bool index_over(const IndexState& st) { return st.done || st.broken; }

struct IndexHop {  // entry in the next (group of) segment's window, blocks on the way
  uint32_t exit, count;
};

// Exponent fields worth parsing: from 6 below the lowest seen (a field's
// smallest values) to 2 above the highest, among those an encoder writes in
// this mode (index_open).  `most` bounds what a wide range may cost: with
// 128 of 2048, or 48 of 256, fields, 3% or 9% of all bits are parsed.
struct IndexRange {
  uint32_t lo, span;  // field - lo <= span
};
template <typename T>
GZ_CX uint32_t index_most() { return sizeof(T) == 8 ? 128u : 48u; }

// The fields an encoder writes: those that leave the block planes to code (a
// single 0 bit is written instead) and, in fixed-accuracy mode, do not claim
// planes far below the type's own precision (legal, but only for values
// 2^kIndexSlack times too large for their last bits to matter).
constexpr int kIndexSlack = 4;
template <int D, typename T>
GZ_HD IndexRange index_open(const General& mode) {
  if constexpr (FT<T>::INT) {
    return IndexRange{0, ~0u};
  } else {
    const int bias = FT<T>::EBIAS + mode.minexp - 2 * D - 2;  // field = precision + bias
    const int most = (1 << FT<T>::EBITS) - 1;
    const int lo = 1 + bias < 0 ? 0 : 1 + bias > most ? most : 1 + bias;
    int hi = mode.minexp == kMinExp ? most : FT<T>::P + kIndexSlack + bias;
    hi = hi > most ? most : hi < lo ? lo : hi;
    return IndexRange{(uint32_t)lo, (uint32_t)(hi - lo)};
  }
}
template <int D, typename T>
GZ_HD IndexRange index_range(const General& mode, uint32_t seen_lo, uint32_t seen_hi) {
  const IndexRange open = index_open<D, T>(mode);
  if (seen_lo > seen_hi) return IndexRange{open.lo, umin(open.span, index_most<T>())};
  const uint32_t a = seen_lo > 6 ? seen_lo - 6 : 0, b = umin(seen_hi + 2, open.lo + open.span);
  const uint32_t lo = a > open.lo ? a : open.lo;
  return IndexRange{lo, b < lo ? 0u : umin(b - lo, index_most<T>())};
}

// Of the 32 bits from `b` on (w0, w1, w2: the words at b / 32), those that
// look like a header: a 1 bit and a field in the range.  All 32 are compared
// at once, bit by bit of the field: ge and le hold, per position, whether the
// bits so far compare as at least lo and at most lo + span.
template <typename T>
GZ_HD uint32_t index_heads(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t sh, IndexRange g) {
  const uint32_t a = fshr(w0, w1, sh), c = fshr(w1, w2, sh);
  const uint32_t lo = g.lo, hi = g.lo + g.span;
  uint32_t ge = ~0u, le = ~0u;
  if constexpr (!FT<T>::INT) {
#pragma unroll
    for (int k = 0; k < FT<T>::EBITS; k++) {
      const uint32_t e = fshr(a, c, (uint32_t)(k + 1));
      const uint32_t L = 0u - ((lo >> k) & 1u), H = 0u - ((hi >> k) & 1u);
      ge = (e & ge) | (~L & (e | ge));
      le = (~e & le) | (H & (~e | le));
    }
  }
  return a & ge & le;
}

// A sampling walk from a 1 bit: kIndexSteady blocks in a row whose fields
// differ by at most 4.  (Of the wrong bits 1 in 10^7 passes: 9 of 2048
// fields three times, of 256 five times.)
template <typename T>
GZ_CX int index_steady() { return sizeof(T) == 8 ? 3 : 5; }

template <int D, typename T, class R>
struct IndexSampler {
  typedef FT<T> F;
  static constexpr int kSteps = D == 3 ? 8 : D == 2 ? 4 : 2;
  BlockParse<D, T, R> parse;
  uint32_t p, limit;  // bits from the job's first; no block beyond the limit is begun
  int last, lo, hi, steady;
  bool in_block, kept;

  GZ_HD void start(uint32_t at, uint32_t limit_) {
    p = at;
    limit = limit_;
    last = -1;
    steady = 0;
    in_block = kept = false;
  }
  // false: ended; kept: the chain is steady, with fields lo .. hi
  GZ_HD bool tick(const General& mode, IndexRange open, const R& r) {
    if (!in_block) {
      if (p > limit) return false;
      const uint32_t head = r.peek32(p);
      if (!(head & 1)) {
        p += ctz32(head);
        return true;
      }
      const BlockHead<D, T> h = block_head<D, T>(head, mode);
      if (h.field - open.lo > open.span) return false;
      const int f = (int)h.field;
      if (last < 0) {
        lo = hi = f;
      } else {
        if (f > last + 4 || f < last - 4) return false;
        lo = f < lo ? f : lo;
        hi = f > hi ? f : hi;
        if (++steady == index_steady<T>()) {
          kept = true;
          return false;
        }
      }
      last = f;
      in_block = !parse.begin(p, h);
    }
#pragma unroll 1
    for (int i = 0; i < kSteps && in_block; i++) in_block = !parse.step(r);
    if (!in_block) p += parse.used(mode);
    return true;
  }
};

// What a CTA of the sampling and of the parsing kernel stages: the stream's
// words from the bits it starts blocks at to the last bit that a block begun
// there is read at (kParseAhead).
struct IndexStage {
  uint32_t bits;   // starts are looked for in the first `bits`
  uint32_t limit;  // and no block beyond `limit` is begun
  uint32_t words;  // 64-bit words staged
};
inline uint32_t index_stage_words(uint32_t limit, uint32_t win) {
  return (limit + win + kParseAhead) / 64 + 1;
}
// Of the stream's `span` bits: `places` places, 2 per SM where there are as
// many.  avg: the stream's bits per block.  (A lane searches its bits one after
// another, a block's parse for each that may be a first one: fewer bits where
// the places do not overlap anyway.)
struct IndexPlaces : IndexStage {
  uint64_t places;
};
template <typename T>
IndexPlaces index_sample_stage(uint64_t span, uint64_t avg, uint32_t win, int sms) {
  const uint32_t block = (uint32_t)(avg < win ? avg : win);
  const uint64_t most = 2 * (uint64_t)sms, each = span / most + 1;
  IndexPlaces s;
  s.bits = (uint32_t)(avg < 100 ? 256 : avg < 1600 ? avg * 5 / 2 : 4000);
  if (each < s.bits) s.bits = each < 256 ? 256 : (uint32_t)each;
  s.limit = s.bits + ((uint32_t)index_steady<T>() + 1) * block + 256;
  s.words = index_stage_words(s.limit, win);
  const uint64_t n = span / s.bits + 1;
  s.places = n < most ? n : most;
  return s;
}
// 256 to 32,768 bits a warp, as many as leave every scheduler 8 warps: a lane
// of a long stream then parses several blocks, and idles less at the end; of a
// short stream as few as there can be, one after another.  (The first word
// staged begins up to 63 bits before the chunk.)
inline IndexStage index_parse_stage(const IndexJob& j, int sms) {
  const uint64_t all = (uint64_t)j.nseg * j.seg_bits;
  IndexStage s;
  s.bits = 256;
  while (s.bits < 32768 && all / s.bits > (uint64_t)sms * 32) s.bits *= 2;
  s.limit = 63 + s.bits;
  s.words = index_stage_words(s.limit, j.win);
  return s;
}

// A walk from any bit to its segment's end, or to where another has been.
// tick() takes up the block at p if it is in none, makes up to kSteps steps
// in it and returns false when the walk ends.  (A warp's lanes are at
// different points of their blocks, so it runs through a block's beginning
// and end on nearly every tick: several steps per tick spread that cost.)
template <int D, typename T, class R>
struct IndexLane {
  typedef FT<T> F;
  static constexpr int kSteps = D == 3 ? 8 : D == 2 ? 4 : 2;
  BlockParse<D, T, R> parse;
  uint32_t p, seg_end;  // bits from the job's first
  bool in_block;

  GZ_HD void start(const IndexJob& j, uint32_t at) {
    p = at;
    seg_end = (at / j.seg_bits + 1) * j.seg_bits;
    in_block = false;
  }
  GZ_HD bool tick(const IndexJob& j, const R& r) {
    if (!in_block) {
      if (p >= seg_end || j.lo + p >= j.nwords * 64) return false;
      if (*(const volatile uint16_t*)(j.table + p)) return false;
      const uint32_t head = F::INT ? 1u : r.peek32(p);
      if (!(head & 1)) {  // zero blocks
        if (!j.zeros) j.table[p] = (uint16_t)j.mode.minbits;
        p += j.zeros ? umin(ctz32(head), seg_end - p) : j.mode.minbits;
        return true;
      }
      in_block = !parse.begin(p, block_head<D, T>(head, j.mode));
    }
#pragma unroll 1
    for (int i = 0; i < kSteps && in_block; i++) in_block = !parse.step(r);
    if (!in_block) {
      const uint32_t len = parse.used(j.mode);
      j.table[p] = (uint16_t)len;
      p += len;
    }
    return true;
  }
};

// Zero blocks of one bit have no entries in the table and are never entries
// of a window: a chain's entry is taken after them, so at the next 1 bit or,
// if there is none, at bit `win`.  The first 1 bit from p on, at most
// `limit` (bits from j.lo).
template <class Words>
GZ_HD uint32_t index_skip(const IndexJob& j, const Words& words, uint32_t p, uint32_t limit) {
  if (!j.zeros) return p;
  while (p < limit) {
    const uint64_t b = j.lo + p;
    const uint64_t v = words.load(b >> 6) >> (b & 63);
    if (v) {
      p += ctz64(v);
      break;
    }
    p += 64 - (uint32_t)(b & 63);
  }
  return umin(p, limit);
}

// Where the chain from window bit w of segment s enters the next segment,
// and the blocks on the way: exit | blocks << 16, or kIndexNone.
template <class Words>
GZ_HD uint32_t index_exit(const IndexJob& j, const Words& words, uint32_t s, uint32_t w) {
  const uint32_t end = (s + 1) * j.seg_bits;
  const uint64_t total = j.nwords * 64;
  uint32_t p = s * j.seg_bits + w, count = 0;
  while (p < end) {
    if (j.lo + p >= total) return kIndexNone;
    const uint32_t v = j.table[p];
    if (v) {
      p += v;
      count++;
    } else {
      const uint32_t q = index_skip(j, words, p, end);
      if (q == p) return kIndexNone;
      count += q - p;
      p = q;
    }
  }
  if (p - end > j.win) return kIndexNone;
  const uint32_t q = index_skip(j, words, p, end + j.win);
  return (q - end) | (count + (q - p)) << 16;
}

// The hop from entry w of segment s: exits holds one where a chain was
// started, which the table tells (the window's end and block 0's bit aside).
GZ_HD IndexHop index_hop(const IndexJob& j, const uint32_t* exits, uint32_t s, uint32_t w) {
  const uint32_t m = exits[(size_t)s * (j.win + 1) + w];
  const bool started = j.table[s * j.seg_bits + w] != 0 || w == j.win || (s == 0 && w == 0);
  return !started || m == kIndexNone ? IndexHop{kIndexNone, 0} : IndexHop{m & 0xffffu, m >> 16};
}

// The composition of hops [g * fan, min((g + 1) * fan, n)) from window bit w.
template <class HopFn>
GZ_HD IndexHop index_compose(uint32_t g, uint32_t fan, uint32_t n, uint32_t w, HopFn&& hop) {
  IndexHop h{w, 0};
  const uint64_t lo = (uint64_t)g * fan, hi = lo + fan < n ? lo + fan : n;
  for (uint64_t i = lo; i < hi; i++) {
    const IndexHop m = hop((uint32_t)i, h.exit);
    if (m.exit == kIndexNone) return m;
    h.exit = m.exit;
    h.count += m.count;
  }
  return h;
}

// The entries of [g * fan, ...) below a node whose own entry is (w, count):
// entry[i], base[i], up to the first whose hop is missing, or that starts
// past the last block; kIndexNone from there on.
template <class HopFn>
GZ_HD void index_descend(uint32_t g, uint32_t fan, uint32_t n, uint32_t w,
                         unsigned long long count, uint64_t nblocks, uint32_t* entry,
                         unsigned long long* base, HopFn&& hop) {
  const uint64_t lo = (uint64_t)g * fan, hi = lo + fan < n ? lo + fan : n;
  for (uint64_t i = lo; i < hi; i++) {
    if (w != kIndexNone && count >= nblocks) w = kIndexNone;
    entry[i] = w;
    base[i] = count;
    if (w == kIndexNone) continue;
    const IndexHop m = hop((uint32_t)i, w);
    w = m.exit;
    count += m.count;
  }
}

// Segment s, entered at window bit w with `count` blocks before it: its
// block starts, up to the entry of the next segment, and (the last segment)
// the state for the next batch.
template <class Words>
GZ_HD void index_emit(const IndexJob& j, const Words& words, uint32_t s, uint32_t w,
                      unsigned long long count, unsigned long long* offsets, IndexState* st) {
  if (w == kIndexNone) return;
  const uint32_t end = (s + 1) * j.seg_bits;
  const uint64_t total = j.nwords * 64;
  uint32_t p = s * j.seg_bits + w;
  for (;;) {
    uint32_t run = 1, len = 1;  // zero blocks, or one block
    if (j.lo + p >= total) return;  // the stream ends before its blocks
    const uint32_t v = p < end ? j.table[p] : 0;
    if (v) {
      len = v;
    } else {
      run = index_skip(j, words, p, p < end ? end : end + j.win) - p;
      if (run == 0 && p >= end) break;
      if (run == 0) {
        const uint64_t b = j.lo + p, sh = b & 63;
        st->head = words.load(b >> 6) >> sh | (sh ? words.load((b >> 6) + 1) << (64 - sh) : 0);
        st->broken = 1;
        return;
      }
    }
    for (; run; run--) {
      offsets[count++] = j.lo + p;
      p += len;
      if (count == j.nblocks) {
        st->end = j.lo + p;
        st->done = 1;
        return;
      }
    }
  }
  if (s + 1 == j.nseg) {
    st->pos = j.lo + p;
    st->count = count;
  }
}

}  // namespace gzfp
