// The parallel block index on the CPU: the per-thread bodies of its kernels
// (gzfp_index_chain.cuh), run thread after thread in the kernels' order.
#include <stddef.h>
#include <stdint.h>

#include <vector>

#include "gzfp_index_chain.cuh"

using namespace gzfp;

namespace {

struct Words {
  const uint64_t* in;
  uint64_t n;
  uint64_t load(uint64_t i) const { return i < n ? in[i] : 0; }
};

struct Reader {
  const Words& w;
  uint64_t lo;
  uint32_t peek32(uint32_t p) const {
    const uint64_t b = lo + p, sh = b & 63;
    return (uint32_t)(w.load(b >> 6) >> sh | (sh ? w.load((b >> 6) + 1) << (64 - sh) : 0));
  }
  const IndexTables* t = index_tables_host();
};

template <int D, typename T>
void batch(IndexJob j, const Words& w, int heads, IndexState& st, unsigned long long* offsets) {
  j.zeros = !FT<T>::INT && j.mode.minbits <= 1;
  const Reader r{w, j.lo};
  std::vector<uint32_t> first;  // window bits the links start from
  if (heads) {
    const IndexRange range = index_range<D, T>(j.mode, st.field_lo, st.field_hi);
    BlockParse<D, T, Reader> parse;
    for (uint32_t s = 0; s < j.nseg; s++) {
      const uint32_t seg0 = s * j.seg_bits;
      for (uint32_t g = 0; g < j.seg_bits; g += 32) {
        // the words at sh's word, as the kernel passes them
        const uint64_t b = j.lo + seg0 + g, i = b >> 5;
        uint32_t v[3];
        for (int k = 0; k < 3; k++) v[k] = (uint32_t)(w.load((i + k) >> 1) >> (32 * ((i + k) & 1)));
        uint32_t m = index_heads<T>(v[0], v[1], v[2], (uint32_t)(b & 31), range);
        for (; m; m &= m - 1) {
          const uint32_t p = g + ctz32(m);
          if (p < j.win) first.push_back(seg0 + p);
          bool done = parse.begin(seg0 + p, block_head<D, T>(r.peek32(seg0 + p), j.mode));
          while (!done) done = parse.step(r);
          j.table[seg0 + p] = (uint16_t)parse.used(j.mode);
        }
      }
      first.push_back(seg0 + j.win);
    }
    first.push_back(0);
  } else {
    for (uint32_t s = 0; s < j.nseg; s++)
      for (uint32_t p = 0; p <= j.win; p++)
        if (FT<T>::INT || !j.zeros || p == j.win || (p == 0 && s == 0) ||
            (r.peek32(s * j.seg_bits + p) & 1))
          first.push_back(s * j.seg_bits + p);
    IndexLane<D, T, Reader> walk;
    for (uint32_t p : first) {
      walk.start(j, p);
      while (walk.tick(j, r)) {
      }
    }
  }
  // the link kernels
  const uint32_t n1 = (j.nseg + j.fan - 1) / j.fan, n2 = (n1 + j.fan - 1) / j.fan;
  std::vector<uint32_t> ex((size_t)j.nseg * (j.win + 1), 77), e0(j.nseg), e1(n1), e2(n2);
  std::vector<IndexHop> h1((size_t)n1 * (j.win + 1)), h2((size_t)n2 * (j.win + 1));
  std::vector<unsigned long long> b0(j.nseg), b1(n1), b2(n2);
  auto hop0 = [&](uint32_t i, uint32_t e) { return index_hop(j, ex.data(), i, e); };
  auto hop1 = [&](uint32_t i, uint32_t e) { return h1[(size_t)i * (j.win + 1) + e]; };
  auto hop2 = [&](uint32_t i, uint32_t e) { return h2[(size_t)i * (j.win + 1) + e]; };
  for (uint32_t p : first) {
    const uint32_t s = p / j.seg_bits, v = p % j.seg_bits;
    ex[(size_t)s * (j.win + 1) + v] = index_exit(j, w, s, v);
  }
  for (uint32_t g = 0; g < n1; g++)
    for (uint32_t v = 0; v <= j.win; v++)
      h1[(size_t)g * (j.win + 1) + v] = index_compose(g, j.fan, j.nseg, v, hop0);
  for (uint32_t g = 0; g < n2; g++)
    for (uint32_t v = 0; v <= j.win; v++)
      h2[(size_t)g * (j.win + 1) + v] = index_compose(g, j.fan, n1, v, hop1);
  uint32_t e = kIndexNone;
  if (!st.done && !st.broken && st.pos >= j.lo) {
    if (st.pos - j.lo <= j.win) e = (uint32_t)(st.pos - j.lo); else st.broken = 1;
  }
  index_descend(0, n2, n2, e, st.count, j.nblocks, e2.data(), b2.data(), hop2);
  for (uint32_t g = 0; g < n2; g++)
    index_descend(g, j.fan, n1, e2[g], b2[g], j.nblocks, e1.data(), b1.data(), hop1);
  for (uint32_t g = 0; g < n1; g++)
    index_descend(g, j.fan, j.nseg, e1[g], b1[g], j.nblocks, e0.data(), b0.data(), hop0);
  for (uint32_t s = 0; s < j.nseg; s++) index_emit(j, w, s, e0[s], b0[s], offsets, &st);
}

template <typename T>
void batch_d(int dims, const IndexJob& j, const Words& w, int heads, IndexState& st,
             unsigned long long* offsets) {
  if (dims == 1) batch<1, T>(j, w, heads, st, offsets);
  if (dims == 2) batch<2, T>(j, w, heads, st, offsets);
  if (dims == 3) batch<3, T>(j, w, heads, st, offsets);
}

// the exponents of the first `bits` bits of the stream, as a sampling CTA
template <int D, typename T>
void sample(const Words& w, const General& mode, uint32_t bits, IndexState& st) {
  const Reader r{w, 0};
  IndexSampler<D, T, Reader> walk;
  for (uint32_t p = 0; p < bits; p++) {
    if (!(r.peek32(p) & 1)) continue;
    walk.start(p, bits + 20000);
    while (walk.tick(mode, index_open<D, T>(mode), r)) {
    }
    if (!walk.kept) continue;
    st.field_lo = umin(st.field_lo, (uint32_t)walk.lo);
    st.field_hi = st.field_hi > (uint32_t)walk.hi ? st.field_hi : (uint32_t)walk.hi;
  }
}

template <typename T>
void sample_d(int dims, const Words& w, const General& mode, uint32_t bits, IndexState& st) {
  if (dims == 1) sample<1, T>(w, mode, bits, st);
  if (dims == 2) sample<2, T>(w, mode, bits, st);
  if (dims == 3) sample<3, T>(w, mode, bits, st);
}

}  // namespace

// Block starts of the stream from bit `first`, heads or walks; returns 1
// done, 0 the stream ends first, 2 broken; end: the bit after the last
// block; field: in, the range of exponent fields (empty: sampled), out, the
// range, or the field that broke the chain, twice.
extern "C" int ic_index(int type, int dims, unsigned long long nblocks, unsigned minbits,
                        unsigned maxbits, unsigned maxprec, int minexp, const uint64_t* in,
                        size_t nwords, unsigned long long first, unsigned seg_bits, unsigned bound,
                        unsigned per, int heads, unsigned* field, unsigned long long* offsets,
                        unsigned long long* end) {
  const Words w{in, nwords};
  const General mode{minbits, maxbits, maxprec, minexp};
  const uint64_t total = nwords * 64, span = total - first;
  const uint64_t nseg = (span + seg_bits - 1) / seg_bits;
  std::vector<uint16_t> table((size_t)per * seg_bits);
  IndexState st{};
  st.pos = first;
  st.field_lo = field[0];
  st.field_hi = field[1];
  if (heads && st.field_lo > st.field_hi) {
    if (type == 3) sample_d<float>(dims, w, mode, 6000, st);
    if (type == 4) sample_d<double>(dims, w, mode, 6000, st);
  }
  for (uint64_t s0 = 0; s0 < nseg; s0 += per) {
    IndexJob j{};
    j.in = in;
    j.nwords = nwords;
    j.mode = mode;
    j.lo = first + s0 * seg_bits;
    j.nseg = (uint32_t)(nseg - s0 < per ? nseg - s0 : per);
    j.seg_bits = seg_bits;
    j.win = bound;
    while ((uint64_t)j.fan * j.fan * j.fan < per) j.fan++;
    j.nblocks = nblocks;
    table.assign(table.size(), 0);
    j.table = table.data();
    if (type == 1) batch_d<int32_t>(dims, j, w, heads, st, offsets);
    if (type == 2) batch_d<int64_t>(dims, j, w, heads, st, offsets);
    if (type == 3) batch_d<float>(dims, j, w, heads, st, offsets);
    if (type == 4) batch_d<double>(dims, j, w, heads, st, offsets);
  }
  *end = st.end;
  field[0] = st.broken ? (unsigned)(st.head >> 1) & (type == 3 ? 255u : 2047u) : st.field_lo;
  field[1] = st.broken ? field[0] : st.field_hi;
  return st.done ? 1 : st.broken ? 2 : 0;
}
