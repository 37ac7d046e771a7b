// gzfp_index_parse.cuh -- parsing a general-mode stream for its block
// lengths, one token at a time.  Host+device: the CPU tests check the parse
// against the oracle's block starts.
#pragma once

#include "gzfp_array.cuh"

namespace gzfp {

// The exponent field of a floating-point block's header, the planes the
// block codes and the bits it may take.
template <int D, typename T>
struct BlockHead {
  uint32_t field;  // emax + EBIAS
  int prec;
  uint32_t maxbits;
};

template <int D, typename T>
GZ_HD BlockHead<D, T> block_head(uint32_t head, const General& mode) {
  typedef FT<T> F;
  BlockHead<D, T> h{0, F::P, mode.maxbits};
  if constexpr (!F::INT) {
    h.field = (head >> 1) & ((1u << F::EBITS) - 1);
    h.prec = mode.template precision<D, F::P>((int)h.field - F::EBIAS);
  } else {
    h.prec = F::P - mode.template int_kmin<F::P>();
  }
  return h;
}

// Tables of the parse.
struct IndexTables {
  // Test bits of planes at frontier n that bring no new coefficient, from
  // the first on: bit 0, then every n + 1 bits.
  uint32_t plain[32];
  // The whole groups (a 1, zeros, a one) in 10 bits from a test bit on, and
  // the 0 test after them if it is among the bits: bits taken | coefficients
  // passed << 4 | plane ended << 8; 0 when the first group is longer.
  uint16_t groups[1024];
};

GZ_CX IndexTables make_index_tables() {
  IndexTables t{};
  for (uint32_t n = 0; n < 32; n++)
    for (uint32_t i = 0; i < 32; i += n + 1) t.plain[n] |= 1u << i;
  for (uint32_t v = 0; v < 1024; v++) {
    uint32_t c = 0, adv = 0, end = 0;
    while (c < 10) {
      if (!((v >> c) & 1)) {  // the plane's last test
        c++;
        end = 1;
        break;
      }
      uint32_t q = c + 1;
      while (q < 10 && !((v >> q) & 1)) q++;
      if (q == 10) break;  // the one is not among the bits
      adv += q - c;
      c = q + 1;
    }
    t.groups[v] = (uint16_t)(c | adv << 4 | end << 8);
  }
  return t;
}

#if defined(__CUDACC__)
__device__ const __align__(16) IndexTables kIndexTables = make_index_tables();
#endif
inline const IndexTables* index_tables_host() {
  static const IndexTables t = make_index_tables();
  return &t;
}

// One block's parse as a state machine over a reader R (peek32(bit), t: the
// tables): begin() at the block's header, then step() until it returns true.
// Only lengths are wanted, so verbatim bits are skipped unread and the state
// sits at a test bit: a step takes the run of planes whose test is 0 (each is
// a 0 and the next plane's verbatim bits) and then, by table, the groups of a
// plane that brings coefficients.  Once every coefficient is significant the
// rest of the planes have known lengths, and a budget that ends inside the
// block just cuts its length (zfp's coder spends the budget to the last bit).
// No step is begun past the budget's end, so that whatever the bits say,
// none is read kParseAhead or more bits past the longest block: up to 22 of
// planes passed, 33 into a group, and 63 more in the two words of a peek.
// Same lengths as block_bits.
constexpr uint32_t kParseAhead = 22 + 33 + 63;
template <int D, typename T, class R>
struct BlockParse {
  static constexpr uint32_t BS = 1u << (2 * D);
  uint32_t cur, start, end, pos, left;  // bits from the job's first; frontier; planes left

  GZ_HD bool begin(uint32_t p, const BlockHead<D, T>& h) {
    start = p;
    end = p + h.maxbits;
    cur = p;
    if constexpr (!FT<T>::INT) cur += FT<T>::EBITS + 1;
    pos = 0;
    left = (uint32_t)h.prec;
    return left == 0;
  }

  // true when the block is complete
  GZ_HD bool step(const R& r) {
    if (cur >= end) return true;  // used() cuts the length
    uint32_t w = r.peek32(cur);
    if (!(w & 1)) {  // planes without new coefficients
      const uint32_t m = r.t->plain[umin(pos, 31u)], hit = w & m;
      const uint32_t k = umin(popcount32(hit ? m & ((hit & (0u - hit)) - 1) : m), left);
      const uint32_t c = k * (pos + 1);
      cur += c;
      left -= k;
      if (left == 0) {
        cur -= pos;  // no plane follows
        return true;
      }
      if (c > 22) return false;  // fewer than 10 bits of the window left
      w >>= c;
      if (!(w & 1)) return false;
    }
    const uint32_t e = r.t->groups[w & 1023u], adv = (e >> 4) & 15u;
    if (e != 0 && pos + adv < BS - 1) {
      pos += adv;
      cur += e & 15u;
      if (e < 256) return false;
      if (--left == 0) return true;
      cur += pos;
      return false;
    }
    // one group: long, or one that may reach the last position
    uint32_t t = ctz32(r.peek32(cur + 1));
    const uint32_t lim = BS - 1 - pos;
    if (BS > 32 && t == 32) t = 32 + ctz32(r.peek32(cur + 33));
    const bool read = t < lim;
    const uint32_t z = read ? t : lim;
    cur += z + 1 + (read ? 1u : 0u);
    pos += z + 1;
    if (pos < BS) return false;
    cur += (left - 1) * BS;
    left = 0;
    return true;
  }
  GZ_HD uint32_t used(const General& mode) const {
    const uint32_t u = umin(cur - start, mode.maxbits);
    return u < mode.minbits ? mode.minbits : u;
  }
};

}  // namespace gzfp
