// 1D blocks coded with fewer words of code than the longest (the 1D kernels'
// choice for small budgets), block after block on the host.
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include "gzfp_array.cuh"

namespace {

struct Words {
  uint64_t* out;
  const uint64_t* in;
  uint64_t n;
  void store(uint64_t i, uint64_t v) { out[i] = v; }
  void merge(uint64_t i, uint64_t v) { out[i] |= v; }
  uint64_t load(uint64_t i) const { return i < n ? in[i] : 0; }
};

template <typename T, int NW>
void go(bool decode, unsigned nx, unsigned maxbits, void* data, uint64_t* words, uint64_t n) {
  gzfp::Geom g = gzfp::make_geom_blocks(nx, 1, 1);
  gzfp::LocalPlanes ps;
  for (uint64_t b = 0; b < g.nblocks; b++) {
    if (decode)
      gzfp::decode_one<1, T, NW ? NW : 1>((T*)data, g, b, maxbits, Words{nullptr, words, n}, ps);
    else
      gzfp::encode_one<1, T, false, NW>((const T*)data, g, b, maxbits, Words{words, nullptr, n}, ps);
  }
}

template <typename T>
void go_t(bool decode, int nw, unsigned nx, unsigned maxbits, void* data, uint64_t* words,
          uint64_t n) {
  if (nw == 0) go<T, 0>(decode, nx, maxbits, data, words, n);  // encoder: up to 32 bits
  if (nw == 1) go<T, 1>(decode, nx, maxbits, data, words, n);
  if (nw == 2) go<T, 2>(decode, nx, maxbits, data, words, n);
}

}  // namespace

extern "C" void sc_code(int decode, int type, int nw, unsigned nx, unsigned maxbits, void* data,
                        uint64_t* words, size_t n) {
  if (!decode) memset(words, 0, n * 8);
  if (type == 1) go_t<int32_t>(decode, nw, nx, maxbits, data, words, n);
  if (type == 2) go_t<int64_t>(decode, nw, nx, maxbits, data, words, n);
  if (type == 3) go_t<float>(decode, nw, nx, maxbits, data, words, n);
  if (type == 4) go_t<double>(decode, nw, nx, maxbits, data, words, n);
}
