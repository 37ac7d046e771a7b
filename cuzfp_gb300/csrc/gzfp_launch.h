// gzfp_launch.h -- internal launcher interface between the host API
// (gzfp_api.cu) and the kernel translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "gzfp_array.cuh"
#include "gzfp_index_chain.cuh"

namespace gzfp {

// Launch the plain-path encoder / decoder for `dims` (1..3) on stream `s`.
cudaError_t launch_encode_f32(int dims, const float* in, const Geom& g, uint32_t maxbits,
                              uint64_t* out, uint64_t nwords, cudaStream_t s);
cudaError_t launch_encode_f64(int dims, const double* in, const Geom& g, uint32_t maxbits,
                              uint64_t* out, uint64_t nwords, cudaStream_t s);
cudaError_t launch_decode_f32(int dims, const uint64_t* in, uint64_t nwords, const Geom& g,
                              uint32_t maxbits, float* out, cudaStream_t s);
cudaError_t launch_decode_f64(int dims, const uint64_t* in, uint64_t nwords, const Geom& g,
                              uint32_t maxbits, double* out, cudaStream_t s);
cudaError_t launch_encode_i32(int dims, const int32_t* in, const Geom& g, uint32_t maxbits,
                              uint64_t* out, uint64_t nwords, cudaStream_t s);
cudaError_t launch_encode_i64(int dims, const int64_t* in, const Geom& g, uint32_t maxbits,
                              uint64_t* out, uint64_t nwords, cudaStream_t s);
cudaError_t launch_decode_i32(int dims, const uint64_t* in, uint64_t nwords, const Geom& g,
                              uint32_t maxbits, int32_t* out, cudaStream_t s);
cudaError_t launch_decode_i64(int dims, const uint64_t* in, uint64_t nwords, const Geom& g,
                              uint32_t maxbits, int64_t* out, cudaStream_t s);

// Random access to listed blocks, each coded from / into its own tile of
// 4^dims values (gzfp_blocks.cuh; instantiated for float, double, int32_t
// and int64_t in gzfp_blocks_*.cu).
template <typename T>
cudaError_t launch_encode_blocks(int dims, const T* tiles, const unsigned long long* index,
                                 const uint8_t* shape, uint64_t count, uint32_t maxbits,
                                 uint64_t* out, uint64_t nwords, cudaStream_t s);
template <typename T>
cudaError_t launch_decode_blocks(int dims, const uint64_t* in, uint64_t nwords,
                                 const unsigned long long* index, const uint8_t* shape,
                                 uint64_t count, uint32_t maxbits, T* tiles, cudaStream_t s);

// zfp's general coding modes (gzfp_modes.cuh; instantiated for the four
// scalar types in gzfp_modes_*.cu): every block into its own scratch slot
// with its length, decoding from known start bits, and the serial walk that
// finds those start bits.  The scan and the placement of the blocks are
// type-independent (gzfp_modes_common.cu).
template <typename T>
cudaError_t launch_encode_mode(int dims, const T* in, const Geom& g, const General& mode,
                               uint64_t* scratch, uint32_t slot_words, uint32_t* lengths,
                               cudaStream_t s);
template <typename T>
cudaError_t launch_decode_mode(int dims, const uint64_t* in, uint64_t nwords,
                               const unsigned long long* offsets, const Geom& g,
                               const General& mode, T* out, cudaStream_t s);
template <typename T>
cudaError_t launch_index_blocks(int dims, const uint64_t* in, uint64_t nwords, uint64_t nblocks,
                                const General& mode, uint64_t first, unsigned long long* offsets,
                                unsigned long long* end, cudaStream_t s);
// Exclusive scan of n block lengths into start bits from `first` (sums:
// room for ceil(n / 4096) + 1 entries; sums[ceil(n / 4096)] receives the
// total length), then the placement of every block at its start bit in a
// zeroed stream.
cudaError_t launch_scan_lengths(const uint32_t* lengths, uint64_t n, uint64_t first,
                                uint64_t* sums, unsigned long long* offsets, cudaStream_t s);
uint64_t scan_sums_count(uint64_t n);
// most bits one block can take under `mode` (gzfp_modes.cuh block_bound)
uint32_t block_bound_host(int dims, int P, int ebits, const General& mode);
// offsets[b] = first + b * maxbits: the start bits of a fixed-rate stream
cudaError_t launch_fixed_offsets(unsigned long long* offsets, uint64_t n, uint64_t first,
                                 uint32_t maxbits, cudaStream_t s);
// Parallel index of a general-mode stream (gzfp_index_chain.cuh): the sample
// of its exponents, and per batch of segments the table (from headers in
// the sampled range, or by walks) and the true chain's block starts.
struct IndexLists {
  uint32_t* first;   // window bits the link kernels start from
  uint32_t* count;   // of them
  uint32_t* next;    // taken so far
};
struct IndexLinks {
  uint32_t n1, n2;               // groups of segments, top groups
  uint32_t* exits;               // nseg * (win + 1) (index_exit)
  IndexHop *hops1, *hops2;       // n1, n2 times (win + 1)
  uint32_t *entry0, *entry1, *entry2;  // nseg, n1, n2: the true chain's entries
  unsigned long long *base0, *base1, *base2;  // blocks before them
};
template <typename T>
cudaError_t launch_index_sample(int dims, const IndexJob& j, IndexState* st, uint64_t avg,
                                int sms, cudaStream_t s);
template <typename T>
cudaError_t launch_index_fill(int dims, const IndexJob& j, const IndexLists& l,
                              const IndexState* st, bool heads, int sms, cudaStream_t s);
cudaError_t launch_index_zero(const IndexJob& j, const IndexLists& l, const IndexState* st, int sms,
                              cudaStream_t s);
cudaError_t launch_index_link(const IndexJob& j, const IndexLists& lists, const IndexLinks& l,
                              int sms, IndexState* st, unsigned long long* offsets,
                              cudaStream_t s);

cudaError_t launch_place_blocks(const uint64_t* scratch, uint32_t slot_words,
                                const uint32_t* lengths, const unsigned long long* offsets,
                                uint64_t nblocks, uint64_t bits, uint64_t* out, cudaStream_t s);

}  // namespace gzfp
