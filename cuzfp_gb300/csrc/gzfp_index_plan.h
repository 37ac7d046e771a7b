// gzfp_index_plan.h -- how the parallel block index cuts a stream into
// segments and batches, and what its workspace holds (gzfp_index_chain.cuh,
// gzfp_modes_api.cu).  No CUDA calls: the CPU tests build it on its own.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include "gzfp_index_chain.cuh"

namespace gzfp {

// A batch covers at most this many bits of the stream (its table takes two
// bytes a bit), and its workspace takes at most this many bytes: a segment's
// maps have an entry per bit of the longest block, so that many short segments
// of long blocks would take several times what the table does.
constexpr uint64_t kIndexBatchBits = 1ull << 28;
constexpr size_t kIndexWorkspace = 1ull << 30;
constexpr uint32_t kIndexLeastSegments = 64;  // the shortest batch, when memory is short

struct IndexPlan {
  uint32_t win, seg_bits;  // longest block; bits per segment
  uint64_t nseg;           // segments of the stream
  uint32_t per, fan;       // segments per batch; per group
  uint32_t n1, n2;         // groups, top groups
  // the workspace: where its parts begin, and its bytes
  size_t state, counters, table, first, exits, hops1, hops2, entry, base, bytes;
};

// The plan for batches of `per` segments.
inline void index_carve(IndexPlan& p, uint32_t per) {
  p.per = per;
  p.fan = 0;
  while ((uint64_t)p.fan * p.fan * p.fan < per) p.fan++;
  p.n1 = (per + p.fan - 1) / p.fan;
  p.n2 = (p.n1 + p.fan - 1) / p.fan;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t a = at;
    at += (bytes + 255) / 256 * 256;
    return a;
  };
  const size_t maps = (size_t)p.win + 1, nodes = (size_t)per + p.n1 + p.n2;
  p.state = take(sizeof(IndexState));
  p.counters = take(2 * sizeof(uint32_t));
  p.table = take((size_t)per * p.seg_bits * 2);
  p.first = take(per * (maps + 1) * 4);
  p.exits = take(per * maps * 4);
  p.hops1 = take(p.n1 * maps * sizeof(IndexHop));
  p.hops2 = take(p.n2 * maps * sizeof(IndexHop));
  p.entry = take(nodes * 4);
  p.base = take(nodes * 8);
  p.bytes = at;
}

// span: the stream's bits (at least 1); win: the longest block, below 32,768;
// heads: by headers, not by walks.
inline IndexPlan index_plan(uint64_t span, uint64_t nblocks, uint32_t win, bool heads) {
  const uint64_t avg = span / nblocks + 1;
  IndexPlan p;
  p.win = win;
  // Segments of about 24 blocks: the link kernels follow a segment's blocks,
  // and the segments of a group, one dependent load after another.  Of a short
  // stream shorter ones, so that there are some hundred; some dozen where every
  // bit of a segment's window is walked from (3D i32, 28 bits of precision: 36
  // blocks 250 -> 115 us, but 4624 blocks in some hundred 402 -> 510).
  const uint64_t few = heads ? 1024 : 64;
  p.seg_bits = 1024;
  while (p.seg_bits < 32768 &&
         (p.seg_bits <= win || (p.seg_bits < 16 * avg && span / p.seg_bits > few)))
    p.seg_bits *= 2;
  p.nseg = (span + p.seg_bits - 1) / p.seg_bits;
  uint64_t per = kIndexBatchBits / p.seg_bits;
  index_carve(p, (uint32_t)(p.nseg < per ? p.nseg : per));
  while (p.bytes > kIndexWorkspace) index_carve(p, p.per - (p.per + 15) / 16);
  return p;
}

// Streams that one thread walks, block after block, in less time than the
// parallel index's launches take: of up to 32 blocks, or of a few more with few
// planes and bits (35 1D blocks of 12 planes: floats 85 us, in parallel 96,
// int32 73, 104; 68: int32 109, 130, but floats, of more bits, 127, 104; 35
// blocks of int64 with 28 planes 118, 104).  prec: planes of a block at most.
inline bool index_serially(uint64_t span, uint64_t nblocks, uint32_t prec) {
  return nblocks <= 32 || (nblocks * prec <= 832 && span <= 2048);
}

// The workspace by `alloc` (0: had; 1: no memory; other: failed), for batches
// a quarter as long where there is no memory, down to kIndexLeastSegments.
// Returns what the last `alloc` did.
template <class Alloc>
int index_reserve(IndexPlan& p, Alloc&& alloc) {
  for (;;) {
    const int r = alloc(p.bytes);
    if (r != 1 || p.per <= kIndexLeastSegments) return r;
    index_carve(p, (p.per + 3) / 4);
  }
}

}  // namespace gzfp
