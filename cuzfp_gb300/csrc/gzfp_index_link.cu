// Type-independent kernels of the parallel block index: the table's zeroing,
// the exits of every candidate, their composition over groups of segments, and the descent of
// the true chain to every segment's block starts (gzfp_index_chain.cuh).
#include "gzfp_index_chain.cuh"
#include "gzfp_launch.h"

namespace gzfp {

constexpr int kLinkThreads = 256;
constexpr int kResolveThreads = 1024;

// stream words, zero past the end
struct IndexWords {
  const uint64_t* in;
  uint64_t n;
  __device__ __forceinline__ uint64_t load(uint64_t i) const { return i < n ? __ldg(in + i) : 0; }
};

// The table and the list's counters, zero.  Up to 8 CTAs an SM write 16 bytes
// a thread and step (the table's size is a multiple of 2 KB); as fast as
// cudaMemsetAsync, which cannot be left out on the device's word.
constexpr int kZeroThreads = 256;
__global__ void __launch_bounds__(kZeroThreads)
    index_zero_kernel(IndexJob j, IndexLists l, const IndexState* st) {
  if (index_over(*st)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) *l.count = *l.next = 0;
  uint4* t = reinterpret_cast<uint4*>(j.table);
  const uint32_t n = j.nseg * (j.seg_bits / 8), step = gridDim.x * kZeroThreads;
  for (uint64_t i = blockIdx.x * kZeroThreads + threadIdx.x; i < n; i += step)
    t[i] = make_uint4(0, 0, 0, 0);
}

// exits of the listed window bits
__global__ void __launch_bounds__(kLinkThreads)
    index_exits_kernel(IndexJob j, const uint32_t* __restrict__ list,
                       const uint32_t* __restrict__ count, uint32_t* exits, const IndexState* st) {
  const uint32_t n = index_over(*st) ? 0 : *count;
  for (uint64_t i = (uint64_t)blockIdx.x * kLinkThreads + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * kLinkThreads) {
    const uint32_t p = list[i], s = p / j.seg_bits, w = p - s * j.seg_bits;
    exits[(size_t)s * (j.win + 1) + w] = index_exit(j, IndexWords{j.in, j.nwords}, s, w);
  }
}

// hops of groups of `fan`: from window exits (FIRST) or from hops
template <bool FIRST>
__global__ void __launch_bounds__(kLinkThreads)
    index_compose_kernel(IndexJob j, const uint32_t* exits, const IndexHop* below, uint32_t n,
                         IndexHop* out, const IndexState* st) {
  if (index_over(*st)) return;
  const uint32_t w = blockIdx.x * kLinkThreads + threadIdx.x, g = blockIdx.y;
  if (w > j.win) return;
  out[(size_t)g * (j.win + 1) + w] = index_compose(g, j.fan, n, w, [&](uint32_t i, uint32_t e) {
    return FIRST ? index_hop(j, exits, i, e) : below[(size_t)i * (j.win + 1) + e];
  });
}

// One CTA: the true chain's entry and block count at every top group, group
// and segment.
__global__ void __launch_bounds__(kResolveThreads)
    index_resolve_kernel(IndexJob j, IndexLinks l, IndexState* st) {
  const uint32_t t = threadIdx.x;
  if (t == 0) {
    uint32_t w = kIndexNone;
    if (!st->done && !st->broken && st->pos >= j.lo) {
      if (st->pos - j.lo <= j.win)
        w = (uint32_t)(st->pos - j.lo);
      else
        st->broken = 1;
    }
    index_descend(0, l.n2, l.n2, w, st->count, j.nblocks, l.entry2, l.base2,
                  [&](uint32_t i, uint32_t e) { return l.hops2[(size_t)i * (j.win + 1) + e]; });
  }
  __syncthreads();
  for (uint32_t g = t; g < l.n2; g += kResolveThreads)
    index_descend(g, j.fan, l.n1, l.entry2[g], l.base2[g], j.nblocks, l.entry1, l.base1,
                  [&](uint32_t i, uint32_t e) { return l.hops1[(size_t)i * (j.win + 1) + e]; });
  __syncthreads();
  for (uint32_t g = t; g < l.n1; g += kResolveThreads)
    index_descend(g, j.fan, j.nseg, l.entry1[g], l.base1[g], j.nblocks, l.entry0, l.base0,
                  [&](uint32_t i, uint32_t e) { return index_hop(j, l.exits, i, e); });
}

__global__ void __launch_bounds__(kLinkThreads)
    index_emit_kernel(IndexJob j, IndexLinks l, unsigned long long* offsets, IndexState* st) {
  const uint32_t s = blockIdx.x * kLinkThreads + threadIdx.x;
  if (s < j.nseg) index_emit(j, IndexWords{j.in, j.nwords}, s, l.entry0[s], l.base0[s], offsets, st);
}

cudaError_t launch_index_zero(const IndexJob& j, const IndexLists& l, const IndexState* st, int sms,
                              cudaStream_t s) {
  const uint32_t most = (uint32_t)sms * 8, need = (j.nseg * (j.seg_bits / 8) + kZeroThreads - 1) / kZeroThreads;
  index_zero_kernel<<<need < most ? need : most, kZeroThreads, 0, s>>>(j, l, st);
  return cudaGetLastError();
}

cudaError_t launch_index_link(const IndexJob& j, const IndexLists& lists, const IndexLinks& l,
                              int sms, IndexState* st, unsigned long long* offsets,
                              cudaStream_t s) {
  const unsigned wx = (j.win + kLinkThreads) / kLinkThreads;
  index_exits_kernel<<<sms * 8, kLinkThreads, 0, s>>>(j, lists.first, lists.count, l.exits, st);
  index_compose_kernel<true><<<dim3(wx, l.n1), kLinkThreads, 0, s>>>(j, l.exits, nullptr, j.nseg,
                                                                     l.hops1, st);
  index_compose_kernel<false><<<dim3(wx, l.n2), kLinkThreads, 0, s>>>(j, nullptr, l.hops1, l.n1,
                                                                      l.hops2, st);
  index_resolve_kernel<<<1, kResolveThreads, 0, s>>>(j, l, st);
  index_emit_kernel<<<(j.nseg + kLinkThreads - 1) / kLinkThreads, kLinkThreads, 0, s>>>(
      j, l, offsets, st);
  return cudaGetLastError();
}

}  // namespace gzfp
