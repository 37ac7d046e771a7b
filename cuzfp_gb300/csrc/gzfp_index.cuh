// gzfp_index.cuh -- the type-dependent kernels of the parallel block index
// (gzfp_index_chain.cuh): sampling, headers and walks.
#pragma once

#include "gzfp_index_chain.cuh"
#include "gzfp_kernels.cuh"
#include "gzfp_launch.h"

namespace gzfp {

// Readers (BlockParse).  Over stream words in shared memory, 32-bit word i at
// buf[i], bit 0 of the buffer being bit `origin` from the job's
// first; and over the stream in device memory (zeros past its end).
// t: the tables, in shared memory.
struct IndexStagedReader {
  const uint32_t* buf;
  const IndexTables* t;
  uint32_t origin;
  __device__ __forceinline__ uint32_t peek32(uint32_t p) const {
    const uint32_t b = p - origin;
    const uint32_t* w = buf + (b >> 5);
    return __funnelshift_r(w[0], w[1], b & 31);
  }
};

struct IndexStreamReader {
  const uint32_t* in;
  const IndexTables* t;
  uint64_t lo, n;  // the job's first bit; 32-bit words in the stream
  __device__ __forceinline__ uint32_t peek32(uint32_t p) const {
    const uint64_t b = lo + p, i = b >> 5;
    const uint32_t a = i < n ? __ldg(in + i) : 0u, c = i + 1 < n ? __ldg(in + i + 1) : 0u;
    return __funnelshift_r(a, c, (uint32_t)b & 31);
  }
};

constexpr uint32_t kLaneAll = 0xffffffffu;
constexpr int kSampleThreads = 256;
constexpr int kWindowThreads = 256;
constexpr int kWalkThreads = 64;

__device__ __forceinline__ void stage_index_tables(IndexTables* t, int threads) {
  const uint32_t* src = reinterpret_cast<const uint32_t*>(&kIndexTables);
  for (uint32_t i = threadIdx.x; i < sizeof(IndexTables) / 4; i += threads)
    reinterpret_cast<uint32_t*>(t)[i] = src[i];
}

// A warp's idle lanes take the next entries of a list with one atomic.
__device__ __forceinline__ uint32_t take_next(uint32_t* next, uint32_t idle) {
  const int lane = threadIdx.x & 31, leader = __ffs(idle) - 1;
  uint32_t i = 0;
  if (lane == leader) i = atomicAdd(next, __popc(idle));
  return __shfl_sync(kLaneAll, i, leader) + __popc(idle & ((1u << lane) - 1));
}

// Step 1, one CTA per sampled place: each lane walks from every 256th bit of
// `bits` (IndexSampler), the words staged in shared memory.
template <int D, typename T>
__global__ void __launch_bounds__(kSampleThreads)
    index_sample_kernel(IndexJob j, uint64_t stride_words, uint32_t bits, uint32_t limit,
                        uint32_t nw, IndexState* st) {
  extern __shared__ uint64_t smem[];
  __shared__ IndexTables tables;
  stage_index_tables(&tables, kSampleThreads);
  const DevWords in{nullptr, j.in, j.nwords};
  const uint64_t w0 = (j.lo >> 6) + blockIdx.x * stride_words;
  for (uint32_t i = threadIdx.x; i < nw; i += kSampleThreads) smem[i] = in.load(w0 + i);
  __syncthreads();
  const IndexStagedReader r{reinterpret_cast<const uint32_t*>(smem), &tables, 0};
  const IndexRange open = index_open<D, T>(j.mode);
  IndexSampler<D, T, IndexStagedReader> walk;
  uint32_t p = threadIdx.x;
  bool live = false;
  for (;;) {
    if (!live && p < bits) {
      live = r.peek32(p) & 1;
      if (live) walk.start(p, limit);
      p += kSampleThreads;
    }
    if (!__ballot_sync(kLaneAll, live || p < bits)) return;
    if (live) {
      live = walk.tick(j.mode, open, r);
      if (!live && walk.kept) {
        atomicMin(&st->field_lo, (unsigned)walk.lo);
        atomicMax(&st->field_hi, (unsigned)walk.hi);
      }
    }
  }
}

// Step 2, one warp per `chunk` bits: their words staged in shared memory, 32 bits a
// lane searched for headers at a time (index_heads), the headers listed, and
// each lane parses listed blocks until none is left.  Those in the window, and
// the window's end, go to the global list that the link kernels start from.
// Bound by issue: searching takes 40 instructions per 1024 bits, a 4^3 block
// about 30 steps of 40 instructions.
constexpr uint32_t kHeadsRoom = 256 + 1024;  // listed before parsing, one search
template <int D, typename T>
__global__ void __launch_bounds__(32)
    index_parse_kernel(IndexJob j, IndexLists l, uint32_t chunk, uint32_t nw,
                       const IndexState* st) {
  typedef IndexStagedReader R;
  extern __shared__ uint64_t smem[];
  __shared__ IndexTables tables;
  __shared__ uint16_t heads[kHeadsRoom];
  __shared__ uint32_t s_next;
  if (index_over(*st)) return;
  const uint32_t lane = threadIdx.x, at0 = blockIdx.x * chunk;
  const uint32_t size = umin(chunk, j.nseg * j.seg_bits - at0), sh = (uint32_t)(j.lo & 63);
  stage_index_tables(&tables, 32);
  const DevWords in{nullptr, j.in, j.nwords};
  const uint64_t w0 = (j.lo + at0) >> 6;
#pragma unroll 4
  for (uint32_t i = lane; i < nw; i += 32) smem[i] = in.load(w0 + i);
  const uint32_t* words = reinterpret_cast<const uint32_t*>(smem);
  const R r{words, &tables, at0 - sh};
  const IndexRange range = index_range<D, T>(j.mode, st->field_lo, st->field_hi);
  __syncwarp();
  auto list_entry = [&](bool is, uint32_t p) {  // all lanes
    const uint32_t m = __ballot_sync(kLaneAll, is);
    if (!m) return;
    const uint32_t at = take_next(l.count, m);
    if (is) l.first[at] = at0 + p;
  };
  for (uint32_t q = (0u - at0) & (j.seg_bits - 1); q < size; q += 32 * j.seg_bits)
    list_entry(q + lane * j.seg_bits < size, q + lane * j.seg_bits + j.win);
  list_entry(lane == 0 && at0 == 0, 0);
  BlockParse<D, T, R> parse;
  for (uint32_t g = 0; g < size / 32;) {
    uint32_t n = 0;
    while (n <= kHeadsRoom - 1024 && g < size / 32) {
      const uint32_t q = g + lane, i = q + (sh >> 5);
      uint32_t m = q < size / 32
                       ? index_heads<T>(words[i], words[i + 1], words[i + 2], sh & 31, range)
                       : 0;
      uint32_t before = __popc(m);  // inclusive scan
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kLaneAll, before, o);
        if (lane >= (uint32_t)o) before += v;
      }
      uint32_t at = n + before - __popc(m);
      n += __shfl_sync(kLaneAll, before, 31);
      for (; m; m &= m - 1) heads[at++] = (uint16_t)(q * 32 + ctz32(m));
      g += 32;
    }
    if (lane == 0) s_next = 0;
    __syncwarp();
    for (uint32_t i = lane; i - lane < n; i += 32)
      list_entry(i < n && ((at0 + heads[i]) & (j.seg_bits - 1)) < j.win, i < n ? heads[i] : 0u);
    bool live = false, more = true;
    for (;;) {
      const uint32_t idle = __ballot_sync(kLaneAll, !live && more);
      if (idle) {
        const uint32_t i = take_next(&s_next, idle);
        if (!live && more) {
          more = live = i < n;
          if (live) {
            const uint32_t p = at0 + heads[i];
            live = !parse.begin(p, block_head<D, T>(r.peek32(p), j.mode));
            if (!live) j.table[p] = (uint16_t)parse.used(j.mode);
          }
        }
      }
      if (!__ballot_sync(kLaneAll, live)) break;
      if (live) {
#pragma unroll 1
        for (int k = 0; k < IndexLane<D, T, R>::kSteps && live; k++) live = !parse.step(r);
        if (!live) j.table[parse.start] = (uint16_t)parse.used(j.mode);
      }
    }
    __syncwarp();  // the list is reused
  }
}

// The window bits where a block could start, without a range of exponents:
// one CTA per segment, one atomic each.
template <int D, typename T>
__global__ void __launch_bounds__(kWindowThreads)
    index_window_kernel(IndexJob j, IndexLists l, const IndexState* st) {
  __shared__ uint32_t s_warp[kWindowThreads / 32];
  if (index_over(*st)) return;
  const uint32_t s = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const DevWords in{nullptr, j.in, j.nwords};
  auto is = [&](uint32_t p) {
    if (p > j.win) return false;
    if (FT<T>::INT || !j.zeros || p == j.win || (p == 0 && s == 0)) return true;
    const uint64_t b = j.lo + (uint64_t)s * j.seg_bits + p;
    return ((in.load(b >> 6) >> (b & 63)) & 1) != 0;
  };
  uint32_t mine = 0;
  for (uint32_t p0 = warp * 32; p0 <= j.win; p0 += kWindowThreads)
    mine += __popc(__ballot_sync(kLaneAll, is(p0 + lane)));
  if (lane == 0) s_warp[warp] = mine;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t all = 0;
    for (int i = 0; i < kWindowThreads / 32; i++) all += s_warp[i];
    uint32_t at = atomicAdd(l.count, all);
    for (int i = 0; i < kWindowThreads / 32; i++) {
      const uint32_t c = s_warp[i];
      s_warp[i] = at;
      at += c;
    }
  }
  __syncthreads();
  uint32_t at = s_warp[warp];
  for (uint32_t p0 = warp * 32; p0 <= j.win; p0 += kWindowThreads) {
    const bool c = is(p0 + lane);
    const uint32_t m = __ballot_sync(kLaneAll, c);
    if (c) l.first[at + __popc(m & ((1u << lane) - 1))] = s * j.seg_bits + p0 + lane;
    at += __popc(m);
  }
}

// Each lane takes listed bits until none is left and walks from them to the
// segment's end or to where another walk has been (IndexLane).
template <int D, typename T>
__global__ void __launch_bounds__(kWalkThreads)
    index_walk_kernel(IndexJob j, IndexLists l, const IndexState* st) {
  typedef IndexStreamReader R;
  __shared__ IndexTables tables;
  const uint32_t n = index_over(*st) ? 0 : *l.count;
  stage_index_tables(&tables, kWalkThreads);
  __syncthreads();
  const R r{reinterpret_cast<const uint32_t*>(j.in), &tables, j.lo, j.nwords * 2};
  IndexLane<D, T, R> walk;
  bool live = false, more = true;
  for (;;) {
    const uint32_t idle = __ballot_sync(kLaneAll, !live && more);
    if (idle) {
      const uint32_t i = take_next(l.next, idle);
      if (!live && more) {
        more = live = i < n;
        if (live) walk.start(j, l.first[i]);
      }
    }
    if (!__ballot_sync(kLaneAll, live)) return;
    if (live) live = walk.tick(j, r);
  }
}

// The table and the list of one batch of segments.
template <int D, typename T>
cudaError_t launch_index_fill_t(const IndexJob& j, const IndexLists& l, const IndexState* st,
                                bool heads, int sms, cudaStream_t s) {
  const cudaError_t e = launch_index_zero(j, l, st, sms, s);
  if (e != cudaSuccess) return e;
  if (heads) {
    const IndexStage g = index_parse_stage(j, sms);
    const uint64_t chunks = ((uint64_t)j.nseg * j.seg_bits + g.bits - 1) / g.bits;
    index_parse_kernel<D, T><<<(unsigned)chunks, 32, (size_t)g.words * 8, s>>>(j, l, g.bits,
                                                                               g.words, st);
  } else {
    index_window_kernel<D, T><<<j.nseg, kWindowThreads, 0, s>>>(j, l, st);
    index_walk_kernel<D, T><<<sms * 16, kWalkThreads, 0, s>>>(j, l, st);
  }
  return cudaGetLastError();
}

// Sample the stream's exponents into st.
template <int D, typename T>
cudaError_t launch_index_sample_t(const IndexJob& j, IndexState* st, uint64_t avg, int sms,
                                  cudaStream_t s) {
  const uint64_t span = j.nwords * 64 - j.lo;
  const IndexPlaces g = index_sample_stage<T>(span, avg, j.win, sms);
  index_sample_kernel<D, T><<<(unsigned)g.places, kSampleThreads, (size_t)g.words * 8, s>>>(
      j, span / 64 / g.places, g.bits, g.limit, g.words, st);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_index_fill(int dims, const IndexJob& j, const IndexLists& l,
                              const IndexState* st, bool heads, int sms, cudaStream_t s) {
  switch (dims) {
    case 1: return launch_index_fill_t<1, T>(j, l, st, heads, sms, s);
    case 2: return launch_index_fill_t<2, T>(j, l, st, heads, sms, s);
    case 3: return launch_index_fill_t<3, T>(j, l, st, heads, sms, s);
    default: return cudaErrorInvalidValue;
  }
}

template <typename T>
cudaError_t launch_index_sample(int dims, const IndexJob& j, IndexState* st, uint64_t avg,
                                int sms, cudaStream_t s) {
  switch (dims) {
    case 1: return launch_index_sample_t<1, T>(j, st, avg, sms, s);
    case 2: return launch_index_sample_t<2, T>(j, st, avg, sms, s);
    case 3: return launch_index_sample_t<3, T>(j, st, avg, sms, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gzfp
