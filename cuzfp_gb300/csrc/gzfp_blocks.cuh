// gzfp_blocks.cuh -- random access to single blocks of a fixed-rate stream.
//
// A list of block indices, each coded from or into its own tile of 4^D
// values (x fastest) in a block buffer: zfp's per-block API
// (zfp_encode_block_* / zfp_decode_block_* and the partial-block forms,
// Z/inc/zfp.h:452-521) as its compressed arrays use it to write back and
// fetch cached blocks (Z/array/zfparray3.h:225-255): block `index` occupies
// bits [index * maxbits, (index + 1) * maxbits) of the stream.  One thread
// per listed block, with the plain path's per-block codec.
#pragma once

#include "gzfp_kernels.cuh"

namespace gzfp {

// zfp's partial-block shape code (Z/array/zfpcodecd.h:5-75): two bits per
// axis, x lowest, each 4 minus the block's extent along that axis.
// Entry i of a list is coded as a one-block field of those extents whose
// values sit in the 4^D tile (strides 1, 4, 16) and whose block starts at
// the slot's first bit.
template <int D>
__device__ __forceinline__ Geom tile_geom(uint32_t shape, uint64_t slot_bit, uint32_t vec) {
  Geom g;
  g.nx = 4 - (shape & 3u);
  g.ny = D >= 2 ? 4 - ((shape >> 2) & 3u) : 1;
  g.nz = D >= 3 ? 4 - ((shape >> 4) & 3u) : 1;
  g.bx = g.by = g.bz = 1;
  g.nblocks = 1;
  g.sx = 1;
  g.sy = 4;
  g.sz = 16;
  g.base = slot_bit;
  g.vec = vec;
  g.dbx = g.dby = FastDiv{1, 1, 0};
  return g;
}

// Clear the stream bits [pos, pos + n) in the words the slot shares with its
// neighbours, so that a rewritten block can be merged in.  The slot's inner
// words are overwritten whole by the bit writer.  Neighbouring slots clear
// and merge disjoint bits of a shared word, so every order gives one result.
__device__ __forceinline__ void clear_slot_edges(uint64_t* words, uint64_t pos, uint32_t n) {
  const uint64_t end = pos + n;
  const uint64_t w0 = pos >> 6, w1 = end >> 6;  // first word, word holding bit `end`
  const uint32_t lo = (uint32_t)(pos & 63), hi = (uint32_t)(end & 63);
  if (lo || w1 == w0) {  // the first word is shared (or holds the whole slot)
    const uint64_t keep = lowmask64(lo) | (w1 == w0 ? ~lowmask64(hi) : 0ull);
    atomicAnd((unsigned long long*)(words + w0), (unsigned long long)keep);
  }
  if (hi && w1 != w0)  // the last word is shared
    atomicAnd((unsigned long long*)(words + w1), (unsigned long long)~lowmask64(hi));
}

// Copy the whole words of a warp's listed slots (lane t's starts at word
// `first`, if `on`) between the stream and the staged buffer (word j of lane t
// at buf[j * kStride + t]), 32 consecutive words or so at a time.
template <bool TO_GLOBAL>
__device__ __forceinline__ void slots_copy(uint64_t* buf, uint64_t* words, uint64_t first, bool on,
                                           uint32_t W, uint32_t bpw) {
  const uint32_t lane = threadIdx.x & 31, total = bpw * W;
  uint32_t t = lane / W, j = lane % W;
  const uint32_t dt = 32 / W, dj = 32 % W;
  const uint32_t act = __ballot_sync(0xffffffffu, on);
  for (uint32_t e = lane; e - lane < total; e += 32) {
    const uint32_t src = t < 32 ? t : 0;
    const uint32_t f0 = __shfl_sync(0xffffffffu, lo32(first), src);
    const uint32_t f1 = __shfl_sync(0xffffffffu, hi32(first), src);
    if (e < total && (act >> src & 1)) {
      uint64_t* g = words + (((uint64_t)f1 << 32) | f0) + j;
      if (TO_GLOBAL)
        *g = buf[j * kStride + t];
      else
        buf[j * kStride + t] = __ldg(g);
    }
    t += dt;
    j += dj;
    if (j >= W) {
      j -= W;
      t++;
    }
  }
}

// STAGED: slots of whole words (blocks_stage says how many) go through
// shared memory, so that a warp reads or writes its slots' words with
// coalesced accesses instead of one dependent access per lane and word
// (3D f64, rate 16, read and written: 20,000 blocks 53.7 -> 49.7 us, 2,000
// blocks 40.5 -> 36.9; f32 42.4 -> 39.7, 28.7 -> 25.6).
template <int D, typename T, bool STAGED>
__global__ void __launch_bounds__(kThreads, (MinBlocks<D, T>::value))
    encode_blocks_kernel(const T* __restrict__ tiles, const unsigned long long* __restrict__ index,
                         const uint8_t* __restrict__ shape, uint64_t count, uint32_t maxbits,
                         uint64_t* __restrict__ out, uint64_t nwords, uint32_t bpw, uint32_t vec) {
  extern __shared__ __align__(16) uint64_t smem[];
  const Tables tables = stage_tables<D, T, false, kThreads>(smem);
  tables_ready<D, T, false>();
  uint64_t* planes = smem + table_words<D, T, false>();
  SmemPlanes ps{planes + threadIdx.x, tables};
  const uint64_t i = lane_block(warp_first_block(bpw), bpw);
  const uint64_t slot = i < count ? index[i] : ~0ull;
  const bool on = slot < nwords * 64 / maxbits;  // slots past the stream are skipped
  const uint64_t pos = slot * maxbits;
  const Geom g = tile_geom<D>(on && shape ? shape[i] : 0u, pos, vec);
  const T* tile = tiles + i * (1u << (2 * D));
  if constexpr (STAGED) {
    const uint32_t W = maxbits >> 6;
    uint64_t* buf = planes + store_slots<D, T>() * kThreads;
    if (on)
      encode_one<D, T, true>(tile, g, 0, maxbits,
                             StagedWords<kStride>{buf + threadIdx.x, slot * W, W}, ps);
    __syncwarp();
    slots_copy<true>(buf + (threadIdx.x & ~31u), out, slot * W, on, W, bpw);
  } else if (on) {
    clear_slot_edges(out, pos, maxbits);
    encode_one<D, T>(tile, g, 0, maxbits, DevWords{out, nullptr, nwords}, ps);
  }
}

template <int D, typename T, bool STAGED>
__global__ void __launch_bounds__(kThreads, (MinBlocks<D, T>::value))
    decode_blocks_kernel(const uint64_t* __restrict__ in, uint64_t nwords,
                         const unsigned long long* __restrict__ index,
                         const uint8_t* __restrict__ shape, uint64_t count, uint32_t maxbits,
                         T* __restrict__ tiles, uint32_t bpw, uint32_t vec) {
  extern __shared__ __align__(16) uint64_t smem[];
  const bool use = D != 3 || groups_by_table<T>(FixedRate{maxbits});
  const Tables tables = stage_tables<D, T, true, kThreads>(smem, use);
  uint64_t* planes = smem + table_words<D, T, true>();
  SmemPlanes ps{planes + threadIdx.x, tables};
  const uint64_t i = lane_block(warp_first_block(bpw), bpw);
  const uint64_t slot = i < count ? index[i] : ~0ull;
  const bool on = slot < nwords * 64 / maxbits;  // slots past the stream are skipped
  const Geom g = tile_geom<D>(on && shape ? shape[i] : 0u, slot * maxbits, vec);
  T* tile = tiles + i * (1u << (2 * D));
  if constexpr (STAGED) {
    const uint32_t W = maxbits >> 6;
    uint64_t* buf = planes + decode_slots<D, T>() * kThreads;
    slots_copy<false>(buf + (threadIdx.x & ~31u), (uint64_t*)in, slot * W, on, W, bpw);
#pragma unroll
    for (uint32_t j = 0; j < kPadRows; j++) buf[(W + j) * kStride + threadIdx.x] = 0;
    __syncwarp();
    tables_ready<D, T, true>(use);
    if (on)
      decode_one<D, T>(tile, g, 0, maxbits,
                       StagedWords<kStride>{buf + threadIdx.x, slot * W, W}, ps);
  } else {
    tables_ready<D, T, true>(use);
    if (on) decode_one<D, T>(tile, g, 0, maxbits, StreamWords<D>{in, nwords}, ps);
  }
}

// Words of the longest staged slot.  Encoder: as elsewhere.  Decoder: longer
// slots too, up to the 32 words of rate 32, where the reads' latency counts for
// more than the shared memory: 3D f64, read and written, 30,000 blocks at rate
// 24 69.7 -> 62.4 us, rate 31 77.3 -> 68.5, 200,000 blocks 284 -> 261, 318 ->
// 288; f32, rate 31, 13,766 blocks 42.8 -> 40.8.  For values of 32 bits in a
// list that fills the chip several times over, resident warps count for more:
// 200,000 blocks at rate 31 186 -> 194 us, so those keep reading the stream, as
// do slots over 32 words (f64, rate 48, 200,000 blocks: 367 -> 401).
constexpr uint32_t kMaxStagedSlot = 32;
constexpr uint64_t kLongList = 1u << 16;

inline int blocks_stage(uint32_t maxbits, uint32_t max_words) {
  return maxbits % 64 == 0 && maxbits <= 64 * max_words ? kStageRows : kStageNone;
}

template <int D, typename T>
cudaError_t launch_encode_blocks_t(const T* tiles, const unsigned long long* index,
                                   const uint8_t* shape, uint64_t count, uint32_t maxbits,
                                   uint64_t* out, uint64_t nwords, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  const uint32_t bpw = blocks_per_warp(count, 0);
  const int stage = blocks_stage(maxbits, kMaxStagedOut);
  const size_t sm = smem_bytes(store_slots<D, T>(), stage, maxbits, table_words<D, T, false>());
  auto k = stage == kStageRows ? encode_blocks_kernel<D, T, true> : encode_blocks_kernel<D, T, false>;
  cudaError_t e = allow_smem(k, sm);
  if (e != cudaSuccess) return e;
  const uint32_t vec = (uintptr_t)tiles % (4 * sizeof(T)) == 0 ? 1u : 0u;
  k<<<grid_ctas(count, bpw), kThreads, sm, s>>>(tiles, index, shape, count, maxbits, out, nwords,
                                               bpw, vec);
  return cudaGetLastError();
}

template <int D, typename T>
cudaError_t launch_decode_blocks_t(const uint64_t* in, uint64_t nwords,
                                   const unsigned long long* index, const uint8_t* shape,
                                   uint64_t count, uint32_t maxbits, T* tiles, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  const uint32_t bpw = blocks_per_warp(count, 0);
  const int stage = blocks_stage(
      maxbits, sizeof(T) == 8 || count <= kLongList ? kMaxStagedSlot : kMaxStagedOut);
  const size_t sm = smem_bytes(decode_slots<D, T>(), stage, maxbits, table_words<D, T, true>());
  auto k = stage == kStageRows ? decode_blocks_kernel<D, T, true> : decode_blocks_kernel<D, T, false>;
  cudaError_t e = allow_smem(k, sm);
  if (e != cudaSuccess) return e;
  const uint32_t vec = (uintptr_t)tiles % (4 * sizeof(T)) == 0 ? 1u : 0u;
  k<<<grid_ctas(count, bpw), kThreads, sm, s>>>(in, nwords, index, shape, count, maxbits, tiles,
                                               bpw, vec);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_encode_blocks(int dims, const T* tiles, const unsigned long long* index,
                                 const uint8_t* shape, uint64_t count, uint32_t maxbits,
                                 uint64_t* out, uint64_t nwords, cudaStream_t s) {
  switch (dims) {
    case 1: return launch_encode_blocks_t<1, T>(tiles, index, shape, count, maxbits, out, nwords, s);
    case 2: return launch_encode_blocks_t<2, T>(tiles, index, shape, count, maxbits, out, nwords, s);
    case 3: return launch_encode_blocks_t<3, T>(tiles, index, shape, count, maxbits, out, nwords, s);
    default: return cudaErrorInvalidValue;
  }
}

template <typename T>
cudaError_t launch_decode_blocks(int dims, const uint64_t* in, uint64_t nwords,
                                 const unsigned long long* index, const uint8_t* shape,
                                 uint64_t count, uint32_t maxbits, T* tiles, cudaStream_t s) {
  switch (dims) {
    case 1: return launch_decode_blocks_t<1, T>(in, nwords, index, shape, count, maxbits, tiles, s);
    case 2: return launch_decode_blocks_t<2, T>(in, nwords, index, shape, count, maxbits, tiles, s);
    case 3: return launch_decode_blocks_t<3, T>(in, nwords, index, shape, count, maxbits, tiles, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gzfp
