// gzfp_kernels.cuh -- the plain-path CUDA kernels: one thread per zfp block.
//
// Encode: gather 4^D values (consecutive threads own consecutive blocks, so
// a warp's row loads are contiguous), run the block codec in registers,
// write the block's bits into its fixed-rate slot [b*maxbits, (b+1)*maxbits).
// Decode: the inverse, reading the slot and storing the valid values.
//
// Shared memory per CTA: each thread's plane store (the coder walks planes in
// a rolled loop), and a word buffer in which the stream's words are staged
// (kStage*): the decoder loads them with coalesced loads, and the encoder
// assembles them there and stores them with coalesced stores.
//
// Replaces cuZFP's cudaEncode / cudaEncode1 / cudaEncode2 and cudaDecode /
// cudaDecode1 / cudaDecode2 (src/cuZFP/encode{1,2,3}.cuh, decode{1,2,3}.cuh).
#pragma once

#include <cuda_runtime.h>

#include "gzfp_array.cuh"

namespace gzfp {

constexpr int kThreads = 128;            // threads (= blocks) per CTA
constexpr int kStride = kThreads + 1;    // staged word buffer row pitch (words)
constexpr uint32_t kMaxStagedWords = 64; // staged decode up to 4096-bit blocks
constexpr uint32_t kMaxStagedOut = 16;   // staged encoder output up to 1024-bit blocks
constexpr uint32_t kPadRows = 2;         // zero rows after each staged slot
// How a CTA reaches the stream's words.
// kStageNone: in place; the encoder ORs the words that neighbouring blocks
// share into a zeroed stream.
// kStageRows: blocks of whole words, word j of thread t's block at
// buf[j * kStride + t], so that the lanes of a warp hit different banks.
// kStageRun: the words of the CTA's 128 blocks in stream order.  These begin
// and end on word boundaries whatever the block's size is, so words are
// shared within the CTA only: no zeroing of the stream, no global atomics.
// 4-value blocks take it up to two words (their slots are short, so the
// lanes' words spread over the banks), others where blocks are not whole words.
// Against words reached in place, with the same coder (compress / decompress):
// 1D f32, 2^25 - 3 values, rate 12, 176 -> 121 / 177 -> 130 us; 1D f64, 2^24
// - 3, rate 12, 150 -> 90 / 137 -> 84; 2D f32 4093 x 4095, rate 11.3, 132 ->
// 126 / 145 -> 124; 3D f64 256^3, rate 15.3, 139 -> 133 / 126 -> 103; 3D f32
// 256^3, rate 15.3, 100 -> 92 / 77 -> 69.  (1D f64, rate 48: 154 -> 155 / 148
// -> 158.)
constexpr int kStageNone = 0, kStageRows = 1, kStageRun = 2;

// dynamic shared memory of a CTA: the plane store (up to 32 slots of 8
// bytes per thread), the tables, and the word buffer
inline size_t smem_bytes(int slots, int stage, uint32_t maxbits, int tables = 0) {
  size_t b = ((size_t)slots * kThreads + (size_t)tables) * 8;
  if (stage == kStageRows) b += (size_t)((maxbits >> 6) + kPadRows) * kStride * 8;
  if (stage == kStageRun) b += (size_t)(kThreads / 64 * maxbits + kPadRows) * 8;
  return b;
}

// Tables that a coder's CTAs copy into the start of their shared memory: the
// 4-value plane tables (1D, 1.6 KB) and the group table (4^3 decoders, 4 KB).
struct Tables {
  const Plane4Tables* t4;
  const GroupTable* gt;
};
template <int D, typename T, bool DECODE>
__host__ __device__ constexpr int table_words() {
  return D == 1 ? (int)(sizeof(Plane4Tables) / 8)
         : DECODE && uses_group_table<D, T>() ? (int)(sizeof(GroupTable) / 8)
                                              : 0;
}

// Start copying the coder's tables into shared memory (16 bytes aligned),
// and wait for them: the CTA's own staging goes between the two, so that the
// copies' latencies overlap.  Every thread of the CTA must call both before
// any thread returns, with the same `use` (is a table looked up at all);
// tables_ready is a CTA barrier where one is (and where ALWAYS is set).
template <int D, typename T, bool DECODE, int NT>
__device__ __forceinline__ Tables stage_tables(uint64_t* smem, bool use = true) {
  constexpr int n = table_words<D, T, DECODE>() / 2;  // 16-byte pieces
  if constexpr (n == 0) {
    return Tables{nullptr, nullptr};
  } else {
    const char* src = D == 1 ? reinterpret_cast<const char*>(&kPlane4Tables)
                             : reinterpret_cast<const char*>(&kGroupTable);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    if (use) {
#pragma unroll
      for (int i = threadIdx.x; i < n; i += NT)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i),
                     "l"(src + 16 * i) : "memory");
    }
    return Tables{reinterpret_cast<const Plane4Tables*>(smem),
                  reinterpret_cast<const GroupTable*>(smem)};
  }
}
template <int D, typename T, bool DECODE, bool ALWAYS = false>
__device__ __forceinline__ void tables_ready(bool use = true) {
  if constexpr (table_words<D, T, DECODE>() > 0) {
    if (use) asm volatile("cp.async.wait_all;" ::: "memory");
    if (use || ALWAYS) __syncthreads();
  } else if constexpr (ALWAYS) {
    __syncthreads();
  }
}
// per-thread plane store in shared memory, slot i at planes[i * kThreads]
struct SmemPlanes {
  uint64_t* p;
  const Plane4Tables* t4;
  const GroupTable* gt;
  __device__ __forceinline__ SmemPlanes(uint64_t* p_, const Tables& t) : p(p_), t4(t.t4), gt(t.gt) {}
  __device__ __forceinline__ uint64_t get(int i) const { return p[i * kThreads]; }
  __device__ __forceinline__ void put(int i, uint64_t v) { p[i * kThreads] = v; }
};

// Global stream words.  `merge` ORs a word that neighbouring zfp blocks share
// (only when maxbits is not a multiple of 64; the stream is zeroed first).
struct DevWords {
  uint64_t* out;
  const uint64_t* in;
  uint64_t n;  // words in the stream
  __device__ __forceinline__ void store(uint64_t i, uint64_t v) { out[i] = v; }
  __device__ __forceinline__ void merge(uint64_t i, uint64_t v) {
    atomicOr((unsigned long long*)(out + i), (unsigned long long)v);
  }
  __device__ __forceinline__ uint64_t load(uint64_t i) const { return i < n ? __ldg(in + i) : 0; }
};

// Global stream words for reading alone.  4^3 blocks: AHEAD, with a reader that
// loads the word behind the two that a peek spans before it is needed.  The
// group decoder looks at the stream up to twice a step, and waited for each new
// word (300^3, rates 6, 12, 24 behind a header: floats 139, 156, 190 -> 131,
// 143, 168 us, smooth 143, 168, 194 -> 133, 155, 170; noisy doubles 200, 224, 307
// -> 193, 205, 265; from start bits, 28 bits of precision, noisy: floats 134 ->
// 125, doubles 224 -> 190).  By token, with shorter steps, it costs more than it
// gives (int32 from start bits, precision 20: 58 -> 60).
template <bool AHEAD>
struct ReadWords {
  const uint64_t* in;
  uint64_t n;
  __device__ __forceinline__ uint64_t load(uint64_t i) const { return i < n ? __ldg(in + i) : 0; }
};
template <int D>
using StreamWords = ReadWords<D == 3>;

// One block's slot in the staged word buffer: word j of the block at
// buf[j * PITCH] (PITCH = threads per CTA + 1, so the 32 lanes of a warp
// hit 32 different banks); words past the slot read as zero.  The buffer has
// two zero rows after the last word of every slot (kPadRows), so a reader
// may load the two words at any bit position up to the slot's end.
template <int PITCH>
struct StagedWords {
  uint64_t* buf;
  uint64_t w0;  // global index of the slot's first word
  uint32_t W;   // words per block
  __device__ __forceinline__ void store(uint64_t i, uint64_t v) { buf[(i - w0) * PITCH] = v; }
  __device__ __forceinline__ void merge(uint64_t i, uint64_t v) { buf[(i - w0) * PITCH] |= v; }
  __device__ __forceinline__ uint64_t load(uint64_t i) const {
    uint64_t j = i - w0;
    return j < W ? buf[j * PITCH] : 0;
  }
};

// The words of a CTA's blocks in stream order in shared memory, zero at
// first: a word that neighbouring blocks share is merged with atomics on its
// halves.
struct RunWords {
  uint64_t* buf;
  uint64_t w0;  // global index of the first word
};
template <>
struct BitWriter<RunWords, false> {
  uint64_t* buf;
  uint64_t acc;
  uint32_t wi, fill, first, last;  // as the general writer's, within the buffer
  __device__ __forceinline__ BitWriter(RunWords w, uint64_t pos, uint32_t maxbits) : buf(w.buf), acc(0) {
    const uint32_t p = (uint32_t)(pos - (w.w0 << 6)), end = p + maxbits;
    wi = p >> 6;
    fill = p & 63;
    first = fill ? wi : ~0u;
    last = end & 63 ? end >> 6 : ~0u;
  }
  __device__ __forceinline__ void emit() {
    if (wi == first || wi == last) {
      uint32_t* h = reinterpret_cast<uint32_t*>(buf + wi);
      if (lo32(acc)) atomicOr(h, lo32(acc));
      if (hi32(acc)) atomicOr(h + 1, hi32(acc));
    } else {
      buf[wi] = acc;
    }
    wi++;
  }
  __device__ __forceinline__ void put(uint64_t v, uint32_t n) {
    acc |= v << fill;
    const uint32_t f = fill + n;
    if (f >= 64) {
      emit();
      acc = (v >> 1) >> (63 - fill);
      fill = f - 64;
    } else {
      fill = f;
    }
  }
  // the first n bits of a string, as the whole block (which starts at fill)
  template <int N>
  __device__ __forceinline__ void put_string(BitString<N> c, uint32_t n) {
    c.cut(n);
    uint64_t low = 0;
#pragma unroll
    for (int i = 0; i <= N; i++) {
      if ((uint32_t)(64 * i) >= fill + n) break;
      acc = (i < N ? c.w[i] << fill : 0) | ((low >> 1) >> (63 - fill));
      low = i < N ? c.w[i] : 0;
      emit();
    }
    fill = 0;
  }
  __device__ __forceinline__ void zeros(uint32_t) {}  // ends the block; the buffer is zero
  __device__ __forceinline__ void finish() {
    if (fill) emit();
  }
};

// Bit reader over a staged slot: only the bit position is kept, and a peek
// loads the two words it spans (the zero rows after the slot cover the end).
template <int PITCH>
struct BitReader<StagedWords<PITCH>> {
  const uint64_t* buf;
  uint32_t pos;  // bit position within the slot
  __device__ __forceinline__ BitReader(StagedWords<PITCH> w, uint64_t p)
      : buf(w.buf), pos((uint32_t)(p - (w.w0 << 6))) {}
  // (window64 written out: called, the 512^3 double decoder takes 0.3% longer)
  __device__ __forceinline__ uint64_t peek64() const {
    const uint32_t j = pos >> 6, s = pos & 63;
    const uint64_t a = buf[j * PITCH], b = buf[(j + 1) * PITCH];
    const uint32_t a0 = lo32(a), a1 = hi32(a), b0 = lo32(b), b1 = hi32(b);
    const bool ge = s >= 32;
    const uint32_t c0 = ge ? a1 : a0, c1 = ge ? b0 : a1, c2 = ge ? b1 : b0;
    const uint32_t t = s & 31;
    return ((uint64_t)__funnelshift_r(c1, c2, t) << 32) | __funnelshift_r(c0, c1, t);
  }
  __device__ __forceinline__ void skip(uint32_t n) { pos += n; }
  __device__ __forceinline__ uint64_t read(uint32_t n) {
    if (n == 0) return 0;
    const uint64_t v = peek64() & lowmask64(n);
    pos += n;
    return v;
  }
};

// Bit reader with a word loaded ahead.
template <>
struct BitReader<ReadWords<true>> {
  ReadWords<true> words;
  uint64_t wi;          // index of w0
  uint64_t w0, w1, w2;
  uint32_t off;
  __device__ __forceinline__ BitReader(ReadWords<true> w, uint64_t pos)
      : words(w), wi(pos >> 6), off((uint32_t)(pos & 63)) {
    w0 = words.load(wi);
    w1 = words.load(wi + 1);
    w2 = words.load(wi + 2);
  }
  __device__ __forceinline__ uint64_t peek64() const { return window64(w0, w1, off); }
  __device__ __forceinline__ void skip(uint32_t n) {  // n <= 64
    off += n;
    if (off >= 64) {
      off -= 64;
      wi++;
      w0 = w1;
      w1 = w2;
      w2 = words.load(wi + 2);
    }
  }
  __device__ __forceinline__ uint64_t read(uint32_t n) {
    if (n == 0) return 0;
    const uint64_t v = peek64() & lowmask64(n);
    skip(n);
    return v;
  }
};

// Copy a warp's 32 consecutive slots between the staged buffer (word j of
// lane t at buf[j * PITCH + t]) and the stream, 32 words per step.
template <bool TO_GLOBAL, int PITCH = kStride>
__device__ __forceinline__ void warp_copy(uint64_t* buf, uint64_t* gwords, uint32_t W,
                                          uint32_t nblocks_valid) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t total = nblocks_valid * W;
  uint32_t t = lane / W, j = lane % W;      // slot and word of element `lane`
  const uint32_t dt = 32 / W, dj = 32 % W;  // advance per step of 32 elements
  for (uint32_t gi = lane; gi < total; gi += 32) {
    if (TO_GLOBAL)
      gwords[gi] = buf[j * PITCH + t];
    else
      buf[j * PITCH + t] = __ldg(gwords + gi);
    t += dt;
    j += dj;
    if (j >= W) {
      j -= W;
      t++;
    }
  }
}

// Register budget: the 4^3 double kernels keep a whole block (64 x 64 bits)
// in registers; 168 registers per thread allow 3 CTAs of 128 threads per SM.
// The 1D kernels need few, and left to itself the compiler takes more (79
// for the float encoder: 22 warps per SM and 68% of the ALU pipe).
template <int D, typename T>
struct MinBlocks {
  static constexpr int value = D == 1 ? (sizeof(T) == 8 ? 10 : 16) : D == 3 && sizeof(T) == 8 ? 3 : 4;
};

// Plane-store slots per thread, as many as the block codec touches, so that
// shared memory does not cap the CTAs per SM below what registers allow:
// 4^3 blocks code and decode 32 planes at a time (32 slots; 64-bit values
// go through two 32-plane halves); 2D blocks hold their transposed words
// (16 per 32 bits of value); 1D blocks keep their planes in registers (none).
template <int D, typename T>
__host__ __device__ constexpr int store_slots() {
  return D == 1 ? 0 : D == 2 ? 16 * (int)(sizeof(T) / 4) : 32;
}
template <int D, typename T>
__host__ __device__ constexpr int decode_slots() {
  return D == 3 ? 32 : store_slots<D, T>();
}

// Blocks a warp codes, one per lane.  A field of few blocks leaves most of the
// chip idle, and a warp whose lanes diverge takes longer than its slowest
// lane; so such a field's blocks are dealt to more warps, as long as no
// scheduler (4 on each of 152 SMs) gets more than one.  3D f32 64^3, rate 16:
// compress 15.7 -> 14.0 us, decompress 12.3 -> 10.2; 3D f64 40^3, rate 8, 15.2
// -> 13.7 / 15.3 -> 14.4; with up to two warps per scheduler 96^3 floats lose
// (16.4 -> 16.7, 12.3 -> 13.0), with up to four a third.  A CTA's blocks must
// end on a word boundary of the stream (run_bits: the block size where its
// words are staged as a run, else 0).
inline uint32_t blocks_per_warp(uint64_t nblocks, uint32_t run_bits) {
  uint32_t bpw = 32;
  while (bpw > 1 && nblocks <= 608ull * (bpw / 2) &&
         (kThreads / 32 * (bpw / 2) * run_bits) % 64 == 0)
    bpw /= 2;
  return bpw;
}
// Let kernel k have `sm` bytes of dynamic shared memory; up to 47 KB need no
// leave (48 KB with a kernel's static memory).
template <class K>
cudaError_t allow_smem(K k, size_t sm) {
  if (sm <= 47 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
}
inline unsigned grid_ctas(uint64_t nblocks, uint32_t bpw) {
  const uint32_t per = kThreads / 32 * bpw;
  return (unsigned)((nblocks + per - 1) / per);
}
// the warp's first block, and the lane's (past every field for idle lanes)
__device__ __forceinline__ uint64_t warp_first_block(uint32_t bpw) {
  return ((uint64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * bpw;
}
__device__ __forceinline__ uint64_t lane_block(uint64_t first, uint32_t bpw) {
  const uint32_t lane = threadIdx.x & 31;
  return lane < bpw ? first + lane : ~0ull;
}

// NW: words of a 1D block's code (encode_block_mode).
template <int D, typename T, int STAGE = kStageNone, int NW = code4_words<T>()>
__global__ void __launch_bounds__(kThreads, (MinBlocks<D, T>::value))
    encode_kernel(const T* __restrict__ in, Geom g, uint32_t maxbits, uint32_t bpw,
                  uint64_t* __restrict__ out, uint64_t nwords) {
  extern __shared__ __align__(16) uint64_t smem[];
  uint64_t* buf = smem + table_words<D, T, false>() + store_slots<D, T>() * kThreads;
  const Tables tables = stage_tables<D, T, false, kThreads>(smem);
  if constexpr (STAGE == kStageRun)
    for (uint32_t i = threadIdx.x; i < bpw * maxbits / 16; i += kThreads) buf[i] = 0;
  tables_ready<D, T, false, STAGE == kStageRun>();
  SmemPlanes ps{smem + table_words<D, T, false>() + threadIdx.x, tables};
  const uint64_t b0 = warp_first_block(bpw), b = lane_block(b0, bpw);
  if constexpr (STAGE == kStageRows) {
    const uint32_t W = maxbits >> 6;
    if (b < g.nblocks)
      encode_one<D, T, true>(in, g, b, maxbits, StagedWords<kStride>{buf + threadIdx.x, b * W, W}, ps);
    __syncwarp();
    if (b0 < g.nblocks) {
      const uint64_t left = g.nblocks - b0;
      warp_copy<true>(buf + (threadIdx.x & ~31u), out + b0 * W, W, left < bpw ? (uint32_t)left : bpw);
    }
  } else if constexpr (STAGE == kStageRun) {
    const uint64_t w0 = (uint64_t)blockIdx.x * (bpw * maxbits / 16);
    if (b < g.nblocks) encode_one<D, T, false, NW>(in, g, b, maxbits, RunWords{buf, w0}, ps);
    __syncthreads();
    const uint64_t left = nwords - w0;
    const uint32_t run = bpw * maxbits / 16, n = left < run ? (uint32_t)left : run;
    for (uint32_t i = threadIdx.x; i < n; i += kThreads) out[w0 + i] = buf[i];
  } else {
    if (b < g.nblocks)
      encode_one<D, T>(in, g, b, maxbits, DevWords{out, nullptr, nwords}, ps);
  }
}

// MINB: resident CTAs per SM the register budget is sized for.  The decoder
// is latency-bound on its plane chain, so a fourth CTA is worth a tighter
// register budget whenever shared memory allows one (dec_min_blocks).
template <int D, typename T, int STAGE, int MINB, int NW = code4_words<T>()>
__global__ void __launch_bounds__(kThreads, MINB)
    decode_kernel(const uint64_t* __restrict__ in, uint64_t nwords, Geom g, uint32_t maxbits,
                  uint32_t bpw, T* __restrict__ out) {
  extern __shared__ __align__(16) uint64_t smem[];
  uint64_t* buf = smem + table_words<D, T, true>() + decode_slots<D, T>() * kThreads;
  const uint64_t w0 = (uint64_t)blockIdx.x * (bpw * maxbits / 16);
  const bool use = D != 3 || groups_by_table<T>(FixedRate{maxbits});
  const Tables tables = stage_tables<D, T, true, kThreads>(smem, use);
  if constexpr (STAGE == kStageRun) {
    const uint64_t left = nwords - w0;
    for (uint32_t i = threadIdx.x; i < bpw * maxbits / 16 + kPadRows; i += kThreads)
      buf[i] = i < left ? __ldg(in + w0 + i) : 0;
  }
  SmemPlanes ps{smem + table_words<D, T, true>() + threadIdx.x, tables};
  const uint64_t b0 = warp_first_block(bpw), b = lane_block(b0, bpw);
  if constexpr (STAGE == kStageRows) {
    const uint32_t W = maxbits >> 6;
    if (b0 < g.nblocks) {
      const uint64_t left = g.nblocks - b0;
      warp_copy<false>(buf + (threadIdx.x & ~31u), (uint64_t*)in + b0 * W, W,
                       left < bpw ? (uint32_t)left : bpw);
    }
#pragma unroll
    for (uint32_t j = 0; j < kPadRows; j++) buf[(W + j) * kStride + threadIdx.x] = 0;
    __syncwarp();
    tables_ready<D, T, true>(use);
    if (b < g.nblocks)
      decode_one<D, T>(out, g, b, maxbits, StagedWords<kStride>{buf + threadIdx.x, b * W, W}, ps);
  } else if constexpr (STAGE == kStageRun) {
    tables_ready<D, T, true, true>(use);
    if (b < g.nblocks)
      decode_one<D, T, NW>(out, g, b, maxbits, StagedWords<1>{buf, w0, bpw * maxbits / 16}, ps);
  } else {
    tables_ready<D, T, true>(use);
    if (b < g.nblocks) decode_one<D, T>(out, g, b, maxbits, StreamWords<D>{in, nwords}, ps);
  }
}

// Kernel launchers shared by the per-type translation units.  The encoder
// stages blocks of up to kMaxStagedOut words when their buffer fits beside
// the plane store without costing a resident CTA (larger blocks measured
// faster with direct stores).
template <int D, typename T>
cudaError_t launch_encode_t(const T* in, const Geom& g, uint32_t maxbits, uint64_t* out,
                            uint64_t nwords, cudaStream_t s) {
  if (g.nblocks == 0) return cudaSuccess;
  constexpr int MB = MinBlocks<D, T>::value;
  int stage = D == 1 || maxbits % 64 ? kStageRun : kStageRows;
  if (g.base != 0 || maxbits > 64 * kMaxStagedOut ||
      (smem_bytes(store_slots<D, T>(), stage, maxbits, table_words<D, T, false>()) + 1024) * MB > 227 * 1024)
    stage = kStageNone;
  const size_t sm = smem_bytes(store_slots<D, T>(), stage, maxbits, table_words<D, T, false>());
  auto k = stage == kStageRun ? encode_kernel<D, T, kStageRun> : encode_kernel<D, T, kStageNone>;
  if constexpr (D == 1) {  // no more words of code than the budget
    if (stage == kStageRun && maxbits <= 128)
      k = maxbits <= kShort1D<T> ? encode_kernel<D, T, kStageRun, 0>
          : maxbits <= 64        ? encode_kernel<D, T, kStageRun, 1>
                                 : encode_kernel<D, T, kStageRun, 2>;
  } else if (stage == kStageRows) {
    k = encode_kernel<D, T, kStageRows>;
  }
  cudaError_t e = allow_smem(k, sm);
  if (e != cudaSuccess) return e;
  // blocks that share words in place: into a zeroed stream (with a header,
  // the caller has zeroed it and written the header)
  if (stage == kStageNone && g.base == 0 && maxbits % 64 &&
      (e = cudaMemsetAsync(out, 0, (size_t)nwords * 8, s)) != cudaSuccess)
    return e;
  const uint32_t bpw = blocks_per_warp(g.nblocks, stage == kStageRun ? maxbits : 0);
  k<<<grid_ctas(g.nblocks, bpw), kThreads, sm, s>>>(in, g, maxbits, bpw, out, nwords);
  return cudaGetLastError();
}

// Shared memory of a staged decode CTA that still lets 4 CTAs share an SM
// (228 KB per SM, 1 KB reserved per CTA).
constexpr size_t kSmemFor4 = 56 * 1024;

template <int D, typename T>
cudaError_t launch_decode_t(const uint64_t* in, uint64_t nwords, const Geom& g, uint32_t maxbits,
                            T* out, cudaStream_t s) {
  if (g.nblocks == 0) return cudaSuccess;
  constexpr int MB = MinBlocks<D, T>::value;
  int stage = kStageNone;
  if (g.base == 0 && maxbits % 64 == 0 && (maxbits >> 6) <= kMaxStagedWords) stage = kStageRows;
  // A run's buffer must not cost a resident CTA; of 4^3 blocks of 32-bit values
  // it may cost the fourth, as the group decoder looks into the stream twice a
  // step (noisy floats 300x301x299 at rates 20.3, 26.93, 31.82: 149, 168, 169
  // us from device memory, 118, 130, 152 staged; int32 144, 154, 152 and 117,
  // 125, 148).
  constexpr int RB = D == 3 && sizeof(T) == 4 ? 3 : MB;
  if (g.base == 0 && (maxbits % 64 != 0 || (D == 1 && maxbits <= 128)) &&
      (smem_bytes(decode_slots<D, T>(), kStageRun, maxbits, table_words<D, T, true>()) + 1024) * RB <=
          227 * 1024)
    stage = kStageRun;
  const size_t sm = smem_bytes(decode_slots<D, T>(), stage, maxbits, table_words<D, T, true>());
  auto k = stage == kStageNone   ? decode_kernel<D, T, kStageNone, MB>
           : stage == kStageRows ? decode_kernel<D, T, kStageRows, MB>
                                 : decode_kernel<D, T, kStageRun, MB>;
  if constexpr (MB < 4) {
    if (sm <= kSmemFor4 && stage != kStageNone)
      k = stage == kStageRows ? decode_kernel<D, T, kStageRows, 4> : decode_kernel<D, T, kStageRun, 4>;
  }
  if constexpr (D == 1) {
    if (stage == kStageRun && maxbits <= 128)
      k = maxbits <= 64 ? decode_kernel<D, T, kStageRun, MB, 1> : decode_kernel<D, T, kStageRun, MB, 2>;
  }
  cudaError_t e = allow_smem(k, sm);
  if (e != cudaSuccess) return e;
  const uint32_t bpw = blocks_per_warp(g.nblocks, stage == kStageRun ? maxbits : 0);
  k<<<grid_ctas(g.nblocks, bpw), kThreads, sm, s>>>(in, nwords, g, maxbits, bpw, out);
  return cudaGetLastError();
}

}  // namespace gzfp
