// gzfp_batch.cu -- host side of the batched path (include/gzfp.h, "batch").
//
// Builds the device work list of a batch (array descriptors and the
// chunk -> array table), launches the per-kind kernels, captures the whole
// batch in a CUDA graph ("plans") and tunes the launch shape.
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "gzfp.h"
#include "gzfp_batch_host.h"

namespace gzfp {

// Fill chunk_item[first_chunk .. first_chunk + chunks) of every array.
__global__ void batch_chunk_table(const BatchDesc* __restrict__ descs, int count,
                                  uint32_t* chunk_item, uint64_t nchunks) {
  const int i = blockIdx.y;
  if (i >= count) return;
  const uint64_t lo = descs[i].first_chunk;
  const uint64_t hi = i + 1 < count ? descs[i + 1].first_chunk : nchunks;
  for (uint64_t cidx = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; cidx < hi;
       cidx += (uint64_t)gridDim.x * blockDim.x)
    chunk_item[cidx] = (uint32_t)i;
}

}  // namespace gzfp

namespace {

thread_local char g_batch_error[256];

int bfail(int status, const char* msg) {
  snprintf(g_batch_error, sizeof g_batch_error, "%s", msg);
  return status;
}
int bcuda(cudaError_t e, const char* what) {
  snprintf(g_batch_error, sizeof g_batch_error, "%s: %s", what, cudaGetErrorString(e));
  return GZFP_ERR_CUDA;
}

constexpr int kMaxBatchItems = 65535;
constexpr int kMaxCtasPerSm = 16;  // the largest gzfp_batch_config::ctas_per_sm

}  // namespace

namespace gzfp {
namespace bhost {

bool valid_config(const gzfp_batch_config& c) {
  return (c.threads == 64 || c.threads == 128 || c.threads == 256) && c.ctas_per_sm >= 0 &&
         c.ctas_per_sm <= kMaxCtasPerSm && (c.blocks_per_thread == 1 || c.blocks_per_thread == 2 ||
                                 c.blocks_per_thread == 4);
}

// kind index of an item (its type and shape already validated)
static int item_kind(const gzfp_batch_item& it) {
  const int dims = it.nz ? 3 : it.ny ? 2 : 1;
  return batch_kind_index(batch_kind(it.type, dims));
}

int layout(const gzfp_batch_item* items, int count, bool decode, uint64_t chunk_blocks,
           BatchDesc* descs, Layout& L) {
  L = Layout{};
  for (int i = 0; i < count; i++) {
    const gzfp_batch_item& it = items[i];
    if (!batch_type_ok(it.type)) return bfail(GZFP_ERR_UNSUPPORTED, "unknown scalar type");
    if (it.nx == 0 || (it.nz != 0 && it.ny == 0)) return bfail(GZFP_ERR_ARG, "bad dimensions");
    if (!it.field || !it.stream) return bfail(GZFP_ERR_ARG, "null pointer");
    if (it.maxbits < batch_ebits(it.type) + 1 || it.maxbits > (1u << 20))
      return bfail(GZFP_ERR_ARG, "bits per block out of range");
    const Geom g = make_geom_blocks(it.nx, it.ny ? it.ny : 1, it.nz ? it.nz : 1);
    if (g.nblocks >= (1ull << 32)) return bfail(GZFP_ERR_ARG, "too many blocks");
    const uint64_t nwords = (g.nblocks * it.maxbits + 63) / 64;
    if (it.stream_capacity < nwords * 8)
      return bfail(decode ? GZFP_ERR_ARG : GZFP_ERR_CAPACITY, "stream buffer too small");
  }
  // descriptors grouped by kind, so each kind's chunks form one range, and
  // within a kind the staged items first
  int slot = 0;
  for (int k = 0; k < kBatchKinds; k++) {
    L.lo[k] = L.nchunks;
    for (int pass = 0; pass < 2; pass++) {
      if (pass == 1) L.mid[k] = L.nchunks;
      for (int i = 0; i < count; i++) {
        const gzfp_batch_item& it = items[i];
        if (item_kind(it) != k) continue;
        if ((batch_item_staged_w(decode, it.maxbits) != 0) != (pass == 0)) continue;
        BatchDesc& d = descs[slot++];
        d.g = make_geom_blocks(it.nx, it.ny ? it.ny : 1, it.nz ? it.nz : 1);
        d.g.vec =
            ((it.nx % 4 == 0 || !it.ny) && (uintptr_t)it.field % batch_row_align(it.type) == 0) ? 1u : 0u;
        d.nwords = (d.g.nblocks * it.maxbits + 63) / 64;
        d.maxbits = it.maxbits;
        d.kind = kBatchKind[k];
        d.in = decode ? it.stream : it.field;
        d.out = decode ? it.field : it.stream;
        d.first_chunk = L.nchunks;
        L.nchunks += (d.g.nblocks + chunk_blocks - 1) / chunk_blocks;
        L.staged_w = std::max(L.staged_w, batch_item_staged_w(decode, it.maxbits));
      }
    }
    L.hi[k] = L.nchunks;
  }
  return GZFP_OK;
}

int prepare(const gzfp_batch_item* items, int count, bool decode, const gzfp_batch_config& cfg,
            Prepared& p) {
  if (!items || count < 0 || count > kMaxBatchItems) return bfail(GZFP_ERR_ARG, "bad item list");
  p.descs.resize(count);
  p.zero.clear();
  const int st = layout(items, count, decode, (uint64_t)cfg.threads * cfg.blocks_per_thread,
                        p.descs.data(), p.lay);
  if (st) return st;
  // streams whose blocks share edge words are zeroed before an encode
  if (!decode)
    for (const BatchDesc& d : p.descs)
      if (d.maxbits % 64) p.zero.push_back({d.out, (size_t)(d.nwords * 8)});
  return GZFP_OK;
}

cudaError_t WorkList::reserve(size_t ndesc, size_t nchunks) {
  cudaError_t e = cudaSuccess;
  if (!counter && (e = cudaMalloc(&counter, kBatchKinds * sizeof(unsigned long long)))) return e;
  if (!done && (e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming))) return e;
  if (!fork && (e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming))) return e;
  for (int i = 0; i < kSides; i++) {
    if (!side[i] && (e = cudaStreamCreateWithFlags(&side[i], cudaStreamNonBlocking))) return e;
    if (!join[i] && (e = cudaEventCreateWithFlags(&join[i], cudaEventDisableTiming))) return e;
  }
  if (ndesc > desc_cap) {
    cudaFree(descs);
    cudaFreeHost(host);
    descs = nullptr;
    host = nullptr;
    desc_cap = 0;
    if ((e = cudaMalloc(&descs, ndesc * sizeof(BatchDesc)))) return e;
    if ((e = cudaMallocHost(&host, ndesc * sizeof(BatchDesc)))) return e;
    desc_cap = ndesc;
  }
  if (nchunks > chunk_cap) {
    cudaFree(chunk_item);
    chunk_item = nullptr;
    chunk_cap = 0;
    if ((e = cudaMalloc(&chunk_item, nchunks * sizeof(uint32_t)))) return e;
    chunk_cap = nchunks;
  }
  return e;
}

void WorkList::release() {
  cudaFree(descs);
  cudaFreeHost(host);
  cudaFree(chunk_item);
  cudaFree(counter);
  if (done) cudaEventDestroy(done);
  if (fork) cudaEventDestroy(fork);
  fork = nullptr;
  for (int i = 0; i < kSides; i++) {
    if (side[i]) cudaStreamDestroy(side[i]);
    if (join[i]) cudaEventDestroy(join[i]);
    side[i] = nullptr;
    join[i] = nullptr;
  }
  descs = nullptr;
  host = nullptr;
  chunk_item = nullptr;
  counter = nullptr;
  done = nullptr;
  desc_cap = chunk_cap = 0;
}

// Queue everything one batch needs on stream s: zeroing of shared-word
// streams, descriptor upload, chunk table, counter reset, per-kind kernels.
cudaError_t enqueue(const Prepared& p, WorkList& wl, bool decode, const gzfp_batch_config& cfg,
                    cudaStream_t s) {
  cudaError_t e;
  const int count = (int)p.descs.size();
  if (count == 0 || p.lay.nchunks == 0) return wl.done ? cudaEventRecord(wl.done, s) : cudaSuccess;
  for (const auto& z : p.zero)
    if ((e = cudaMemsetAsync(z.first, 0, z.second, s))) return e;
  if ((e = cudaMemcpyAsync(wl.descs, wl.host, count * sizeof(BatchDesc),
                           cudaMemcpyHostToDevice, s)))
    return e;
  const dim3 tgrid(64, (unsigned)count);
  batch_chunk_table<<<tgrid, 256, 0, s>>>(wl.descs, count, wl.chunk_item, p.lay.nchunks);
  if ((e = cudaGetLastError())) return e;
  if ((e = cudaMemsetAsync(wl.counter, 0, kBatchKinds * sizeof(unsigned long long), s))) return e;
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev))) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))) return e;
  const uint32_t sw = p.lay.staged_w;
  const bool ahead = cfg.claim_ahead != 0;
  if (cfg.ctas_per_sm == 0) {
    // the grid kernels, two per kind (staged items, the others), largest first
    // and over up to four streams: most are about a wave of CTAs, and one after
    // another each would end in a tail that leaves the chip half idle (96 mixed
    // 3D arrays of 17 to 129 values an edge, compressed and decompressed: 354 ->
    // 307 us)
    struct Part {
      uint64_t lo, hi;
      int kind;
      uint32_t sw;
    };
    Part part[2 * kBatchKinds];
    int n = 0;
    for (int k = 0; k < kBatchKinds; k++) {
      if (p.lay.mid[k] > p.lay.lo[k]) part[n++] = Part{p.lay.lo[k], p.lay.mid[k], k, sw};
      if (p.lay.hi[k] > p.lay.mid[k]) part[n++] = Part{p.lay.mid[k], p.lay.hi[k], k, 0};
    }
    std::sort(part, part + n, [](const Part& a, const Part& b) { return a.hi - a.lo > b.hi - b.lo; });
    const int sides = std::min(n - 1, WorkList::kSides);
    if (sides > 0 && (e = cudaEventRecord(wl.fork, s))) return e;
    int open = 0;  // side streams that wait for the fork, so must be joined
    for (; open < sides && !e; open++)
      if ((e = cudaStreamWaitEvent(wl.side[open], wl.fork, 0))) break;
    for (int i = 0; i < n && !e; i++) {
      const int at = i % (sides + 1);
      e = launch_batch(cfg.threads, decode, part[i].kind, 0, cfg.blocks_per_thread, false,
                       part[i].sw, wl.descs, wl.chunk_item, part[i].lo, part[i].hi,
                       wl.counter + part[i].kind, at ? wl.side[at - 1] : s);
    }
    for (int i = 0; i < open; i++) {
      cudaError_t ej = cudaEventRecord(wl.join[i], wl.side[i]);
      if (!ej) ej = cudaStreamWaitEvent(s, wl.join[i], 0);
      if (!e) e = ej;
    }
  } else {
    // per kind present, in sequence on the stream, one persistent kernel
    for (int k = 0; k < kBatchKinds && !e; k++) {
      if (p.lay.hi[k] == p.lay.lo[k]) continue;
      const int grid =
          sms * std::min(cfg.ctas_per_sm, std::max(1, batch_occupancy(cfg.threads, decode, k, sw)));
      e = launch_batch(cfg.threads, decode, k, grid, cfg.blocks_per_thread, ahead, sw, wl.descs,
                       wl.chunk_item, p.lay.lo[k], p.lay.hi[k], wl.counter + k, s);
    }
  }
  if (e) return e;
  return wl.done ? cudaEventRecord(wl.done, s) : cudaSuccess;
}

}  // namespace bhost
}  // namespace gzfp

namespace {

using gzfp::bhost::Prepared;
using gzfp::bhost::valid_config;
using gzfp::bhost::WorkList;

// The work lists of one device: batches take them in turn, so that a batch is
// described and queued while the previous ones still run, and waits only for
// the one that last used its list.  (One list for all held the host up until
// the previous batch had finished on the device.)
constexpr int kWorkLists = 4;
struct DeviceWork {
  std::mutex mu;
  WorkList wl[kWorkLists];
  int next = 0;
};
constexpr int kMaxDevices = 64;
DeviceWork g_work[kMaxDevices];

int run_batch(const gzfp_batch_item* items, int count, const gzfp_batch_config* cfg_in,
              void* cuda_stream, bool decode) {
  g_batch_error[0] = 0;
  gzfp_batch_config cfg;
  gzfp_batch_default_config(&cfg);
  if (cfg_in) cfg = *cfg_in;
  if (!valid_config(cfg)) return bfail(GZFP_ERR_ARG, "bad batch configuration");
  Prepared p;
  int st = prepare(items, count, decode, cfg, p);
  if (st) return st;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e) return bcuda(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return bfail(GZFP_ERR_CUDA, "device index out of range");
  cudaStream_t s = (cudaStream_t)cuda_stream;
  DeviceWork& dw = g_work[dev];
  std::lock_guard<std::mutex> lock(dw.mu);
  WorkList& wl = dw.wl[dw.next];
  dw.next = (dw.next + 1) % kWorkLists;
  // wait until the batch that last used this list, on whatever stream it
  // ran, has finished with it
  if (wl.done && (e = cudaEventSynchronize(wl.done)))
    return bcuda(e, "cudaEventSynchronize(previous batch)");
  if ((e = wl.reserve(p.descs.size(), p.lay.nchunks))) return bcuda(e, "batch work list allocation");
  memcpy(wl.host, p.descs.data(), p.descs.size() * sizeof(gzfp::BatchDesc));
  if ((e = enqueue(p, wl, decode, cfg, s))) return bcuda(e, "batch launch");
  return GZFP_OK;
}

}  // namespace

void gzfp::batch_set_error(const char* msg) {
  snprintf(g_batch_error, sizeof g_batch_error, "%s", msg);
}

struct gzfp_batch_plan {
  WorkList wl;
  Prepared p;
  bool decode = false;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int device = 0;
};

extern "C" {

const char* gzfp_batch_last_error(void) { return g_batch_error; }

void gzfp_batch_default_config(gzfp_batch_config* cfg) {
  if (!cfg) return;
  cfg->threads = 128;
  cfg->ctas_per_sm = 0;  // the grid kernel
  cfg->blocks_per_thread = 1;
  cfg->claim_ahead = 1;
}

int gzfp_batch_compress(const gzfp_batch_item* items, int count, const gzfp_batch_config* cfg,
                        void* cuda_stream) {
  return run_batch(items, count, cfg, cuda_stream, false);
}

int gzfp_batch_decompress(const gzfp_batch_item* items, int count, const gzfp_batch_config* cfg,
                          void* cuda_stream) {
  return run_batch(items, count, cfg, cuda_stream, true);
}

int gzfp_batch_plan_create(const gzfp_batch_item* items, int count, int decompress,
                           const gzfp_batch_config* cfg_in, gzfp_batch_plan** out) {
  g_batch_error[0] = 0;
  if (!out) return bfail(GZFP_ERR_ARG, "null plan pointer");
  *out = nullptr;
  gzfp_batch_config cfg;
  gzfp_batch_default_config(&cfg);
  if (cfg_in) cfg = *cfg_in;
  if (!valid_config(cfg)) return bfail(GZFP_ERR_ARG, "bad batch configuration");
  gzfp_batch_plan* plan = new gzfp_batch_plan();
  plan->decode = decompress != 0;
  int st = prepare(items, count, plan->decode, cfg, plan->p);
  cudaError_t e = cudaSuccess;
  cudaStream_t s = nullptr;
  if (!st && (e = cudaGetDevice(&plan->device))) st = bcuda(e, "cudaGetDevice");
  if (!st && (e = plan->wl.reserve(plan->p.descs.size(), plan->p.lay.nchunks)))
    st = bcuda(e, "plan work list allocation");
  if (!st) memcpy(plan->wl.host, plan->p.descs.data(), plan->p.descs.size() * sizeof(gzfp::BatchDesc));
  if (!st && (e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking))) st = bcuda(e, "cudaStreamCreate");
  if (!st && (e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)))
    st = bcuda(e, "cudaStreamBeginCapture");
  if (!st) {
    cudaError_t el = enqueue(plan->p, plan->wl, plan->decode, cfg, s);
    cudaError_t ec = cudaStreamEndCapture(s, &plan->graph);
    if (el) st = bcuda(el, "plan capture");
    else if (ec) st = bcuda(ec, "cudaStreamEndCapture");
  }
  if (!st && (e = cudaGraphInstantiate(&plan->exec, plan->graph, 0)))
    st = bcuda(e, "cudaGraphInstantiate");
  if (s) cudaStreamDestroy(s);
  if (st) {
    gzfp_batch_plan_destroy(plan);
    return st;
  }
  *out = plan;
  return GZFP_OK;
}

int gzfp_batch_plan_launch(gzfp_batch_plan* plan, void* cuda_stream) {
  g_batch_error[0] = 0;
  if (!plan || !plan->exec) return bfail(GZFP_ERR_ARG, "null plan");
  cudaError_t e = cudaGraphLaunch(plan->exec, (cudaStream_t)cuda_stream);
  return e ? bcuda(e, "cudaGraphLaunch") : GZFP_OK;
}

void gzfp_batch_plan_destroy(gzfp_batch_plan* plan) {
  if (!plan) return;
  if (plan->exec) cudaGraphExecDestroy(plan->exec);
  if (plan->graph) cudaGraphDestroy(plan->graph);
  plan->wl.release();
  delete plan;
}

int gzfp_batch_autotune(const gzfp_batch_item* items, int count, int decompress, int repeats,
                        gzfp_batch_config* best, float* best_ms, void* cuda_stream) {
  g_batch_error[0] = 0;
  if (!best) return bfail(GZFP_ERR_ARG, "null result pointer");
  if (repeats < 1) repeats = 1;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  cudaEvent_t a = nullptr, b = nullptr;
  cudaError_t e;
  if ((e = cudaEventCreate(&a)) || (e = cudaEventCreate(&b))) return bcuda(e, "cudaEventCreate");
  float top = -1;
  int st = GZFP_OK;
  const int threads[] = {64, 128, 256};
  const int bpts[] = {1, 2, 4};
  uint32_t sw = 0;  // the staging depth the kernels will use for this batch
  if (items)
    for (int i = 0; i < count; i++)
      sw = std::max(sw, gzfp::batch_item_staged_w(decompress != 0, items[i].maxbits));
  // the kinds present: their occupancy bounds the CTAs per SM worth trying
  bool present[gzfp::kBatchKinds] = {};
  if (items)
    for (int i = 0; i < count; i++)
      if (gzfp::batch_type_ok(items[i].type)) {
        const int dims = items[i].nz ? 3 : items[i].ny ? 2 : 1;
        present[gzfp::batch_kind_index(gzfp::batch_kind(items[i].type, dims))] = true;
      }
  // every candidate is timed as it is meant to run: a graph replay
  for (int nt : threads) {
    int occ = 1;
    for (int k = 0; k < gzfp::kBatchKinds; k++)
      if (present[k]) occ = std::max(occ, gzfp::batch_occupancy(nt, decompress != 0, k, sw));
    occ = std::min(occ, kMaxCtasPerSm);
    // per_sm 0: the grid kernel (no claims, so no claim-ahead either)
    for (int per_sm = 0; per_sm <= occ && !st; per_sm++) {
      for (int bpt : bpts) {
        for (int ahead = 0; ahead < (per_sm ? 2 : 1) && !st; ahead++) {
          const gzfp_batch_config cfg{nt, per_sm, bpt, ahead};
          gzfp_batch_plan* plan = nullptr;
          st = gzfp_batch_plan_create(items, count, decompress, &cfg, &plan);
          if (!st) st = gzfp_batch_plan_launch(plan, s);  // untimed
          if (!st && (e = cudaEventRecord(a, s))) st = bcuda(e, "cudaEventRecord");
          for (int r = 0; r < repeats && !st; r++) st = gzfp_batch_plan_launch(plan, s);
          if (!st && ((e = cudaEventRecord(b, s)) || (e = cudaEventSynchronize(b))))
            st = bcuda(e, "timing");
          float ms = 0;
          if (!st) cudaEventElapsedTime(&ms, a, b);
          gzfp_batch_plan_destroy(plan);
          if (st) break;
          ms /= repeats;
          if (top < 0 || ms < top) {
            top = ms;
            *best = cfg;
          }
        }
      }
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (!st && best_ms) *best_ms = top;
  return st;
}

}  // extern "C"
