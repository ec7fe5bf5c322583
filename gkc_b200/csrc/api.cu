// C ABI: contexts, device workspaces, and the partition / count pipelines.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/gkc/gkc.h"
#include "common.cuh"
#include "ctx.h"
#include "kernels.h"

using namespace gkc;

// ------------------------------------------------------------------ helpers

const char *gkc_status_string(gkc_status s) {
  switch (s) {
    case GKC_OK: return "ok";
    case GKC_ERR_INVALID_ARG: return "invalid argument";
    case GKC_ERR_CUDA: return "CUDA error";
    case GKC_ERR_NO_DEVICE: return "no CUDA device";
    case GKC_ERR_OUT_OF_MEMORY: return "out of device memory";
    case GKC_ERR_BUDGET: return "HBM budget exceeded";
    case GKC_ERR_CAPACITY: return "capacity exceeded";
    case GKC_ERR_DEVICE_TIMEOUT: return "device-side wait timed out";
    case GKC_ERR_NOT_READY: return "not ready";
    case GKC_ERR_CANCELLED: return "cancelled";
    case GKC_ERR_NOT_FOUND: return "not found";
    default: return "internal error";
  }
}

int gkc_abi_version(void) { return GKC_ABI_VERSION; }

// Stages of the batched pipeline.
static const char *kStageNames[] = {"prepare", "partition", "bin_scatter", "coarse_hist",
                                    "coarse_scatter", "coarse_count", "finish"};
constexpr int kNumStages = 7;
const char *gkc_stage_name(int i) { return (i >= 0 && i < kNumStages) ? kStageNames[i] : ""; }

// The first kernel of each stage writes the device's clock to its place (an
// event between two kernels of a captured pipeline is a node of the graph that
// the next one waits for: a job of 100 k bases takes 163 us, with eight of
// them 217).
static void read_stage_times(gkc_ctx *c) {
  c->tm.n_stages = kNumStages;
  for (int i = 0; i < kNumStages; i++)
    c->tm.stage_ms[i] = (float)((double)(int64_t)(c->h_tot->stamp[i + 1] - c->h_tot->stamp[i]) * 1e-6);
}

gkc_status ctx_fail(gkc_ctx *c, gkc_status s, const std::string &msg) {
  if (c) c->err = msg;
  return s;
}

gkc_status ctx_cuda(gkc_ctx *c, cudaError_t e, const char *what) {
  if (e == cudaSuccess) return GKC_OK;
  cudaGetLastError();
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  return ctx_fail(c, e == cudaErrorMemoryAllocation ? GKC_ERR_OUT_OF_MEMORY : GKC_ERR_CUDA, m);
}

#define CK(call)                                                  \
  do {                                                            \
    gkc_status _s = ctx_cuda(c, (call), #call);                   \
    if (_s != GKC_OK) return _s;                                  \
  } while (0)
#define LAUNCHED(c)                                               \
  do {                                                            \
    (c)->launches++;                                              \
    cudaError_t _e = cudaPeekAtLastError();                       \
    if (_e != cudaSuccess) return ctx_cuda((c), _e, "kernel launch"); \
  } while (0)

// Workspaces come from one stream-ordered memory pool per device, owned by
// the library: allocations and frees are ordered on the context's stream and
// do not synchronise the device, and freed blocks stay cached in the pool for
// the next request (from any context) until a context is destroyed or its
// workspace released through the public call, which trims the pool.
static std::mutex g_pool_mu;
static cudaMemPool_t g_pool[64];

static cudaMemPool_t device_pool(int dev, cudaError_t *err) {
  *err = cudaSuccess;
  if (dev < 0 || dev >= 64) {
    *err = cudaErrorInvalidDevice;
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props;
    memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool;
    *err = cudaMemPoolCreate(&pool, &props);
    if (*err != cudaSuccess) return nullptr;
    uint64_t keep = ~0ull;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    g_pool[dev] = pool;
  }
  return g_pool[dev];
}

static void trim_pool(int dev) {
  cudaError_t e;
  cudaMemPool_t pool = device_pool(dev, &e);
  if (pool) cudaMemPoolTrimTo(pool, 0);
}

// A buffer from the device pool outside any context (ordered on st).
cudaError_t result_alloc(int dev, void **p, size_t bytes, cudaStream_t st) {
  cudaError_t e;
  cudaMemPool_t pool = device_pool(dev, &e);
  if (!pool) return e;
  return cudaMallocFromPoolAsync(p, bytes, pool, st);
}

void *ws_get(gkc_ctx *c, const char *name, size_t bytes, gkc_status *st) {
  *st = GKC_OK;
  if (bytes == 0) bytes = 16;
  bytes = (bytes + 255) & ~(size_t)255;
  auto it = c->bufs.find(name);
  if (it != c->bufs.end() && it->second.bytes >= bytes) return it->second.p;
  if (c->capturing) {  // the capture pass repeats the sizing pass: nothing may grow
    *st = ctx_fail(c, GKC_ERR_INTERNAL, std::string("workspace '") + name + "' grew during capture");
    return nullptr;
  }
  size_t old = 0;
  if (it != c->bufs.end()) {
    old = it->second.bytes;
    cudaFreeAsync(it->second.p, c->st);
    c->used -= old;
    c->bufs.erase(it);
    graphs_invalidate(c);
  }
  size_t want = std::max(bytes, old + old / 4);
  if (c->budget && c->used + want > c->budget) want = bytes;
  if (c->budget && c->used + want > c->budget) {
    *st = ctx_fail(c, GKC_ERR_BUDGET, std::string("workspace '") + name + "' needs " +
                                          std::to_string(bytes) + " bytes beyond the HBM budget");
    return nullptr;
  }
  cudaError_t e;
  cudaMemPool_t pool = device_pool(c->dev, &e);
  void *p = nullptr;
  if (pool) e = cudaMallocFromPoolAsync(&p, want, pool, c->st);
  if (e != cudaSuccess) {
    *st = ctx_cuda(c, e, (std::string("allocating ") + name).c_str());
    return nullptr;
  }
  c->used += want;
  c->bufs[name] = DevBuf{p, want};
  if (old) graphs_invalidate(c);  // captured graphs may hold the freed buffer; a new one is in none
  return p;
}

// Frees every workspace of c into the pool (ordered on c's stream).
void ws_release_all(gkc_ctx *c) {
  cudaStreamSynchronize(c->st);
  for (auto &g : c->graphs)
    if (g.exec) {
      cudaGraphExecDestroy(g.exec);
      g.exec = nullptr;
    }
  for (auto &kv : c->bufs) cudaFreeAsync(kv.second.p, c->st);
  cudaStreamSynchronize(c->st);
  c->bufs.clear();
  c->used = 0;
  graphs_invalidate(c);
  c->have_part = c->have_count = false;
}

#define WS(ptr, type, name, count)                                      \
  type *ptr;                                                            \
  do {                                                                  \
    gkc_status _s;                                                      \
    ptr = (type *)ws_get(c, name, sizeof(type) * (size_t)(count), &_s); \
    if (_s != GKC_OK) return _s;                                        \
  } while (0)

// ------------------------------------------------------------------ context

static cudaError_t set_dyn_smem_limit(const void *f, int optin) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, f);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
}

gkc_status gkc_ctx_create(int device_id, uint64_t hbm_budget_bytes, gkc_ctx **out) {
  if (!out) return GKC_ERR_INVALID_ARG;
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    return GKC_ERR_NO_DEVICE;
  }
  if (device_id < 0 || device_id >= n) return GKC_ERR_INVALID_ARG;
  gkc_ctx *c = new gkc_ctx();
  c->dev = device_id;
  c->budget = hbm_budget_bytes;
  if (cudaSetDevice(device_id) != cudaSuccess) {
    delete c;
    return GKC_ERR_CUDA;
  }
  cudaDeviceProp prop;
  cudaGetDeviceProperties(&prop, device_id);
  c->n_sms = prop.multiProcessorCount;
  c->max_smem_optin = (int)prop.sharedMemPerBlockOptin;
  // The dynamic shared-memory limit of a kernel is process-wide: set it to
  // the device maximum (less the kernel's static shared memory) once, here,
  // and never per launch, where one thread could lower it between another
  // thread's setting and launch.
  if (set_dyn_smem_limit((const void *)k_partition, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bin_place, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_sort<uint64_t, false>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_sort<uint64_t, true>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_sort<u128, false>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_open<uint64_t>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_open<u128>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_slices<uint64_t>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_slices<u128>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_scatter<uint64_t, 1>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_scatter<uint64_t, 2>, c->max_smem_optin) != cudaSuccess ||
      set_dyn_smem_limit((const void *)k_bucket_scatter<u128, 1>, c->max_smem_optin) != cudaSuccess) {

    cudaGetLastError();
    delete c;
    return GKC_ERR_CUDA;
  }
  if (cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMallocHost(&c->h_tots[0], 2 * sizeof(DevTotals)) != cudaSuccess) {
    delete c;
    return GKC_ERR_CUDA;
  }
  c->h_tots[1] = c->h_tots[0] + 1;
  c->h_tot = c->h_tots[0];
  c->own_stream = true;
  for (int i = 0; i < 4; i++) cudaEventCreate(&c->ev[i]);
  *out = c;
  return GKC_OK;
}

void gkc_ctx_destroy(gkc_ctx *c) {
  if (!c) return;
  cudaSetDevice(c->dev);
  if (c->st) cudaStreamSynchronize(c->st);
  ws_release_all(c);
  trim_pool(c->dev);
  for (int i = 0; i < 4; i++)
    if (c->ev[i]) cudaEventDestroy(c->ev[i]);
  if (c->h_tots[0]) cudaFreeHost(c->h_tots[0]);
  if (c->st_up) cudaStreamDestroy(c->st_up);
  if (c->st_dl) cudaStreamDestroy(c->st_dl);
  for (int i = 0; i < 2; i++) {
    if (c->ev_up[i]) cudaEventDestroy(c->ev_up[i]);
    if (c->ev_comp[i]) cudaEventDestroy(c->ev_comp[i]);
  }
  for (int i = 0; i < 4; i++)
    if (c->ev_dl[i]) cudaEventDestroy(c->ev_dl[i]);
  if (c->own_stream && c->st) cudaStreamDestroy(c->st);
  delete c;
}

const char *gkc_ctx_last_error(const gkc_ctx *c) { return c ? c->err.c_str() : "no context"; }

gkc_status gkc_ctx_set_filter(gkc_ctx *c, int filter) {
  if (!c) return GKC_ERR_INVALID_ARG;
  if (filter < GKC_FILTER_NEW2 || filter > GKC_FILTER_SIGNATURE)
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "unknown minimizer filter");
  if (filter != c->filter) {
    c->filter = filter;
    graphs_invalidate(c);
    c->have_part = c->have_count = false;
  }
  return GKC_OK;
}

gkc_status gkc_ctx_set_stream(gkc_ctx *c, void *stream) {
  if (!c) return GKC_ERR_INVALID_ARG;
  cudaSetDevice(c->dev);
  cudaStreamSynchronize(c->st);
  if (c->own_stream) cudaStreamDestroy(c->st);
  c->st = (cudaStream_t)stream;
  c->own_stream = false;
  graphs_invalidate(c);
  return GKC_OK;
}

gkc_status gkc_ctx_synchronize(gkc_ctx *c) {
  if (!c) return GKC_ERR_INVALID_ARG;
  CK(cudaStreamSynchronize(c->st));
  return GKC_OK;
}

uint64_t gkc_ctx_device_bytes(const gkc_ctx *c) { return c ? c->used : 0; }

gkc_status gkc_ctx_release_workspace(gkc_ctx *c) {
  if (!c) return GKC_ERR_INVALID_ARG;
  cudaSetDevice(c->dev);
  ws_release_all(c);
  trim_pool(c->dev);
  return GKC_OK;
}

gkc_status gkc_last_timings(const gkc_ctx *c, gkc_timings *out) {
  if (!c || !out) return GKC_ERR_INVALID_ARG;
  *out = c->tm;
  return GKC_OK;
}

// ------------------------------------------------------------- validation

static gkc_status check_params(gkc_ctx *c, const gkc_params *prm) {
  if (!prm) return ctx_fail(c, GKC_ERR_INVALID_ARG, "params is NULL");
  if (prm->k < 1 || prm->k > 64) return ctx_fail(c, GKC_ERR_INVALID_ARG, "k must be in [1, 64]");
  if (prm->p < 3 || prm->p > 16 || prm->p > prm->k)
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "p must be in [3, 16] and <= k");
  if (prm->nbins < 1 || prm->nbins > (1 << 20))
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "nbins must be in [1, 2^20]");
  return GKC_OK;
}

// --------------------------------------------------------------- totals

// The totals go straight to the slot's page-locked record (no copy follows).
__global__ void k_finalize(DevTotals *t, const unsigned long long *cursors, const uint32_t *err,
                           const uint64_t *bin_kstart, uint32_t nbins, const uint64_t *n_bytes_dev,
                           const uint64_t *bin_out, const unsigned long long *stamp) {
  for (int i = 0; i < kNumStages; i++) t->stamp[i] = stamp[i];
  t->n_skm = cursors[0];
  t->n_packed = cursors[1];
  t->err = *err;
  t->n_kmers = bin_kstart ? bin_kstart[nbins] : 0;
  t->n_bytes = n_bytes_dev ? *n_bytes_dev : 0;
  t->n_distinct = bin_out ? bin_out[nbins] : 0;
  stamp_now(&t->stamp[kNumStages]);
  __threadfence_system();
}

// ------------------------------------------------------------- partition

// Capacity estimates for the superkmer outputs (exact sizes are re-derived
// from the device cursors when a run overflows them).
static void partition_caps(const gkc_params *prm, uint64_t n_bytes, uint64_t n_reads,
                           uint64_t *cap_skm, uint64_t *cap_bytes) {
  const double omega = prm->k - prm->p + 1;
  uint64_t w = n_bytes;
  uint64_t s = (uint64_t)((double)w * 3.0 / (omega + 1.0)) + n_reads + 4096;
  if (s > w + 16) s = w + 16;
  uint64_t tiles = n_bytes / kPartTile + 2;
  *cap_skm = s;
  *cap_bytes = (w + s * (uint64_t)(prm->k - 1)) / 4 + s + tiles * 16 + 64;
}

// Device bytes one pipeline run over n_bases bases in n_reads reads needs: a
// bound over the workspaces that the batched pipeline sizes for it, with room
// (64 MB and more) for reads that hold more superkmers than that.  The room
// comes from terms charged above their size: two words a superkmer for one
// k-mer offset, chunks of 32 K k-mers (small inputs have smaller ones, but few),
// buckets for every digit.  It also takes what is not named here: the flags and
// prefixes of HPC, the placement matrices of small chunks, the slices of
// opened buckets.
uint64_t gkc_job_hbm_estimate(const gkc_params *prm, uint64_t n_bases, uint64_t n_reads) {
  if (!prm || prm->k < 1 || prm->k > 64 || prm->nbins < 1) return 0;
  const uint64_t B = n_bases, R = n_reads, w = prm->k <= 32 ? 8 : 16;
  uint64_t cap_skm, cap_bytes;
  partition_caps(prm, B, R, &cap_skm, &cap_bytes);
  uint64_t e = (B + 64) + 8 * (R + 1);                                  // reads, offsets
  if (prm->hpc) e += 8 * (R + 1) + 8 * (R + 2) + (B + 64) + 4 * (B + 16);  // HPC copies
  e += (B + 1) / 8 + 16;                                                 // read starts
  e += cap_skm * (8 + 4 + 8 + 4) + cap_bytes;                            // superkmers
  e += cap_skm * 16;                                                     // k-mer offsets
  if ((uint32_t)prm->nbins <= (uint32_t)kBinPlaceMaxBins)                // bin placement matrices
    e += 17 * ((cap_skm + kBinChunk - 1) / kBinChunk) * (uint64_t)prm->nbins;
  const uint64_t kc = std::max<uint64_t>(B, 16);
  uint32_t max_bits = kCoarseMaxBits;
  while (max_bits > 0 && ((uint64_t)prm->nbins << max_bits) > (1ull << 20)) max_bits--;
  const uint64_t chunks = kc / 32768 + prm->nbins + 1;
  e += 4 * (chunks << max_bits) + 8 * chunks;                            // chunk matrix, first superkmers
  e += w * kc * 2 + 4 * kc * 2;                                          // keys, output keys, staged and output counts
  e += ((uint64_t)prm->nbins << max_bits) * (8 * 5 + 4 * 2);             // bucket starts, sizes, distinct counts,
                                                                         // offsets, scan; bins, large-bucket list
  e += 8ull << 20;                                                       // tables of the buckets' digits, tasks
  e += 80 * (uint64_t)prm->nbins;                                        // counters, prefixes and offsets per bin
  return e + (64ull << 20);
}

// Enqueues HPC (optional), partition and bin scatter on c->st.
static gkc_status enqueue_partition(gkc_ctx *c, const gkc_params *prm, const char *d_reads,
                                    uint64_t n_bytes, const uint64_t *d_offs, uint64_t n_reads,
                                    uint64_t cap_skm, uint64_t cap_bytes) {
  const uint32_t nbins = (uint32_t)prm->nbins;
  const uint8_t *src = reinterpret_cast<const uint8_t *>(d_reads);
  const uint64_t *offs = d_offs;
  const uint64_t *nbytes_dev = nullptr;
  WS(tot, unsigned long long, "cursors", 4);
  WS(err, uint32_t, "err", 4);
  WS(stamp, unsigned long long, "stamps", GKC_MAX_STAGES + 1);
  c->part_hpc_reads = nullptr;
  c->part_hpc_offs = nullptr;
  c->part_hpc_orig = nullptr;
  if (prm->hpc) {
    WS(hoffs, uint64_t, "hpc_offs", n_reads + 2);
    WS(hreads, uint8_t, "hpc_reads", n_bytes + 64);
    WS(horig, int32_t, "hpc_orig", n_bytes + 16);
    const gkc_status hs = hpc_enqueue(c, src, n_bytes, offs, n_reads, hreads, hoffs, horig, stamp);
    if (hs != GKC_OK) return hs;
    src = hreads;
    offs = hoffs;
    nbytes_dev = hoffs + n_reads;
    c->part_hpc_reads = (const char *)hreads;
    c->part_hpc_offs = hoffs;
    c->part_hpc_orig = horig;
  }
  const uint64_t rs_words = (n_bytes + 1 + 31) / 32 + 2;
  WS(rs, uint32_t, "rs_bits", rs_words);  // with HPC: the original reads' bitmap until here
  WS(bin_nskm, unsigned long long, "bin_nskm", nbins + 1);
  WS(bin_nkm, unsigned long long, "bin_nkmers", nbins + 1);
  const ClearArgs ca{tot, err, bin_nskm, bin_nkm, nbins, rs, rs_words, prm->hpc ? nullptr : stamp};
  k_partition_clear<<<(unsigned)std::min<uint64_t>(rs_words / 1024 + 1, (uint64_t)c->n_sms * 8), 256, 0, c->st>>>(ca);
  LAUNCHED(c);
  k_read_start_bits<<<(unsigned)std::min<uint64_t>((n_reads + 256) / 256, 65535), 256, 0, c->st>>>(
      offs, n_reads, rs);
  LAUNCHED(c);

  WS(desc, uint64_t, "skm_desc_tile", cap_skm);
  WS(mm, uint32_t, "skm_mm_tile", cap_skm);
  WS(packed, uint8_t, "packed", cap_bytes + 16);  // k-mers are cut from whole words

  PartArgs a;
  memset(&a, 0, sizeof(a));
  a.filter = c->filter;
  a.reads = src;
  a.nbytes = n_bytes;
  a.nbytes_dev = nbytes_dev;
  a.aligned16 = ((uintptr_t)src % 16) == 0;
  a.rs_bits = rs;
  a.rs_words = rs_words;
  a.k = prm->k;
  a.p = prm->p;
  a.nbins = (int)nbins;
  a.nbins_smem = nbins <= 1024 ? (int)((nbins + 1) & ~1u) : 0;
  a.skm_desc = desc;
  a.skm_mm = mm;
  a.skm_gpos = nullptr;
  a.packed = packed;
  a.cursors = tot;
  a.cap_skm = cap_skm;
  a.cap_bytes = cap_bytes;
  a.bin_nskm = bin_nskm;
  a.bin_nkmers = bin_nkm;
  a.err = err;
  size_t smem = partition_smem_bytes(a.nbins_smem);
  if ((int)smem > c->max_smem_optin) return ctx_fail(c, GKC_ERR_INVALID_ARG, "too many bins for shared memory");
  int occ = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_partition, kPartThreads, smem));
  uint64_t tiles = (n_bytes + kPartTile - 1) / kPartTile;
  unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)c->n_sms * std::max(occ, 1)));
  a.stamp = stamp + 1;
  k_partition<<<grid, kPartThreads, smem, c->st>>>(a);
  LAUNCHED(c);

  WS(bin_start, uint64_t, "bin_start", nbins + 1);
  WS(bin_kstart, uint64_t, "bin_kstart", nbins + 1);
  k_bin_prefix<<<1, kBinPrefixThreads, 0, c->st>>>(bin_nskm, bin_nkm, nbins, bin_start, bin_kstart, stamp + 2);
  LAUNCHED(c);
  WS(bdesc, uint64_t, "skm_desc_bin", cap_skm);
  WS(bmm, uint32_t, "skm_mm_bin", cap_skm);
  if (nbins <= (uint32_t)kBinPlaceMaxBins) {
    // (bin, chunk) counts, one scan, then placement: no global atomics
    // few superkmers: chunks of one round, so that more CTAs share them
    const uint32_t chunk = cap_skm < (uint64_t)kBinChunk * c->n_sms * 2 ? kBinRound : kBinChunk;
    const uint64_t nch_cap = (cap_skm + chunk - 1) / chunk;
    const uint64_t cells = nch_cap * nbins;
    WS(bmat, unsigned long long, "bin_chunk_cnt", cells + 1);
    WS(boff, uint64_t, "bin_chunk_off", cells + 2);
    WS(btmp, uint64_t, "bin_chunk_scan", scan_u64_tmp_words(cells + 1) + 8);
    const unsigned g = (unsigned)std::min<uint64_t>(nch_cap, (uint64_t)c->n_sms * 8);
    k_bin_count<<<g, 256, nbins * 4, c->st>>>(tot, mm, nbins, chunk, nch_cap, bmat, err);
    LAUNCHED(c);
    c->launches += scan_u64(bmat, boff, cells, btmp, c->st);
    k_bin_place<<<(unsigned)std::min<uint64_t>(nch_cap, (uint64_t)c->n_sms * 2), kBinPlaceThreads,
                  bin_place_smem_bytes(nbins), c->st>>>(tot, desc, mm, nbins, chunk, nch_cap, boff, bdesc, bmm, err);
    LAUNCHED(c);
  } else {
    WS(bfill, unsigned long long, "bin_fill", nbins + 1);
    CK(cudaMemsetAsync(bfill, 0, (nbins + 1) * 8, c->st));
    k_bin_scatter<<<c->n_sms * 8, 256, 0, c->st>>>(tot, desc, mm, nbins, bin_start, bfill, bdesc,
                                                   bmm, nullptr, nullptr, err);
    LAUNCHED(c);
  }
  c->part_packed = packed;  // descriptors point into the tile-order bases

  c->part_cap_skm = cap_skm;
  c->part_cap_bytes = cap_bytes;
  c->part_nbytes_dev = nbytes_dev;
  return GKC_OK;
}

static gkc_status fill_partition_view(gkc_ctx *c, const gkc_params *prm, uint64_t n_reads,
                                      uint64_t n_bytes) {
  gkc_partition_view &v = c->pv;
  memset(&v, 0, sizeof(v));
  v.n_reads = n_reads;
  v.n_bases = prm->hpc ? c->h_tot->n_bytes : n_bytes;
  v.n_superkmers = c->h_tot->n_skm;
  v.n_packed_bytes = c->h_tot->n_packed;
  v.n_kmers = c->h_tot->n_kmers;
  v.nbins = (uint32_t)prm->nbins;
  v.bin_skm_off = (const uint64_t *)c->bufs["bin_start"].p;
  v.bin_kmer_off = (const uint64_t *)c->bufs["bin_kstart"].p;
  v.skm_desc = (const uint64_t *)c->bufs["skm_desc_bin"].p;
  v.skm_minimizer = (const uint32_t *)c->bufs["skm_mm_bin"].p;
  v.packed = c->part_packed;
  v.hpc_reads = c->part_hpc_reads;
  v.hpc_offs = c->part_hpc_offs;
  v.hpc_orig_pos = c->part_hpc_orig;
  c->pp = *prm;
  c->have_part = true;
  return GKC_OK;
}

static gkc_status read_totals(gkc_ctx *c, bool with_count, uint32_t nbins) {
  const uint64_t *bk = (const uint64_t *)c->bufs["bin_kstart"].p;
  const uint64_t *bo = with_count ? (const uint64_t *)c->bufs[slot_name(c, "bin_out")].p : nullptr;
  k_finalize<<<1, 1, 0, c->st>>>(c->h_tot, (const unsigned long long *)c->bufs["cursors"].p,
                                 (const uint32_t *)c->bufs["err"].p, bk, nbins, c->part_nbytes_dev, bo,
                                 (const unsigned long long *)c->bufs["stamps"].p);
  LAUNCHED(c);
  return GKC_OK;
}

static gkc_status device_err(gkc_ctx *c, uint32_t e) {
  if (e & ERR_BIN_TOO_LARGE)
    return ctx_fail(c, GKC_ERR_CAPACITY, "a bin holds 2^32 or more k-mers: use more bins");
  if (e & ERR_BOUNDS) return ctx_fail(c, GKC_ERR_INTERNAL, "device bounds check failed");
  if (e & ERR_SPIN_TIMEOUT) return ctx_fail(c, GKC_ERR_DEVICE_TIMEOUT, "device look-back wait timed out");
  if (e & ERR_BAD_READ) return ctx_fail(c, GKC_ERR_INVALID_ARG, "read longer than supported");
  return GKC_OK;
}
static gkc_status check_device_err(gkc_ctx *c) { return device_err(c, c->h_tot->err); }

gkc_status partition_device_impl(gkc_ctx *c, const gkc_params *prm, const char *d_reads,
                                 uint64_t n_bytes, const uint64_t *d_offs, uint64_t n_reads) {
  uint64_t cap_skm, cap_bytes;
  partition_caps(prm, n_bytes, n_reads, &cap_skm, &cap_bytes);
  for (int attempt = 0; attempt < 2; attempt++) {
    graphs_invalidate(c);
    gkc_status s = enqueue_partition(c, prm, d_reads, n_bytes, d_offs, n_reads, cap_skm, cap_bytes);
    if (s != GKC_OK) return s;
    s = read_totals(c, false, (uint32_t)prm->nbins);
    if (s != GKC_OK) return s;
    CK(cudaStreamSynchronize(c->st));
    if (!(c->h_tot->err & ERR_CAPACITY)) break;
    cap_skm = c->h_tot->n_skm + 16;
    cap_bytes = c->h_tot->n_packed + 64;
    if (attempt == 1) return ctx_fail(c, GKC_ERR_CAPACITY, "partition capacity");
  }
  gkc_status s = check_device_err(c);
  if (s != GKC_OK) return s;
  return fill_partition_view(c, prm, n_reads, n_bytes);
}

gkc_status gkc_partition_device(gkc_ctx *c, const gkc_params *prm, const char *d_reads,
                                uint64_t n_bytes, const uint64_t *d_offs, uint64_t n_reads,
                                gkc_partition_view *out) {
  if (!c) return GKC_ERR_INVALID_ARG;
  gkc_status s = check_params(c, prm);
  if (s != GKC_OK) return s;
  if (n_bytes > 0 && (!d_reads || !d_offs)) return ctx_fail(c, GKC_ERR_INVALID_ARG, "null input");
  cudaSetDevice(c->dev);
  c->launches = 0;
  CK(cudaEventRecord(c->ev[0], c->st));
  s = partition_device_impl(c, prm, d_reads, n_bytes, d_offs, n_reads);
  if (s != GKC_OK) return s;
  CK(cudaEventRecord(c->ev[1], c->st));
  CK(cudaEventSynchronize(c->ev[1]));
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
  c->tm = gkc_timings{};
  c->tm.partition_ms = ms;
  c->tm.total_ms = ms;
  c->tm.launches = c->launches;
  if (out) *out = c->pv;
  return GKC_OK;
}

// ------------------------------------------------------------------ count

// Whether a group of some 96 keys of a bin of bin_keys k-mers mostly lies
// within 2^29 consecutive values, so that no more than one in eight has keys
// that differ in the upper word: counted from the k-mers' 2 k bits, as if they
// were spread evenly (where they are not, more groups or fewer qualify; the
// kernel looks at each).
static bool narrow_groups(int k, uint64_t bin_keys) {
  int bits = 2 * k;
  for (uint64_t groups = bin_keys / 96; groups > 1; groups >>= 1) bits--;
  return bits <= 29;
}

template <typename K>
static gkc_status enqueue_count_batched(gkc_ctx *c, const gkc_params *prm, uint64_t keys_cap,
                                        uint64_t) {
  const uint32_t nbins = (uint32_t)prm->nbins;
  uint32_t max_bits = kCoarseMaxBits;
  while (max_bits > 0 && ((uint64_t)nbins << max_bits) > (1ull << 20)) max_bits--;
  const uint32_t bucket_keys = bucket_target<K>(c->tune.coarse_target ? c->tune.coarse_target : kCoarseTarget);
  // any two neighbouring buckets of a bin hold more than bucket_keys keys
  const uint64_t max_buckets =
      std::min<uint64_t>((uint64_t)nbins << max_bits, keys_cap / bucket_keys * 2 + 2 + nbins);
  const uint64_t cap_skm = std::max<uint64_t>(c->part_cap_skm, 1);
  WS(err, uint32_t, "err", 4);
  const unsigned long long *n_skm_dev = (const unsigned long long *)c->bufs["cursors"].p;
  const uint64_t *desc = (const uint64_t *)c->bufs["skm_desc_bin"].p;
  const uint64_t *bin_start = (const uint64_t *)c->bufs["bin_start"].p;
  const uint64_t *bin_kstart = (const uint64_t *)c->bufs["bin_kstart"].p;

  // k-mer offset of every bin-ordered superkmer
  WS(stamp, unsigned long long, "stamps", GKC_MAX_STAGES + 1);
  WS(koff, uint64_t, "skm_koff", cap_skm + 2);
  WS(stmp, uint64_t, "scan_tmp2", scan_u64_tmp_words(cap_skm + 1) + 8);
  c->launches += scan_kmers_dev(desc, prm->k, koff, cap_skm, (const uint64_t *)n_skm_dev, stmp, c->st, stamp + 3);

  WS(bin_bits, uint32_t, "bin_bits", nbins + 1);
  WS(bucket_base, uint64_t, "bucket_base", nbins + 1);
  WS(chunk_base, uint64_t, "chunk_base", nbins + 1);
  WS(hist_base, uint64_t, "hist_base", nbins + 1);
  CountPlan pl;
  pl.nbins = nbins;
  pl.bin_start = bin_start;
  pl.bin_kstart = bin_kstart;
  pl.bucket_keys = bucket_keys;
  pl.max_bits = max_bits;
  const uint64_t chunk_kmers = c->tune.chunk_kmers ? c->tune.chunk_kmers : default_chunk(keys_cap, c->n_sms);
  pl.chunk_kmers = chunk_kmers;
  pl.k = prm->k;
  pl.err = err;
  pl.bin_bits = bin_bits;
  pl.chunk_base = chunk_base;
  pl.hist_base = hist_base;
  // [0] bucket ticket, [2] large buckets listed, [3] their ticket, [4] slices listed, [5] their ticket,
  // [6] bins scanned
  WS(ticket, unsigned long long, "count_ticket", 8);
  pl.tickets = ticket;
  k_count_plan<<<1, kCountPlanThreads, 0, c->st>>>(pl);
  LAUNCHED(c);

  // chunks: at most keys_cap / kChunkKmers + nbins; histogram cells: chunks << max_bits
  const uint64_t max_chunks = keys_cap / chunk_kmers + nbins + 1;
  WS(chunk_s0, uint64_t, "chunk_s0", max_chunks);
  WS(hist, uint32_t, "bucket_hist", max_chunks << max_bits);
  WS(lut, uint16_t, "bucket_lut", (uint64_t)nbins << max_bits);
  WS(digit_total, uint32_t, "digit_total", (uint64_t)nbins << max_bits);
  WS(unit_start, uint32_t, "unit_start", (uint64_t)nbins << max_bits);
  WS(bin_units, uint32_t, "bin_units", nbins);
  WS(keys, K, "keys", keys_cap);
  // the result's key array holds the k-mer-order keys until the count stage is done with them
  WS(out_keys, K, slot_name(c, "out_keys").c_str(), keys_cap);
  WS(bstart, uint64_t, "bucket_start", max_buckets + 1);
  WS(bsize, uint64_t, "bucket_size", max_buckets + 1);
  ExpandArgs ea;
  memset(&ea, 0, sizeof(ea));
  ea.desc = desc;
  ea.koff = koff;
  ea.packed = c->part_packed;
  ea.nbins = nbins;
  ea.bin_start = bin_start;
  ea.bin_kstart = bin_kstart;
  ea.chunk_base = chunk_base;
  ea.hist_base = hist_base;
  ea.bucket_base = bucket_base;
  ea.bin_bits = bin_bits;
  ea.chunk_kmers = chunk_kmers;
  ea.k = prm->k;
  ea.chunk_s0 = chunk_s0;
  ea.hist = hist;
  ea.lut = lut;
  ea.digit_total = digit_total;
  ea.unit_start = unit_start;
  ea.bin_units = bin_units;
  ea.scan_done = ticket + 6;
  ea.max_bits = max_bits;
  ea.bucket_keys = bucket_keys;
  ea.keys = keys;
  ea.flat = out_keys;
  ea.keys_cap = keys_cap;
  ea.err = err;
  const uint64_t first_n = 32 * std::max<uint64_t>(max_chunks, nbins);
  k_chunk_first<<<(unsigned)std::min<uint64_t>((first_n + 255) / 256, 65535), 256, 0, c->st>>>(ea);
  LAUNCHED(c);
  k_bucket_hist<K><<<(unsigned)std::min<uint64_t>(max_chunks, (uint64_t)c->n_sms * 8), kBucketHistThreads, 0, c->st>>>(ea);
  LAUNCHED(c);
  WS(big_list, uint32_t, "big_list", max_buckets + 1);
  WS(bucket_head, uint32_t, "bucket_head", max_buckets + 1);
  ea.bucket_head = bucket_head;
  ea.big_list = big_list;
  ea.big_count = ticket + 2;
  ea.big_min = bucket_count_cap<K>() + 1;
  k_bucket_scan<<<std::min<uint32_t>(nbins, 65535), kBucketScanThreads, 0, c->st>>>(ea);
  LAUNCHED(c);
  k_bucket_offsets<<<(unsigned)std::min<uint64_t>((32 * max_buckets + kBucketOffsetThreads - 1) / kBucketOffsetThreads,
                                                  (uint64_t)c->n_sms * 64),
                     kBucketOffsetThreads, 0, c->st>>>(ea, bstart, bsize);
  LAUNCHED(c);
  ea.stamp = stamp + 4;
  const int sc_ctas = sizeof(K) == 8 && keys_cap / nbins <= kScatterPairBin ? 2 : 1;
  const size_t sct_smem = bucket_scatter_smem_bytes<K>(sc_ctas);
  if ((int)sct_smem > c->max_smem_optin) return ctx_fail(c, GKC_ERR_INTERNAL, "scatter tile exceeds shared memory");
  const unsigned sc_grid = (unsigned)std::min<uint64_t>(max_chunks, (uint64_t)c->n_sms * sc_ctas);
  if (sc_ctas == 2) k_bucket_scatter<uint64_t, 2><<<sc_grid, 512, sct_smem, c->st>>>(ea);
  else k_bucket_scatter<K, 1><<<sc_grid, 1024, sct_smem, c->st>>>(ea);
  LAUNCHED(c);

  // counting: buckets independently, each bucket's runs staged over its own
  // keys (counts beside them), then moved to the scan of the distinct counts;
  // oversized buckets are placed at their own key range of the result's key
  // array (free between the scatter and the compaction)
  WS(stage_counts, uint32_t, "stage_counts", keys_cap);
  WS(bucket_d, unsigned long long, "bucket_d", max_buckets + 1);
  WS(bucket_out, uint64_t, "bucket_out", max_buckets + 2);
  WS(dtmp, uint64_t, "scan_tmp3", scan_u64_tmp_words(max_buckets + 1) + 8);
  SortCountArgs sa;
  memset(&sa, 0, sizeof(sa));
  sa.nbins = nbins;
  sa.bucket_base = bucket_base;
  sa.bucket_start = bstart;
  sa.bucket_size = bsize;
  sa.keys = keys;
  sa.scratch = out_keys;
  sa.stage_keys = keys;
  sa.stage_counts = stage_counts;
  sa.stage_cap = keys_cap;
  sa.bucket_d = bucket_d;
  sa.ticket = ticket;
  sa.big_list = big_list;
  sa.big_count = ticket + 2;
  sa.big_ticket = ticket + 3;
  sa.big_min = ea.big_min;
  // an opened bucket of n > cap keys has at most 3 n / cap + 1 slices
  const uint64_t task_cap = 4 * keys_cap / bucket_count_cap<K>() + 1024;
  WS(tasks, uint4, "count_tasks", task_cap);
  sa.tasks = tasks;
  sa.task_cap = task_cap;
  sa.task_count = ticket + 4;
  sa.task_ticket = ticket + 5;
  sa.bucket_head = bucket_head;
  sa.err = err;
  const size_t smem = bucket_count_smem_bytes<K>();
  if ((int)smem > c->max_smem_optin) return ctx_fail(c, GKC_ERR_INTERNAL, "count tables exceed shared memory");
  int occ = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_bucket_slices<K>, kBucketCountThreads, smem));
  sa.stamp = stamp + 5;
  const size_t sort_smem = bucket_sort_smem_bytes<K>();
  if ((int)sort_smem > c->max_smem_optin) return ctx_fail(c, GKC_ERR_INTERNAL, "sort areas exceed shared memory");
  int sort_occ = 0;
  auto sort_kernel = k_bucket_sort<K, false>;
  if constexpr (sizeof(K) == 8)
    if (narrow_groups(prm->k, keys_cap / nbins)) sort_kernel = k_bucket_sort<uint64_t, true>;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sort_occ, sort_kernel, kBucketSortThreads, sort_smem));
  sort_kernel<<<(unsigned)std::min<uint64_t>(max_buckets, (uint64_t)c->n_sms * std::max(sort_occ, 1)), kBucketSortThreads, sort_smem, c->st>>>(sa);
  LAUNCHED(c);
  // the large and rejected buckets, persistent, taken by ticket
  const int ctas = std::max(1, std::min(occ, c->tune.count_ctas ? (int)c->tune.count_ctas : 2));
  const unsigned open_grid = (unsigned)std::min<uint64_t>(keys_cap / bucket_count_cap<K>() + 1, (uint64_t)c->n_sms * ctas);
  k_bucket_open<K><<<open_grid, kBucketCountThreads, smem, c->st>>>(sa);
  LAUNCHED(c);
  k_bucket_slices<K><<<open_grid, kBucketCountThreads, smem, c->st>>>(sa);
  LAUNCHED(c);
  // final offsets: the exclusive scan of the distinct counts (the bucket count is read on the device)
  c->launches += scan_u64_dev(bucket_d, bucket_out, max_buckets, bucket_base + nbins, dtmp, c->st, stamp + 6);
  WS(out_counts, uint32_t, slot_name(c, "counts").c_str(), keys_cap);
  WS(bin_out, uint64_t, slot_name(c, "bin_out").c_str(), nbins + 1);
  // warps for every bucket and every 512 keys, at most what the chip holds
  const uint64_t compact_n = std::max(max_buckets, keys_cap / 512) / 8 + 1;
  k_compact_runs<K><<<(unsigned)std::min<uint64_t>(compact_n, (uint64_t)c->n_sms * 8), 256, 0, c->st>>>(keys, stage_counts, bstart, bucket_d, bucket_out, bucket_base,
                                                      nbins, out_keys, out_counts, bin_out, bucket_head, tasks, ticket + 4, err);
  LAUNCHED(c);
  c->count_keys_cap = keys_cap;
  return GKC_OK;
}

static gkc_status enqueue_count(gkc_ctx *c, const gkc_params *prm, uint64_t keys_cap) {
  if (prm->k <= 32) return enqueue_count_batched<uint64_t>(c, prm, keys_cap, 0);
  return enqueue_count_batched<u128>(c, prm, keys_cap, 0);
}

static void fill_count_view(gkc_ctx *c, const gkc_params *prm) {
  gkc_count_view &v = c->cv;
  memset(&v, 0, sizeof(v));
  v.n_distinct = c->h_tot->n_distinct;
  v.n_kmers = c->h_tot->n_kmers;
  v.nbins = (uint32_t)prm->nbins;
  v.key_words = prm->k <= 32 ? 1 : 2;
  v.bin_off = (const uint64_t *)c->bufs[slot_name(c, "bin_out")].p;
  v.keys = (const uint64_t *)c->bufs[slot_name(c, "out_keys")].p;
  v.counts = (const uint32_t *)c->bufs[slot_name(c, "counts")].p;
  c->ck = prm->k;
  c->have_count = true;
  c->count_gen++;
}

gkc_status count_device_impl(gkc_ctx *c, const gkc_params *prm, gkc_mode mode) {
  if (!c->have_part) return ctx_fail(c, GKC_ERR_INVALID_ARG, "no partition in the context");
  if (mode == GKC_MODE_PLAIN) return count_plain_impl(c, prm);
  uint64_t n_kmers = c->pv.n_kmers;
  uint64_t keys_cap = n_kmers + 16;
  CK(cudaMemsetAsync(c->bufs["err"].p, 0, 16, c->st));
  gkc_status s = enqueue_count(c, prm, keys_cap);
  if (s != GKC_OK) return s;
  s = read_totals(c, true, (uint32_t)prm->nbins);
  if (s != GKC_OK) return s;
  CK(cudaStreamSynchronize(c->st));
  if (c->h_tot->err & ERR_CAPACITY) return ctx_fail(c, GKC_ERR_CAPACITY, "key capacity");
  if (c->h_tot->err & ERR_BOUNDS) return check_device_err(c);
  s = check_device_err(c);
  if (s != GKC_OK) return s;
  fill_count_view(c, prm);
  return GKC_OK;
}

gkc_status gkc_count_device(gkc_ctx *c, const gkc_params *prm, gkc_mode mode, gkc_count_view *out) {
  if (!c) return GKC_ERR_INVALID_ARG;
  gkc_status s = check_params(c, prm);
  if (s != GKC_OK) return s;
  if (c->have_part && (prm->k != c->pp.k || prm->nbins != c->pp.nbins))
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "params differ from the partition's");
  cudaSetDevice(c->dev);
  c->launches = 0;
  CK(cudaEventRecord(c->ev[0], c->st));
  s = count_device_impl(c, prm, mode);
  if (s != GKC_OK) return s;
  CK(cudaEventRecord(c->ev[1], c->st));
  CK(cudaEventSynchronize(c->ev[1]));
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
  c->tm = gkc_timings{};
  c->tm.count_ms = ms;
  c->tm.total_ms = ms;
  c->tm.launches = c->launches;
  if (out) *out = c->cv;
  return GKC_OK;
}

// -------------------------------------------------------------- pipeline

// The batched pipeline's launches, on the context stream.
static gkc_status enqueue_pipeline(gkc_ctx *c, const gkc_params *prm, const GraphKey &key, const PipelineCaps &cap) {
  c->launches = 0;
  gkc_status s = enqueue_partition(c, prm, (const char *)key.reads, key.n_bytes, (const uint64_t *)key.offs, key.n_reads,
                                   cap.skm, cap.bytes);
  if (s == GKC_OK) s = enqueue_count(c, prm, cap.keys);
  if (s == GKC_OK) s = read_totals(c, true, (uint32_t)prm->nbins);
  return s;
}

// Grows the capacities to what the device reported.
static void grow_caps(PipelineCaps *cap, const DevTotals *t) {
  cap->skm = std::max<uint64_t>(cap->skm, t->n_skm + 16);
  cap->bytes = std::max<uint64_t>(cap->bytes, t->n_packed + 64);
  cap->keys = std::max<uint64_t>(cap->keys, t->n_kmers + 16);
}

// The launches as a graph: the workspaces were sized by a call with the same
// key and capacities, and nothing was freed or grown since (G.seen).
static gkc_status capture_pipeline(gkc_ctx *c, const gkc_params *prm, SlotGraph &G, bool async) {
  // the replaced graph has ended: a streaming call waits for the slot's previous call before it comes here
  if (!async) CK(cudaStreamSynchronize(c->st));
  if (G.exec) {
    cudaGraphExecDestroy(G.exec);
    G.exec = nullptr;
  }
  cudaGraph_t g;
  CK(cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal));
  c->capturing = true;
  const gkc_status s = enqueue_pipeline(c, prm, G.key, G.cap);
  const cudaError_t e = cudaStreamEndCapture(c->st, &g);
  c->capturing = false;
  if (s != GKC_OK) {
    if (e == cudaSuccess) cudaGraphDestroy(g);
    return s;
  }
  CK(e);
  const cudaError_t ei = cudaGraphInstantiate(&G.exec, g, 0);
  cudaGraphDestroy(g);
  if (ei != cudaSuccess) G.exec = nullptr;
  CK(ei);
  G.launches = c->launches;
  G.valid = true;
  return GKC_OK;
}

// Batched: the first call with some inputs and parameters enqueues the
// partition -> count pipeline launch by launch; the second one in a row (per
// buffer slot) captures the same launches as a CUDA graph, which is replayed
// from then on.  So inputs that are not run again pay for no capture, and a
// streaming call of a new size waits for nothing: the sizing run, the wait for
// it, the capture and the instantiation cost 1.7-2.7 ms of a 2.2 ms call when
// every size was captured at its first call.  All sizes the kernels need are
// read on the device.  With `async`, the pipeline is only enqueued: its totals
// land in the slot's pinned totals and are checked by the caller after the
// stream (`cap_used`: what it was run with, for a rerun).
static gkc_status pipeline_batched(gkc_ctx *c, const gkc_params *prm, const char *d_reads,
                                   uint64_t n_bytes, const uint64_t *d_offs, uint64_t n_reads,
                                   bool async = false, PipelineCaps *cap_used = nullptr) {
  const GraphKey key{d_reads, d_offs, n_bytes, n_reads, prm->k, prm->p, prm->hpc, prm->nbins, c->filter};
  SlotGraph &G = c->graphs[c->slot];
  PipelineCaps cap;
  if (G.key == key && (G.seen || G.valid)) {
    cap = G.cap;
  } else {
    partition_caps(prm, n_bytes, n_reads, &cap.skm, &cap.bytes);
    cap.keys = std::max<uint64_t>(n_bytes, 16);
  }
  cudaStreamCaptureStatus cs;
  CK(cudaStreamIsCapturing(c->st, &cs));
  if (cs != cudaStreamCaptureStatusNone) return ctx_fail(c, GKC_ERR_INVALID_ARG, "stream already capturing");
  for (int attempt = 0;; attempt++) {
    gkc_status s = GKC_OK;
    if (!(G.valid && G.key == key && G.exec) && G.seen && G.key == key && !c->one_shot) {
      s = capture_pipeline(c, prm, G, async);
      if (s != GKC_OK) {
        G.seen = false;
        return s;
      }
    }
    if (G.valid && G.key == key && G.exec) {
      CK(cudaGraphLaunch(G.exec, c->st));
      c->tm.graph_replayed = 1;
      c->launches = G.launches;
    } else {
      G.valid = G.seen = false;
      s = enqueue_pipeline(c, prm, key, cap);
      if (s != GKC_OK) return s;
      c->tm.graph_replayed = 0;
      G.key = key;
      G.cap = cap;
      G.seen = true;
    }
    if (async) {
      if (cap_used) *cap_used = cap;
      return GKC_OK;
    }
    CK(cudaStreamSynchronize(c->st));
    if (!(c->h_tot->err & ERR_CAPACITY)) break;
    // grow to the sizes the device reported and retry
    graphs_invalidate(c);
    if (attempt == 2) return ctx_fail(c, GKC_ERR_CAPACITY, "pipeline capacity");
    grow_caps(&cap, c->h_tot);
  }
  gkc_status s = check_device_err(c);
  if (s != GKC_OK) return s;
  read_stage_times(c);
  fill_partition_view(c, prm, n_reads, n_bytes);
  fill_count_view(c, prm);
  return GKC_OK;
}

gkc_status gkc_pipeline_device(gkc_ctx *c, const gkc_params *prm, gkc_mode mode,
                               const char *d_reads, uint64_t n_bytes, const uint64_t *d_offs,
                               uint64_t n_reads, gkc_partition_view *part, gkc_count_view *cnt) {
  if (!c) return GKC_ERR_INVALID_ARG;
  gkc_status s = check_params(c, prm);
  if (s != GKC_OK) return s;
  if (n_bytes > 0 && (!d_reads || !d_offs)) return ctx_fail(c, GKC_ERR_INVALID_ARG, "null input");
  cudaSetDevice(c->dev);
  c->tm = gkc_timings{};
  CK(cudaEventRecord(c->ev[0], c->st));
  if (mode == GKC_MODE_BATCHED) {
    s = pipeline_batched(c, prm, d_reads, n_bytes, d_offs, n_reads);
  } else {
    c->launches = 0;
    s = partition_plain_impl(c, prm, d_reads, n_bytes, d_offs, n_reads);
    if (s == GKC_OK) {
      CK(cudaEventRecord(c->ev[2], c->st));
      s = count_plain_impl(c, prm);
    }
  }
  if (s != GKC_OK) return s;
  CK(cudaEventRecord(c->ev[1], c->st));
  CK(cudaEventSynchronize(c->ev[1]));
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
  c->tm.total_ms = ms;
  c->tm.launches = c->launches;
  if (part) *part = c->pv;
  if (cnt) *cnt = c->cv;
  return GKC_OK;
}

// A call with inputs in host memory that fails while they are being copied
// ends only when they are no longer read: page-locked ones are copied after
// the copy's own call has returned.
struct SettleOnError {
  gkc_ctx *c;
  bool ok = false;
  explicit SettleOnError(gkc_ctx *ctx) : c(ctx) {}
  ~SettleOnError() {
    if (ok) return;
    if (c->st_up) cudaStreamSynchronize(c->st_up);
    cudaStreamSynchronize(c->st);
  }
};

// Host entry: H2D of reads and rebased offsets, then the device pipeline.
gkc_status upload_reads(gkc_ctx *c, const char *reads, const uint64_t *offs, uint64_t n_reads,
                        char **d_reads, uint64_t **d_offs, uint64_t *n_bytes) {
  const uint64_t base = n_reads ? offs[0] : 0;
  const uint64_t nb = n_reads ? offs[n_reads] - base : 0;
  WS(dr, char, slot_name(c, "in_reads").c_str(), nb + 64);
  WS(doffs, uint64_t, slot_name(c, "in_offs").c_str(), n_reads + 1);
  if (nb) CK(cudaMemcpyAsync(dr, reads + base, nb, cudaMemcpyHostToDevice, c->st));
  if (base == 0) {
    CK(cudaMemcpyAsync(doffs, offs, (n_reads + 1) * 8, cudaMemcpyHostToDevice, c->st));
  } else {
    c->offs_tmp.resize(n_reads + 1);
    for (uint64_t r = 0; r <= n_reads; r++) c->offs_tmp[r] = offs[r] - base;
    CK(cudaMemcpyAsync(doffs, c->offs_tmp.data(), (n_reads + 1) * 8, cudaMemcpyHostToDevice, c->st));
    CK(cudaStreamSynchronize(c->st));
  }
  *d_reads = dr;
  *d_offs = doffs;
  *n_bytes = nb;
  return GKC_OK;
}

gkc_status gkc_partition_host(gkc_ctx *c, const gkc_params *prm, const char *reads,
                              const uint64_t *offs, uint64_t n_reads, gkc_partition_view *out) {
  if (!c || (n_reads && (!reads || !offs))) return GKC_ERR_INVALID_ARG;
  gkc_status s = check_params(c, prm);
  if (s != GKC_OK) return s;
  cudaSetDevice(c->dev);
  SettleOnError settle(c);
  char *dr;
  uint64_t *doffs, nb;
  s = upload_reads(c, reads, offs, n_reads, &dr, &doffs, &nb);
  if (s != GKC_OK) return s;
  s = gkc_partition_device(c, prm, dr, nb, doffs, n_reads, out);
  settle.ok = s == GKC_OK;
  return s;
}

gkc_status gkc_pipeline_host(gkc_ctx *c, const gkc_params *prm, gkc_mode mode, const char *reads,
                             const uint64_t *offs, uint64_t n_reads, gkc_count_view *cnt) {
  if (!c || (n_reads && (!reads || !offs))) return GKC_ERR_INVALID_ARG;
  gkc_status s = check_params(c, prm);
  if (s != GKC_OK) return s;
  cudaSetDevice(c->dev);
  CK(cudaEventRecord(c->ev[3], c->st));
  SettleOnError settle(c);
  char *dr;
  uint64_t *doffs, nb;
  s = upload_reads(c, reads, offs, n_reads, &dr, &doffs, &nb);
  if (s != GKC_OK) return s;
  s = gkc_pipeline_device(c, prm, mode, dr, nb, doffs, n_reads, nullptr, cnt);
  if (s != GKC_OK) return s;
  settle.ok = true;
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev[3], c->ev[0]);
  c->tm.h2d_ms = ms;
  return GKC_OK;
}

// ------------------------------------------------------ streaming host form

// offs[i] -= offs[0] (offsets of a batch cut from a larger CSR); one CTA
__global__ void k_rebase_offs(uint64_t *offs, uint64_t n) {
  const uint64_t base = offs[0];
  __syncthreads();  // every thread has read offs[0]
  for (uint64_t i = threadIdx.x + 1; i <= n; i += blockDim.x) offs[i] -= base;
  __syncthreads();
  if (threadIdx.x == 0) offs[0] = 0;
}
// The context on a streaming call's slot; every way out leaves it on slot 0.
struct OnSlot {
  gkc_ctx *c;
  OnSlot(gkc_ctx *ctx, int slot) : c(ctx) {
    c->slot = slot;
    c->h_tot = c->h_tots[slot];
  }
  ~OnSlot() {
    c->slot = 0;
    c->h_tot = c->h_tots[0];
  }
};

static void set_results(gkc_ctx *c, StreamCall &sc) {
  sc.d_bin_off = c->bufs[slot_name(c, "bin_out")].p;
  sc.d_keys = c->bufs[slot_name(c, "out_keys")].p;
  sc.d_counts = c->bufs[slot_name(c, "counts")].p;
}

// A streaming call whose workspaces were too small for its reads (sized from
// their number of bases, or by an earlier call of that size) is run again with
// the sizes the device reported: its inputs stay in the slot until its
// download is enqueued.  Waits for the device.
static gkc_status rerun_larger(gkc_ctx *c, StreamCall &sc, int slot) {
  OnSlot on(c, slot);
  const int filter = c->filter;
  c->filter = sc.key.filter;
  gkc_status s = GKC_OK;
  for (int attempt = 0; attempt < 2 && s == GKC_OK && (c->h_tot->err & ERR_CAPACITY); attempt++) {
    grow_caps(&sc.cap, c->h_tot);
    graphs_invalidate(c);
    s = enqueue_pipeline(c, &sc.prm, sc.key, sc.cap);
    const cudaError_t e = cudaStreamSynchronize(c->st);
    if (s == GKC_OK && e != cudaSuccess) s = ctx_cuda(c, e, "rerunning a streaming call");
  }
  c->filter = filter;
  if (s != GKC_OK) return s;
  set_results(c, sc);
  SlotGraph &G = c->graphs[slot];
  if (!(c->h_tot->err & ERR_CAPACITY)) {
    G.key = sc.key;
    G.cap = sc.cap;
    G.seen = true;
  }
  return GKC_OK;
}

// The download of a streaming call: once its pipeline is done, its totals
// (copied to page-locked memory inside the captured pipeline) give the exact
// sizes, and three DMA copies on the download stream move the bin offsets,
// keys and counts into the caller's page-locked buffers while the next call
// computes.  Blocks until the call's pipeline is done.  rec: the call's
// record (ticket & 3); its slot is ticket & 1.
static gkc_status issue_download(gkc_ctx *c, int rec) {
  StreamCall &sc = c->calls[rec];
  if (sc.dl_issued) return GKC_OK;
  const int slot = (int)(sc.ticket & 1);
  CK(cudaEventSynchronize(c->ev_comp[slot]));
  if (c->h_tots[slot]->err & ERR_CAPACITY) {
    sc.status = rerun_larger(c, sc, slot);
    if (sc.status != GKC_OK) sc.message = c->err;
  }
  sc.tot = *c->h_tots[slot];  // the slot's next call overwrites them
  const DevTotals *h = &sc.tot;
  const bool bad = sc.status != GKC_OK ||
                   (h->err & (ERR_CAPACITY | ERR_BIN_TOO_LARGE | ERR_SPIN_TIMEOUT | ERR_BOUNDS |
                              ERR_BAD_READ)) != 0;
  if (!bad) {
    const uint64_t nd = std::min<uint64_t>(h->n_distinct, sc.capacity);
    if (sc.h_bin_off)
      CK(cudaMemcpyAsync(sc.h_bin_off, sc.d_bin_off, 8 * ((uint64_t)sc.prm.nbins + 1), cudaMemcpyDeviceToHost, c->st_dl));
    if (sc.h_keys && nd)
      CK(cudaMemcpyAsync(sc.h_keys, sc.d_keys, nd * 8 * (uint64_t)sc.key_words, cudaMemcpyDeviceToHost, c->st_dl));
    if (sc.h_counts && nd)
      CK(cudaMemcpyAsync(sc.h_counts, sc.d_counts, nd * 4, cudaMemcpyDeviceToHost, c->st_dl));
  }
  CK(cudaEventRecord(c->ev_dl[rec], c->st_dl));
  sc.dl_issued = true;
  return GKC_OK;
}

static bool host_visible(const void *p) {
  if (!p) return true;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost && a.devicePointer != nullptr;
}

gkc_status gkc_stream_submit(gkc_ctx *c, const gkc_params *prm, const char *reads, const uint64_t *offs,
                             uint64_t n_reads, uint64_t *bin_off, uint64_t *keys, uint32_t *counts,
                             uint64_t capacity, uint64_t *ticket) {
  if (!c || !ticket || (n_reads && (!reads || !offs))) return GKC_ERR_INVALID_ARG;
  gkc_status s = check_params(c, prm);
  if (s != GKC_OK) return s;
  if (!host_visible(reads) || !host_visible(offs) || !host_visible(bin_off) || !host_visible(keys) ||
      !host_visible(counts))
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "streaming buffers must be page-locked host memory");
  cudaSetDevice(c->dev);
  if (!c->st_up) {
    CK(cudaStreamCreateWithFlags(&c->st_up, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&c->st_dl, cudaStreamNonBlocking));
    for (int i = 0; i < 2; i++) {
      CK(cudaEventCreateWithFlags(&c->ev_up[i], cudaEventDisableTiming));
      CK(cudaEventCreateWithFlags(&c->ev_comp[i], cudaEventDisableTiming));
    }
    for (int i = 0; i < 4; i++) CK(cudaEventCreateWithFlags(&c->ev_dl[i], cudaEventDisableTiming));
  }
  const uint64_t t = c->next_ticket;
  const int slot = (int)(t & 1), rec = (int)(t & 3);
  if (!c->calls[rec].waited)
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "four calls await their wait: wait for the oldest first");
  // the slot's previous call must have its download enqueued before its
  // buffers are reused
  const int prev = (int)((t + 2) & 3);  // record of call t - 2
  if (t >= 2) {
    s = issue_download(c, prev);
    if (s != GKC_OK) return s;
  }
  // the slot's input buffers; growing them waits for everything in flight
  const uint64_t base = n_reads ? offs[0] : 0, nb = n_reads ? offs[n_reads] - base : 0;
  OnSlot on(c, slot);
  const std::string rn = slot_name(c, "in_reads"), ofn = slot_name(c, "in_offs");
  auto fits = [&](const std::string &n, size_t bytes) {
    auto it = c->bufs.find(n);
    return it != c->bufs.end() && it->second.bytes >= bytes;
  };
  if (!fits(rn, nb + 64) || !fits(ofn, 8 * (n_reads + 1))) {
    CK(cudaStreamSynchronize(c->st_up));
    CK(cudaStreamSynchronize(c->st_dl));
    CK(cudaStreamSynchronize(c->st));
  }
  WS(dr, char, rn.c_str(), nb + 64);
  WS(doffs, uint64_t, ofn.c_str(), n_reads + 1);
  SettleOnError settle(c);
  // inputs of the slot's previous call must have been read before they are replaced
  if (t >= 2) CK(cudaStreamWaitEvent(c->st_up, c->ev_comp[slot], 0));
  if (nb) CK(cudaMemcpyAsync(dr, reads + base, nb, cudaMemcpyHostToDevice, c->st_up));
  CK(cudaMemcpyAsync(doffs, offs, 8 * (n_reads + 1), cudaMemcpyHostToDevice, c->st_up));
  CK(cudaEventRecord(c->ev_up[slot], c->st_up));
  CK(cudaStreamWaitEvent(c->st, c->ev_up[slot], 0));
  // and its outputs must have been copied out before they are recomputed
  if (t >= 2) CK(cudaStreamWaitEvent(c->st, c->ev_dl[prev], 0));
  if (base) {
    k_rebase_offs<<<1, 1024, 0, c->st>>>(doffs, n_reads);
    LAUNCHED(c);
  }
  c->tm = gkc_timings{};
  StreamCall sc;
  s = pipeline_batched(c, prm, dr, nb, doffs, n_reads, true, &sc.cap);
  if (s != GKC_OK) return s;
  CK(cudaEventRecord(c->ev_comp[slot], c->st));
  sc.key = GraphKey{dr, doffs, nb, n_reads, prm->k, prm->p, prm->hpc, prm->nbins, c->filter};
  sc.prm = *prm;
  sc.ticket = t;
  sc.capacity = capacity;
  sc.key_words = prm->k <= 32 ? 1 : 2;
  sc.h_bin_off = bin_off;
  sc.h_keys = keys;
  sc.h_counts = counts;
  set_results(c, sc);
  sc.dl_issued = false;
  sc.waited = false;
  c->calls[rec] = sc;
  c->next_ticket = t + 1;
  *ticket = t;
  settle.ok = true;  // the call is in flight: its inputs are read until its wait
  // the previous call (the other slot), if its pipeline is already done:
  // start its download now
  if (t >= 1) {
    const int last = (int)((t + 3) & 3);
    if (!c->calls[last].dl_issued && cudaEventQuery(c->ev_comp[slot ^ 1]) == cudaSuccess) {
      s = issue_download(c, last);
      if (s != GKC_OK) return s;
    }
  }
  return GKC_OK;
}

gkc_status gkc_stream_wait(gkc_ctx *c, uint64_t ticket, uint64_t *n_distinct, uint64_t *n_kmers) {
  if (!c) return GKC_ERR_INVALID_ARG;
  const int rec = (int)(ticket & 3);
  StreamCall &sc = c->calls[rec];
  if (sc.ticket != ticket || sc.waited) return ctx_fail(c, GKC_ERR_NOT_FOUND, "no call in flight with this ticket");
  cudaSetDevice(c->dev);
  gkc_status s = issue_download(c, rec);
  if (s != GKC_OK) return s;
  CK(cudaEventSynchronize(c->ev_dl[rec]));
  sc.waited = true;
  if (sc.status != GKC_OK) return ctx_fail(c, sc.status, sc.message);
  const DevTotals *h = &sc.tot;
  if (n_distinct) *n_distinct = h->n_distinct;
  if (n_kmers) *n_kmers = h->n_kmers;
  if (h->err & ERR_CAPACITY)
    return ctx_fail(c, GKC_ERR_CAPACITY, "pipeline capacity");
  s = device_err(c, h->err);
  if (s != GKC_OK) return s;
  if (h->n_distinct > sc.capacity)
    return ctx_fail(c, GKC_ERR_CAPACITY, "result larger than the output capacity (bin offsets and the first entries copied)");
  return GKC_OK;
}

// --------------------------------------------------------------- copy out

gkc_status gkc_partition_copy_out(gkc_ctx *c, uint64_t *bin_skm_off, uint32_t *skm_len,
                                  uint64_t *skm_byte_off, uint8_t *packed, uint32_t *minimizer) {
  if (!c || !c->have_part) return GKC_ERR_INVALID_ARG;
  cudaSetDevice(c->dev);
  const gkc_partition_view &v = c->pv;
  if (bin_skm_off)
    CK(cudaMemcpyAsync(bin_skm_off, v.bin_skm_off, (v.nbins + 1) * 8, cudaMemcpyDeviceToHost, c->st));
  if (minimizer && v.n_superkmers) {
    if (v.skm_minimizer)
      CK(cudaMemcpyAsync(minimizer, v.skm_minimizer, v.n_superkmers * 4, cudaMemcpyDeviceToHost, c->st));
    else  // an imported partition and superkmers from the host have no minimizers
      memset(minimizer, 0xFF, v.n_superkmers * 4);
  }
  if (packed && v.n_packed_bytes)
    CK(cudaMemcpyAsync(packed, v.packed, v.n_packed_bytes, cudaMemcpyDeviceToHost, c->st));
  if ((skm_len || skm_byte_off) && v.n_superkmers) {
    c->desc_tmp.resize(v.n_superkmers);
    CK(cudaMemcpyAsync(c->desc_tmp.data(), v.skm_desc, v.n_superkmers * 8, cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    for (uint64_t i = 0; i < v.n_superkmers; i++) {
      if (skm_len) skm_len[i] = (uint32_t)(c->desc_tmp[i] & 0xFFFFFFu);
      if (skm_byte_off) skm_byte_off[i] = c->desc_tmp[i] >> 24;
    }
  }
  CK(cudaStreamSynchronize(c->st));
  return GKC_OK;
}

// The partition kernels already hold, per bin, the superkmer prefix and the
// k-mer prefix; a superkmer of w k-mers has w + k - 1 bases, so the bases of
// bin b are its k-mers plus (k - 1) per superkmer.  Only the two prefix
// arrays (nbins + 1 words each) cross to the host.
gkc_status gkc_partition_balance(gkc_ctx *c, uint64_t *bin_bases, uint32_t capacity,
                                 gkc_balance_stats *st) {
  if (!c || !c->have_part) return GKC_ERR_INVALID_ARG;
  cudaSetDevice(c->dev);
  const gkc_partition_view &v = c->pv;
  const uint32_t nb = v.nbins;
  if (bin_bases && capacity < nb)
    return ctx_fail(c, GKC_ERR_CAPACITY, "bin_bases holds " + std::to_string(capacity) + " entries, the partition has " +
                                             std::to_string(nb) + " bins");
  std::vector<uint64_t> so(nb + 1), ko(nb + 1);
  CK(cudaMemcpyAsync(so.data(), v.bin_skm_off, (nb + 1) * 8, cudaMemcpyDeviceToHost, c->st));
  CK(cudaMemcpyAsync(ko.data(), v.bin_kmer_off, (nb + 1) * 8, cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  const uint64_t km1 = (uint64_t)(c->pp.k - 1);
  gkc_balance_stats s{};
  s.min = ~0ull;
  std::vector<uint64_t> sz(nb);
  for (uint32_t b = 0; b < nb; b++) {
    sz[b] = (ko[b + 1] - ko[b]) + km1 * (so[b + 1] - so[b]);
    s.total += sz[b];
    s.max = std::max(s.max, sz[b]);
    s.min = std::min(s.min, sz[b]);
  }
  s.mean = nb ? s.total / nb : 0;
  double acc = 0.0;
  for (uint32_t b = 0; b < nb; b++) {
    const uint64_t d = sz[b] - s.mean;  // wraps below the mean; the square is the same mod 2^64
    acc += (double)(d * d);
  }
  s.variance = nb ? acc / nb : 0.0;
  s.stdev = std::sqrt(s.variance);
  s.cv = s.stdev / (double)s.mean;
  if (bin_bases) std::copy(sz.begin(), sz.end(), bin_bases);
  if (st) *st = s;
  return GKC_OK;
}

gkc_status gkc_count_copy_out(gkc_ctx *c, uint64_t *bin_off, uint64_t *keys, uint32_t *counts) {
  if (!c || !c->have_count) return GKC_ERR_INVALID_ARG;
  cudaSetDevice(c->dev);
  const gkc_count_view &v = c->cv;
  CK(cudaEventRecord(c->ev[2], c->st));
  // cudaMemcpyDefault: each destination may be host or device memory
  if (bin_off)
    CK(cudaMemcpyAsync(bin_off, v.bin_off, (v.nbins + 1) * 8, cudaMemcpyDefault, c->st));
  if (keys && v.n_distinct)
    CK(cudaMemcpyAsync(keys, v.keys, v.n_distinct * 8 * v.key_words, cudaMemcpyDefault, c->st));
  if (counts && v.n_distinct)
    CK(cudaMemcpyAsync(counts, v.counts, v.n_distinct * 4, cudaMemcpyDefault, c->st));
  CK(cudaEventRecord(c->ev[3], c->st));
  CK(cudaStreamSynchronize(c->st));
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev[2], c->ev[3]);
  c->tm.d2h_ms = ms;
  return GKC_OK;
}

// Descriptors of one bin of superkmers from their lengths and byte offsets,
// and the bin's totals where the count stage reads a partition's.
__global__ void k_one_bin(const uint32_t *len, const uint64_t *boff, uint64_t n, uint64_t n_bytes, uint64_t n_kmers,
                          uint64_t *desc, uint64_t *bin_start, uint64_t *bin_kstart, unsigned long long *cursors,
                          uint32_t *err) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    desc[i] = (boff[i] << 24) | len[i];
  if (blockIdx.x == 0 && threadIdx.x < 4) {
    const int t = threadIdx.x;
    if (t < 2) bin_start[t] = t ? n : 0;
    if (t < 2) bin_kstart[t] = t ? n_kmers : 0;
    cursors[t] = t == 0 ? n : t == 1 ? n_bytes : 0;
    err[t] = 0;
  }
}

// One bin of packed superkmers from the host (kmc_counting_GPU drop-in).  The
// host only sums the lengths (the packed bytes to copy, the k-mers to expect)
// and checks them; descriptors are built on the device from the lengths, which
// are half their bytes: 1 M superkmers of 42 bases from pageable memory took
// 2.7 ms with the descriptors built and copied by the host, 2.0 so (0.6 of it
// the count stage, the rest mostly the copies).
gkc_status gkc_count_superkmers_host(gkc_ctx *c, int k, const uint32_t *skm_len,
                                     const uint8_t *packed, uint64_t n_skm, gkc_mode mode,
                                     uint64_t *n_distinct) {
  if (!c || k < 1 || k > 64 || (n_skm && (!skm_len || !packed))) return GKC_ERR_INVALID_ARG;
  cudaSetDevice(c->dev);
  uint64_t off = 0, nk = 0;
  uint32_t longest = 0;
  const uint32_t ku = (uint32_t)k;
  for (uint64_t i = 0; i < n_skm; i++) {  // no branch: the compiler makes vectors of it
    const uint32_t len = skm_len[i];
    longest = std::max(longest, len);
    off += ((uint64_t)len + 3) / 4;
    nk += len >= ku ? len - ku + 1 : 0u;
  }
  if (longest > 0xFFFFFFu) return ctx_fail(c, GKC_ERR_INVALID_ARG, "superkmer too long");
  WS(dd, uint64_t, "skm_desc_bin", n_skm + 1);
  WS(dp, uint8_t, "packed_bin", off + 16);
  WS(dl, uint32_t, "skm_mm_bin", n_skm + 1);  // the lengths, where a partition keeps its minimizers
  WS(bs, uint64_t, "bin_start", 2);
  WS(bk, uint64_t, "bin_kstart", 2);
  WS(cur, unsigned long long, "cursors", 4);
  WS(err, uint32_t, "err", 4);
  WS(boff, uint64_t, "skm_koff", n_skm + 3);  // filled again by the count stage
  WS(btmp, uint64_t, "scan_tmp2", scan_u64_tmp_words(n_skm + 1) + 8);
  SettleOnError settle(c);
  // both copies before the kernels: a copy from pageable memory waits for the stream
  if (n_skm) CK(cudaMemcpyAsync(dl, skm_len, n_skm * 4, cudaMemcpyHostToDevice, c->st));
  if (off) CK(cudaMemcpyAsync(dp, packed, off, cudaMemcpyHostToDevice, c->st));
  c->part_packed = dp;
  if (n_skm) scan_len_bytes(dl, boff, n_skm, btmp, c->st);
  k_one_bin<<<(unsigned)std::min<uint64_t>(n_skm / 256 + 1, (uint64_t)c->n_sms * 8), 256, 0, c->st>>>(
      dl, boff, n_skm, off, nk, dd, bs, bk, cur, err);
  CK(cudaPeekAtLastError());
  c->pv = gkc_partition_view{};
  c->pv.n_superkmers = n_skm;
  c->pv.n_packed_bytes = off;
  c->pv.n_kmers = nk;
  c->pv.nbins = 1;
  c->pv.bin_skm_off = bs;
  c->pv.bin_kmer_off = bk;
  c->pv.skm_desc = dd;
  c->pv.skm_minimizer = nullptr;  // these superkmers come without
  c->pv.packed = dp;
  c->part_nbytes_dev = nullptr;
  // the count path sizes its per-superkmer arrays from the partition's
  // capacities, which a fresh context has not set
  c->part_cap_skm = n_skm + 1;
  c->part_cap_bytes = off + 16;
  c->have_part = true;
  gkc_params prm{k, 3, 0, 1};
  c->pp = prm;
  graphs_invalidate(c);
  gkc_status s = gkc_count_device(c, &prm, mode, nullptr);
  if (s != GKC_OK) return s;
  settle.ok = true;
  if (n_distinct) *n_distinct = c->cv.n_distinct;
  return GKC_OK;
}
