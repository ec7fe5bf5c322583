// Count output options on the device: the frequency filter of the reference
// (kmc_counting_GPU keeps a k-mer when kmer_min_freq <= count <=
// kmer_max_freq, kmer_counting.cu:188-190, defaults utilities.hpp:109; the
// filter is commented out there) and the merged global list (one sorted list
// over all bins, with the counts of a k-mer that occurs in several bins --
// possible when reads hold N -- added up).
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "ctx.h"
#include "kernels.h"
#include "onesweep.h"

namespace gkc {

constexpr int KP_NT = 256;
constexpr int KP_ROWS = 8;  // rows of 32 entries a warp
constexpr int KP_TILE = KP_NT * KP_ROWS;

// Entries with a count in [lo, hi], of the warp's rows from w0 on: bit l of
// h[t] is entry l of row t, c[t] the lane's count there.
GKC_DEV uint32_t keep_rows(const uint32_t *counts, uint64_t n, uint64_t w0, uint32_t lo, uint32_t hi,
                           uint32_t (&c)[KP_ROWS], uint32_t (&h)[KP_ROWS]) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int t = 0; t < KP_ROWS; t++) {
    const uint64_t i = w0 + 32 * t + lane;
    c[t] = i < n ? counts[i] : 0u;
  }
  uint32_t sum = 0;
#pragma unroll
  for (int t = 0; t < KP_ROWS; t++) {
    h[t] = __ballot_sync(0xffffffffu, w0 + 32 * t + lane < n && c[t] >= lo && c[t] <= hi);
    sum += __popc(h[t]);
  }
  return sum;
}

// The filter as one compaction over tiles: kept entries per tile, a scan of
// the tiles, then keys and counts written in order.  Bound by memory: the
// counts are read twice, the keys once.  (A flag and a place of eight bytes
// each for every entry: 8.7 M entries 110 us, so 50.)
__global__ void __launch_bounds__(KP_NT) k_keep_count(const uint32_t *counts, uint64_t n, uint32_t lo, uint32_t hi,
                                                      unsigned long long *blk) {
  __shared__ uint32_t cnt[KP_NT / 32];
  uint32_t c[KP_ROWS], h[KP_ROWS];
  const int warp = threadIdx.x >> 5;
  const uint32_t sum = keep_rows(counts, n, (uint64_t)blockIdx.x * KP_TILE + warp * 32 * KP_ROWS, lo, hi, c, h);
  if ((threadIdx.x & 31) == 0) cnt[warp] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = 0;
    for (int w = 0; w < KP_NT / 32; w++) s += cnt[w];
    blk[blockIdx.x] = s;
  }
}

template <typename K>
__global__ void __launch_bounds__(KP_NT) k_keep_copy(const K *keys, const uint32_t *counts, uint64_t n, uint32_t lo,
                                                     uint32_t hi, const uint64_t *blk_off, K *out_keys,
                                                     uint32_t *out_counts) {
  __shared__ uint32_t cnt[KP_NT / 32];
  uint32_t c[KP_ROWS], h[KP_ROWS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t w0 = (uint64_t)blockIdx.x * KP_TILE + warp * 32 * KP_ROWS;
  const uint32_t sum = keep_rows(counts, n, w0, lo, hi, c, h);
  if (lane == 0) cnt[warp] = sum;
  __syncthreads();
  uint64_t at = blk_off[blockIdx.x];
  for (int w = 0; w < warp; w++) at += cnt[w];
#pragma unroll
  for (int t = 0; t < KP_ROWS; t++) {
    if ((h[t] >> lane) & 1u) {
      const uint64_t to = at + __popc(h[t] & ((1u << lane) - 1u));
      out_keys[to] = keys[w0 + 32 * t + lane];
      out_counts[to] = c[t];
    }
    at += __popc(h[t]);
  }
}

// bin b of the kept list starts where bin b of the full list started: the
// kept entries of the tiles before, and of its tile up to there (a warp a bin)
__global__ void k_keep_bins(const uint64_t *bin_off, uint32_t nbins, const uint32_t *counts, uint32_t lo, uint32_t hi,
                            const uint64_t *blk_off, uint64_t *out) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint64_t b = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; b <= nbins;
       b += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint64_t e = bin_off[b], tile = e / KP_TILE;
    uint32_t k = 0;
    for (uint64_t i = tile * KP_TILE + lane; i < e; i += 32) k += counts[i] >= lo && counts[i] <= hi ? 1u : 0u;
    k = __reduce_add_sync(0xffffffffu, k);
    if (lane == 0) out[b] = blk_off[tile] + k;
  }
}

// sum of the counts of each run of equal keys (runs start at starts[j])
__global__ void k_run_sums(const uint32_t *vals, const uint64_t *starts, uint64_t d, uint64_t n, uint32_t *out) {
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < d; j += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t e = j + 1 < d ? starts[j + 1] : n;
    uint64_t s = 0;
    for (uint64_t i = starts[j]; i < e; i++) s += vals[i];
    out[j] = s > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)s;
  }
}

}  // namespace gkc

using namespace gkc;

#define CK(call)                                  \
  do {                                            \
    gkc_status _s = ctx_cuda(c, (call), #call);   \
    if (_s != GKC_OK) return _s;                  \
  } while (0)
#define WS(ptr, type, name, count)                                      \
  type *ptr;                                                            \
  do {                                                                  \
    gkc_status _s;                                                      \
    ptr = (type *)ws_get(c, name, sizeof(type) * (size_t)(count), &_s); \
    if (_s != GKC_OK) return _s;                                        \
  } while (0)

// Keeps the entries of (keys, counts, bin_off) whose count is in [lo, hi];
// returns the kept list in the "flt_*" workspaces.
template <typename K>
static gkc_status keep_range(gkc_ctx *c, const K *keys, const uint32_t *counts, const uint64_t *bin_off,
                             uint32_t nbins, uint64_t n, uint32_t lo, uint32_t hi, uint64_t *n_out) {
  const uint64_t tiles = (n + KP_TILE - 1) / KP_TILE;
  WS(blk, unsigned long long, "flt_tile_cnt", tiles + 1);
  WS(off, uint64_t, "flt_tile_off", tiles + 2);
  WS(stmp, uint64_t, "flt_scan_tmp", scan_u64_tmp_words(tiles + 1) + 8);
  WS(ok, K, "flt_keys", n + 1);
  WS(oc, uint32_t, "flt_counts", n + 1);
  WS(ob, uint64_t, "flt_bin_off", nbins + 1);
  if (tiles) k_keep_count<<<(unsigned)tiles, KP_NT, 0, c->st>>>(counts, n, lo, hi, blk);
  scan_u64(blk, off, tiles, stmp, c->st);
  if (tiles) k_keep_copy<K><<<(unsigned)tiles, KP_NT, 0, c->st>>>(keys, counts, n, lo, hi, off, ok, oc);
  k_keep_bins<<<(unsigned)std::min<uint64_t>((nbins + 8) / 8, (uint64_t)c->n_sms * 8), 256, 0, c->st>>>(
      bin_off, nbins, counts, lo, hi, off, ob);
  CK(cudaPeekAtLastError());
  CK(cudaMemcpyAsync(n_out, off + tiles, 8, cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  return GKC_OK;
}

template <typename K>
static gkc_status count_output_t(gkc_ctx *c, uint32_t lo, uint32_t hi, int merged, uint64_t *n_out,
                                 uint32_t *nbins_out) {
  const gkc_count_view &v = c->cv;
  const uint64_t n = v.n_distinct;
  const K *keys = reinterpret_cast<const K *>(v.keys);
  if (!merged) {
    *nbins_out = v.nbins;
    return keep_range<K>(c, keys, v.counts, v.bin_off, v.nbins, n, lo, hi, n_out);
  }
  // merged: sort (key, count) pairs by key, sum the counts of equal keys
  const unsigned grid = c->n_sms * 8;
  WS(mk, K, "merge_keys", n + 16);
  WS(mk2, K, "merge_keys_alt", n + 16);
  WS(mv, uint32_t, "merge_vals", n + 16);
  WS(mv2, uint32_t, "merge_vals_alt", n + 16);
  WS(nd, uint64_t, "merge_n", 2);
  CK(cudaMemcpyAsync(mk, keys, n * sizeof(K), cudaMemcpyDeviceToDevice, c->st));
  CK(cudaMemcpyAsync(mv, v.counts, n * 4, cudaMemcpyDeviceToDevice, c->st));
  uint64_t hn = n;
  CK(cudaMemcpyAsync(nd, &hn, 8, cudaMemcpyHostToDevice, c->st));
  WS(os_hist, unsigned long long, "merge_os_hist", 16 * 256);
  WS(os_lb, unsigned long long, "merge_os_lookback", onesweep_lookback_words(n + 1));
  WS(os_ticket, unsigned long long, "merge_os_ticket", 2);
  WS(err, uint32_t, "merge_err", 4);
  CK(cudaMemsetAsync(err, 0, 16, c->st));
  OnesweepScratch os{os_hist, os_lb, os_ticket, err, c->n_sms * 4};
  uint32_t launches = 0;
  const PairsStatus r = sort_pairs<K>(mk, mk2, mv, mv2, nd, n, 2 * c->ck, os, c->st, &launches);
  int in_alt = r.result_in_alt;
  const uint64_t nblk = rle_block_count(n);
  WS(rblk, unsigned long long, "merge_rle_blk", nblk + 1);
  WS(roff, uint64_t, "merge_rle_off", nblk + 2);
  WS(rtmp, uint64_t, "merge_rle_tmp", scan_u64_tmp_words(nblk + 1) + 8);
  WS(cur, unsigned long long, "merge_cursor", 2);
  WS(uk, K, "merge_unique_keys", n + 1);
  WS(st, uint64_t, "merge_starts", n + 1);
  WS(us, uint32_t, "merge_sums", n + 1);
  WS(bo, uint64_t, "merge_bin_off", 2);
  uint64_t d = 0;
  uint32_t e = 0;
  unsigned long long rest = 0;
  for (int pass = 0; pass < 2; pass++) {  // once more where long runs were left
    CK(cudaMemsetAsync(cur, 0, 16, c->st));
    rle_runs<K>(in_alt ? mk2 : mk, n, rblk, roff, rtmp, cur, uk, st, c->st);
    if (nblk) CK(cudaMemcpyAsync(&d, roff + nblk, 8, cudaMemcpyDeviceToHost, c->st));
    CK(cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, c->st));
    if (r.partial && pass == 0) CK(cudaMemcpyAsync(&rest, os_lb, 8, cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    if (e & ERR_SPIN_TIMEOUT) return ctx_fail(c, GKC_ERR_DEVICE_TIMEOUT, "sort look-back timed out");
    if (!rest || pass) break;
    in_alt = sort_pairs_rest<K>(r, rest, mk, mk2, mv, mv2, nd, n, 2 * c->ck, os, c->st, &launches);
  }
  const uint32_t *sv = in_alt ? mv2 : mv;
  if (d) k_run_sums<<<grid, 256, 0, c->st>>>(sv, st, d, n, us);
  uint64_t hb[2] = {0, d};
  CK(cudaMemcpyAsync(bo, hb, 16, cudaMemcpyHostToDevice, c->st));
  CK(cudaStreamSynchronize(c->st));
  *nbins_out = 1;
  return keep_range<K>(c, uk, us, bo, 1, d, lo, hi, n_out);
}

gkc_status gkc_count_output(gkc_ctx *c, uint32_t min_count, uint32_t max_count, int merged, uint64_t *n_out,
                            uint64_t *bin_off, uint64_t *keys, uint32_t *counts) {
  if (!c || !n_out) return GKC_ERR_INVALID_ARG;
  if (!c->have_count) return ctx_fail(c, GKC_ERR_INVALID_ARG, "no count result in the context");
  if (min_count > max_count) return ctx_fail(c, GKC_ERR_INVALID_ARG, "min_count > max_count");
  cudaSetDevice(c->dev);
  const int kw = c->cv.key_words;
  const bool same = c->have_out && c->out_gen == c->count_gen && c->out_min == min_count &&
                    c->out_max == max_count && c->out_merged == merged;
  if (!same) {
    uint64_t n = 0;
    uint32_t nb = 0;
    gkc_status s = kw == 1 ? count_output_t<uint64_t>(c, min_count, max_count, merged, &n, &nb)
                           : count_output_t<u128>(c, min_count, max_count, merged, &n, &nb);
    if (s != GKC_OK) return s;
    c->have_out = true;
    c->out_gen = c->count_gen;
    c->out_min = min_count;
    c->out_max = max_count;
    c->out_merged = merged;
    c->out_n = n;
    c->out_nbins = nb;
  }
  *n_out = c->out_n;
  const uint64_t n = c->out_n;
  if (bin_off) CK(cudaMemcpy(bin_off, c->bufs["flt_bin_off"].p, 8 * (c->out_nbins + 1), cudaMemcpyDeviceToHost));
  if (keys && n) CK(cudaMemcpy(keys, c->bufs["flt_keys"].p, 8 * kw * n, cudaMemcpyDeviceToHost));
  if (counts && n) CK(cudaMemcpy(counts, c->bufs["flt_counts"].p, 4 * n, cudaMemcpyDeviceToHost));
  return GKC_OK;
}
