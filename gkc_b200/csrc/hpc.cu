// Homopolymer compression (HPC): collapse maximal runs of equal bytes in each
// read, keeping for every kept base its in-read original position
// (reference: GPU_HPCEncoding, gkc_cuda.cu:164-192, with the per-read start
// index of :180).  The compacted reads form a new contiguous CSR.
//
// Reads are contiguous, so this is one compaction of all bytes: a byte is kept
// when a read starts there or it differs from the byte before.  Tiles of 8192
// bytes, 16 a thread: flags (compared four bytes at a time) as a bitmap with
// each word's count in its tile, a scan of the tiles, then the kept bytes and
// positions put together in shared memory and written as one run per tile.
// Bound by HBM in the model (the bytes twice, 1 + 4 bytes per kept base); a
// warp per read with one byte a lane, runs by ballot, took 1.46 ms for 200 M
// bases of 8 kbp reads (imbalance and byte loads), these four 0.55 ms.
#include <algorithm>

#include "common.cuh"
#include "ctx.h"
#include "kernels.h"

namespace gkc {

constexpr int HP_NT = 512;
constexpr int HP_TILE = HP_NT * 16;
constexpr int HP_WORDS = HP_TILE / 32;

struct HpcArgs {
  const uint8_t *reads;
  uint64_t n_bytes;
  int aligned16;
  const uint64_t *offs;
  uint64_t n_reads;
  const uint32_t *starts;       // bit i: a read starts at byte i
  uint32_t *flags;              // bit i: byte i is kept; whole tiles
  uint16_t *pre;                // kept bytes of the tile before each flag word
  unsigned long long *tile_cnt;
  const uint64_t *tile_off;
  uint64_t n_tiles;
  uint8_t *out;
  uint64_t *out_offs;
  int32_t *orig;                // may be null
};

// One bit per read start inside [offs[0], offs[n]).
__global__ void k_hpc_starts(HpcArgs a, uint32_t *starts, unsigned long long *stamp) {
  stamp_now(stamp);
  const uint64_t lo = a.offs[0], hi = min(a.offs[a.n_reads], a.n_bytes);
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < a.n_reads;
       r += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t pos = a.offs[r];
    if (pos >= lo && pos < hi) atomicOr(&starts[pos >> 5], 1u << (pos & 31));
  }
}

// The thread's 16 bytes; bytes past n_bytes read as 0.
GKC_DEV uint4 hpc_load(const HpcArgs &a, uint64_t i) {
  if (a.aligned16 && i + 16 <= a.n_bytes) return __ldg(reinterpret_cast<const uint4 *>(a.reads + i));
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  for (int t = 0; t < 16; t++)
    if (i + t < a.n_bytes) w[t >> 2] |= (uint32_t)a.reads[i + t] << (8 * (t & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void __launch_bounds__(HP_NT) k_hpc_flags(HpcArgs a) {
  __shared__ uint32_t tmp[64];
  const uint64_t lo = a.offs[0], hi = min(a.offs[a.n_reads], a.n_bytes);
  for (uint64_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
    const uint64_t i = tile * HP_TILE + 16 * (uint64_t)threadIdx.x;
    const uint4 v = hpc_load(a, i);
    uint32_t prev = __shfl_up_sync(0xffffffffu, v.w >> 24, 1);
    if ((threadIdx.x & 31) == 0) prev = i > 0 && i - 1 < a.n_bytes ? a.reads[i - 1] : 0u;
    const uint32_t w[5] = {prev << 24, v.x, v.y, v.z, v.w};
    uint32_t f = 0;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const uint32_t z = w[t + 1] ^ __funnelshift_l(w[t], w[t + 1], 8);  // against the byte before
      const uint32_t nz = (((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z) & 0x80808080u;
      f |= (((nz >> 7) * 0x01020408u) >> 24) << (4 * t);                 // first byte in the lowest bit
    }
    if (i < a.n_bytes) f |= (a.starts[i >> 5] >> (i & 31)) & 0xFFFFu;
    // bytes inside the reads only
    const uint64_t b = lo > i ? lo - i : 0, e = hi > i ? hi - i : 0;
    f = b < 16 && e > b ? f & (0xFFFFu << b) & (e < 16 ? (1u << e) - 1u : 0xFFFFu) : 0u;
    uint32_t total;
    const uint32_t before = block_exclusive_scan<HP_NT>(__popc(f), tmp, &total);
    const uint32_t other = __shfl_down_sync(0xffffffffu, f, 1);
    if ((threadIdx.x & 1) == 0) {
      const uint64_t word = tile * HP_WORDS + (threadIdx.x >> 1);
      a.flags[word] = f | (other << 16);
      a.pre[word] = (uint16_t)before;
    }
    if (threadIdx.x == 0) a.tile_cnt[tile] = total;
  }
}

// Compressed offset of every read: the kept bytes before its first one.
GKC_DEV void hpc_offsets(const HpcArgs &a) {
  const uint64_t lo = a.offs[0], hi = min(a.offs[a.n_reads], a.n_bytes);
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r <= a.n_reads;
       r += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t pos = a.offs[r];
    uint64_t o;
    if (pos <= lo) o = 0;
    else if (pos >= hi) o = a.tile_off[a.n_tiles];
    else o = a.tile_off[pos / HP_TILE] + a.pre[pos >> 5] + __popc(a.flags[pos >> 5] & ((1u << (pos & 31)) - 1u));
    a.out_offs[r] = o;
  }
}

__global__ void __launch_bounds__(256) k_hpc_offsets(HpcArgs a) { hpc_offsets(a); }

// OFFSETS: the reads' offsets as well, where a launch costs more than what they
// take from this kernel's registers (one tile a CTA: 15 kB 67 -> 63 us; 150 M
// bytes, many tiles: 494 -> 604).
template <bool OFFSETS>
__global__ void __launch_bounds__(HP_NT) k_hpc_write(HpcArgs a) {
  __shared__ uint8_t sb[HP_TILE];
  __shared__ int32_t so[HP_TILE];
  __shared__ unsigned long long wlast[HP_NT / 32];
  __shared__ unsigned long long first;  // start of the read that holds the tile's first byte
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint64_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
    const uint64_t t0 = tile * HP_TILE, i = t0 + 16 * (uint64_t)threadIdx.x;
    const uint4 v = hpc_load(a, i);
    const uint64_t word = tile * HP_WORDS + (threadIdx.x >> 1);
    const uint32_t whole = a.flags[word];
    uint32_t f = threadIdx.x & 1 ? whole >> 16 : whole & 0xFFFFu;
    uint32_t at = a.pre[word] + (threadIdx.x & 1 ? __popc(whole & 0xFFFFu) : 0);
    const uint32_t s = a.orig && i < a.n_bytes ? (a.starts[i >> 5] >> (i & 31)) & 0xFFFFu : 0u;
    uint64_t start = 0;  // of the read that holds the thread's first byte
    if (a.orig) {
      // the last read start up to the thread's own bytes, plus one (0: none)
      unsigned long long x = s ? i + 32 - __clz((int)s) : 0ull;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d && y > x) x = y;
      }
      if (lane == 31) wlast[warp] = x;
      if (warp == 0) {  // the last offset up to the tile's first byte
        uint64_t l = 0, h = a.n_reads;
        while (l < h) {
          const uint64_t step = (h - l) / 32 + 1, p = l + lane * step;
          const uint32_t le = __ballot_sync(0xffffffffu, p <= h && __ldg(a.offs + p) <= t0);
          if (!le) break;
          l += (uint64_t)(31 - __clz((int)le)) * step;
          h = min(h, l + step - 1);
        }
        if (lane == 0) first = a.offs[l];
      }
      x = __shfl_up_sync(0xffffffffu, x, 1);
      if (lane == 0) x = 0;
      __syncthreads();
      for (int w = 0; w < warp; w++) x = wlast[w] > x ? wlast[w] : x;
      start = x ? x - 1 : first;
    }
    const uint32_t b[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int t = 0; t < 16; t++) {
      if ((s >> t) & 1u) start = i + t;
      if ((f >> t) & 1u) {
        sb[at] = (uint8_t)(b[t >> 2] >> (8 * (t & 3)));
        if (a.orig) so[at] = (int32_t)(i + t - start);
        at++;
      }
    }
    __syncthreads();
    const uint64_t o = a.tile_off[tile], n = a.tile_off[tile + 1] - o;
    for (uint64_t x = threadIdx.x; x < n; x += HP_NT)
      if (a.orig) a.orig[o + x] = so[x];
    // bytes up to the first word boundary, whole words, the rest
    const uint64_t lead = min(n, (uint64_t)((0ull - (reinterpret_cast<uintptr_t>(a.out) + o)) & 3ull));
    if (threadIdx.x < lead) a.out[o + threadIdx.x] = sb[threadIdx.x];
    const uint64_t nw = (n - lead) / 4;
    uint32_t *ow = reinterpret_cast<uint32_t *>(a.out + o + lead);
    for (uint64_t x = threadIdx.x; x < nw; x += HP_NT) {
      const uint8_t *q = sb + lead + 4 * x;
      ow[x] = (uint32_t)q[0] | (uint32_t)q[1] << 8 | (uint32_t)q[2] << 16 | (uint32_t)q[3] << 24;
    }
    for (uint64_t x = lead + 4 * nw + threadIdx.x; x < n; x += HP_NT) a.out[o + x] = sb[x];
    __syncthreads();
  }
  if (OFFSETS) hpc_offsets(a);
}

}  // namespace gkc

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

gkc_status hpc_enqueue(gkc_ctx *c, const uint8_t *reads, uint64_t n_bytes, const uint64_t *offs, uint64_t n_reads,
                       uint8_t *out, uint64_t *out_offs, int32_t *orig, unsigned long long *stamp) {
  using namespace gkc;
  const uint64_t tiles = std::max<uint64_t>(1, (n_bytes + HP_TILE - 1) / HP_TILE);
  // the bitmap of read starts; the partition's own, made afterwards, takes its place
  const uint64_t words = std::max((n_bytes + 1 + 31) / 32 + 2, tiles * HP_WORDS);
  WS(starts, uint32_t, "rs_bits", words);
  WS(flags, uint32_t, "hpc_flags", tiles * HP_WORDS);
  WS(pre, uint16_t, "hpc_pre", tiles * HP_WORDS);
  WS(cnt, unsigned long long, "hpc_tile_cnt", tiles + 1);
  WS(off, uint64_t, "hpc_tile_off", tiles + 2);
  WS(stmp, uint64_t, "hpc_scan_tmp", scan_u64_tmp_words(tiles + 1) + 8);
  const HpcArgs a{reads, n_bytes, ((uintptr_t)reads % 16) == 0, offs, n_reads, starts, flags, pre, cnt, off, tiles,
                  out, out_offs, orig};
  CK(cudaMemsetAsync(starts, 0, words * 4, c->st));
  const unsigned rgrid = (unsigned)std::min<uint64_t>((n_reads + 256) / 256, (uint64_t)c->n_sms * 16);
  k_hpc_starts<<<rgrid, 256, 0, c->st>>>(a, starts, stamp);
  k_hpc_flags<<<(unsigned)std::min<uint64_t>(tiles, (uint64_t)c->n_sms * 4), HP_NT, 0, c->st>>>(a);
  c->launches += 3 + scan_u64(cnt, off, tiles, stmp, c->st);
  const uint64_t most = (uint64_t)c->n_sms * 4;
  if (tiles <= most) {
    k_hpc_write<true><<<(unsigned)tiles, HP_NT, 0, c->st>>>(a);
  } else {
    k_hpc_write<false><<<(unsigned)most, HP_NT, 0, c->st>>>(a);
    k_hpc_offsets<<<rgrid, 256, 0, c->st>>>(a);
    c->launches++;
  }
  CK(cudaPeekAtLastError());
  return GKC_OK;
}

// Homopolymer compression alone: d_out_reads gets the compressed reads back
// to back, d_out_offs[n_reads+1] their CSR offsets (from 0), d_orig_pos (may
// be NULL) the in-read position of the first base of every run.
gkc_status gkc_hpc_device(gkc_ctx *c, const char *d_reads, uint64_t n_bytes, const uint64_t *d_offs,
                          uint64_t n_reads, char *d_out_reads, uint64_t *d_out_offs,
                          int32_t *d_orig_pos) {
  if (!c) return GKC_ERR_INVALID_ARG;
  if (!d_offs || !d_out_offs || (n_bytes && (!d_reads || !d_out_reads)))
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "null input or output");
  cudaSetDevice(c->dev);
  uint64_t ends[2] = {0, 0};
  CK(cudaMemcpyAsync(&ends[0], d_offs, 8, cudaMemcpyDeviceToHost, c->st));
  CK(cudaMemcpyAsync(&ends[1], d_offs + n_reads, 8, cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  if (ends[0] > ends[1] || ends[1] > n_bytes)
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "read offsets decrease or pass n_bytes");
  const gkc_status s = hpc_enqueue(c, reinterpret_cast<const uint8_t *>(d_reads), n_bytes, d_offs, n_reads,
                                   reinterpret_cast<uint8_t *>(d_out_reads), d_out_offs, d_orig_pos);
  if (s != GKC_OK) return s;
  CK(cudaStreamSynchronize(c->st));
  return GKC_OK;
}
