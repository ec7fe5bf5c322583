// Per-window outputs over the read CSR:
//  * gkc_minimizers_device: the canonical minimizer of every k-window with the
//    position of the selected p-mer inside the window and its strand.  The
//    reference declares these outputs (d_mm_pos / d_mm_strand,
//    gkc_cuda.cu:159-160; CountTask::StoreMinimizerPos, gkc_cuda.hpp:50) but
//    never fills them; the definition here is the rightmost p-mer whose
//    passing forward or reverse-complement value equals the window's
//    minimizer (the ">=" updates at gkc_cuda.cu:283-284 let later candidates
//    win ties), strand -1 for a palindromic p-mer, 1 for the reverse
//    complement, 0 forward.
//  * gkc_subsample_positions_device: the canonical k-mers whose window
//    minimizer % mod == 0, each with the ascending list of its window starts
//    (README.md:16 use case; no reference code).
// Windows are indexed by their first byte's position in d_reads; a window
// that does not lie inside one read is invalid.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "ctx.h"
#include "kernels.h"
#include "minimizer.cuh"
#include "onesweep.h"
#include "tile.cuh"

namespace gkc {

// Bit i set for every read start offs[r] (r <= n_reads, so the end of the
// last read is marked too).  Offsets past n_bytes are flagged, not written.
__global__ void k_window_starts(const uint64_t *offs, uint64_t n_reads, uint64_t n_bytes,
                                uint32_t *bits, uint32_t *err) {
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r <= n_reads;
       r += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t pos = offs[r];
    if (pos > n_bytes || (r > 0 && offs[r - 1] > pos)) {
      atomicOr(err, ERR_BAD_READ);
      continue;
    }
    atomicOr(&bits[pos >> 5], 1u << (pos & 31));
  }
}

// Minimizer (x), position (y, lowest byte) and strand (the byte above) of
// tile window l, inside a read.
GKC_DEV uint2 window_min_pos(const TileBases &S, int l, int k, int p, int filter) {
  const WindowBases b = window_bases(S, l);
  const uint32_t mm = exact_minimizer(b, k, p, filter);
  const uint32_t M = 0xFFFFFFFFu >> (32 - 2 * p);
  uint32_t f = 0, r = 0;
  int bpos = 255, bstr = 0, at = 1 - p;
  each_base(b, 0, k, [&](uint32_t c, bool bad) {  // a byte that is no base counts as T here, and so does its complement
    f = ((f << 2) | c) & M;
    r = (r >> 2) | ((bad ? 3u : 3u - c) << (2 * p - 2));
    if (at >= 0 && (f == mm || r == mm)) {
      const bool mf = f == mm && mm_filter(f, p, filter), mr = r == mm && mm_filter(r, p, filter);
      if (mf || mr) {
        bpos = at;
        bstr = (f == r) ? -1 : (mr ? 1 : 0);
      }
    }
    at++;
  });
  return make_uint2(mm, (uint32_t)bpos | (uint32_t)(uint8_t)bstr << 8);
}

struct WinArgs {
  const uint8_t *reads;
  uint64_t n_bytes;
  int aligned16;
  const uint64_t *offs;
  uint64_t n_reads;
  const uint32_t *bits;  // read starts
  uint64_t bit_words;
  int k, p, filter;
  int strip;             // windows per warp (window_strip)
};

// The lane's 16 windows of the warp's strip from tile window P0 on: bit i of
// *vw and *tw: window i lies in a read; it touches a byte that is no base.
GKC_DEV void lane_valid(const TileBases &S, const WinArgs &a, int64_t G0, int64_t lo, int64_t hi, int P0, int strip,
                        uint32_t *vw, uint32_t *tw) {
  const int x = TL_W * (threadIdx.x & 31), P = P0 + x;
  *vw = *tw = 0;
  if (x < strip) {
    tile_valid(S, P >> 5, G0, lo, hi, a.k, vw, tw);
    *vw = (*vw >> (P & 31)) & 0xFFFFu;
    *tw = (*tw >> (P & 31)) & *vw;
  }
}

// Minimizer, position and strand of every window, one tile per CTA turn; a
// lane's 16 windows are written as whole 16-byte words.  Windows with a byte
// that is no base follow the exact per-window rule, and so do those whose
// minimizer is the largest p-mer value (it may stand for "none passed", which
// has no position).
__global__ void __launch_bounds__(TL_NT, 3) k_window_minimizers(WinArgs a, uint32_t *mm, uint8_t *pos,
                                                                int8_t *strand, int aligned) {
  __shared__ TileBases S;
  __shared__ uint16_t redo[TL_WARPS][TL_REDO];
  const uint64_t hi = a.offs[a.n_reads];
  const int64_t lo = (int64_t)a.offs[0], end = hi <= a.n_bytes ? (int64_t)hi : 0;
  const int strip = a.strip, NW = TL_WARPS * strip;
  const uint64_t n_tiles = (a.n_bytes + NW - 1) / NW;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, P0 = warp * strip, P = P0 + TL_W * lane;
  const uint32_t M = 0xFFFFFFFFu >> (32 - 2 * a.p);
  uint4 bytes = make_uint4(0u, 0u, 0u, 0u);
  if (blockIdx.x < n_tiles && threadIdx.x < TL_GROUPS)
    bytes = tile_fetch(a.reads, a.n_bytes, a.aligned16, (int64_t)blockIdx.x * NW, threadIdx.x);
  for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t G0 = (int64_t)(tile * NW);
    tile_store(S, bytes, a.bits, a.bit_words, G0);
    __syncthreads();
    if (tile + gridDim.x < n_tiles && threadIdx.x < TL_GROUPS)
      bytes = tile_fetch(a.reads, a.n_bytes, a.aligned16, (int64_t)((tile + gridDim.x) * NW), threadIdx.x);
    uint32_t vw, tw, m[TL_W] = {}, q[TL_W] = {};
    lane_valid(S, a, G0, lo, end, P0, strip, &vw, &tw);
    if (__any_sync(0xffffffffu, vw != 0u)) tile_minima<true>(S, P0, a.k, a.p, a.filter, m, q);
#pragma unroll
    for (int i = 0; i < TL_W; i++) {
      if (m[i] == M) tw |= vw & (1u << i);
      const uint32_t code = q[i] & 3u;
      q[i] = ((q[i] >> 2) - (uint32_t)(P + i)) | (code == 2u ? 0xFF00u : code << 8);  // strand byte, position byte
    }
#pragma unroll
    for (int i = 0; i < TL_W; i++)
      if (!((vw >> i) & 1u)) {
        m[i] = 0xFFFFFFFFu;
        q[i] = 255u;
      }
    const uint64_t at = (uint64_t)G0 + P;
    if (TL_W * lane < strip) {
      if (aligned && at + TL_W <= a.n_bytes) {
        uint4 *om = reinterpret_cast<uint4 *>(mm + at);
#pragma unroll
        for (int x = 0; x < 4; x++) om[x] = make_uint4(m[4 * x], m[4 * x + 1], m[4 * x + 2], m[4 * x + 3]);
        uint32_t pw[4], sw[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
          const uint32_t lo2 = __byte_perm(q[4 * x], q[4 * x + 1], 0x5140), hi2 = __byte_perm(q[4 * x + 2], q[4 * x + 3], 0x5140);
          pw[x] = __byte_perm(lo2, hi2, 0x5410);  // bytes: position 0, 1 (low halves of lo2), 2, 3
          sw[x] = __byte_perm(lo2, hi2, 0x7632);
        }
        if (pos) *reinterpret_cast<uint4 *>(pos + at) = make_uint4(pw[0], pw[1], pw[2], pw[3]);
        if (strand) *reinterpret_cast<uint4 *>(strand + at) = make_uint4(sw[0], sw[1], sw[2], sw[3]);
      } else {
#pragma unroll
        for (int i = 0; i < TL_W; i++)
          if (at + i < a.n_bytes) {
            mm[at + i] = m[i];
            if (pos) pos[at + i] = (uint8_t)q[i];
            if (strand) strand[at + i] = (int8_t)(q[i] >> 8);
          }
      }
    }
    if (__any_sync(0xffffffffu, tw != 0u)) {  // over what was written above: the lanes' registers are free again
      uint32_t rank;
      const uint32_t total = tile_list(tw, P0, redo[warp], &rank);  // its barrier orders the writes
      for (uint32_t r = lane; r < total; r += 32) {
        const int l = redo[warp][r];
        const uint2 w = window_min_pos(S, l, a.k, a.p, a.filter);
        mm[G0 + l] = w.x;
        if (pos) pos[G0 + l] = (uint8_t)w.y;
        if (strand) strand[G0 + l] = (int8_t)(w.y >> 8);
      }
    }
    __syncthreads();  // before the next tile's bases
  }
}

// ---- subsampling: windows whose minimizer % mod == 0, in window order ----

constexpr int SUB_NT = TL_NT;
constexpr int SUB_WORDS = TL_NW_MAX / 32;  // selection words kept per tile

// Selection bitmap (SUB_WORDS words a tile) and count of every tile.
__global__ void __launch_bounds__(SUB_NT, 4) k_sub_flags(WinArgs a, uint32_t mod, uint32_t *sel,
                                                         unsigned long long *tile_cnt, uint64_t n_tiles) {
  __shared__ TileBases S;
  __shared__ RedoArea redo[TL_WARPS];
  __shared__ uint32_t cnt[TL_WARPS];
  const uint64_t hi = a.offs[a.n_reads];
  const int64_t lo = (int64_t)a.offs[0], end = hi <= a.n_bytes ? (int64_t)hi : 0;
  const int strip = a.strip, NW = TL_WARPS * strip;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, P0 = warp * strip, P = P0 + TL_W * lane;
  for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t G0 = (int64_t)(tile * NW);
    uint4 bytes = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < TL_GROUPS) bytes = tile_fetch(a.reads, a.n_bytes, a.aligned16, G0, threadIdx.x);
    tile_store(S, bytes, a.bits, a.bit_words, G0);
    __syncthreads();
    uint32_t vw, tw, m[TL_W], none[1];
    lane_valid(S, a, G0, lo, end, P0, strip, &vw, &tw);
    tile_minima<false>(S, P0, a.k, a.p, a.filter, m, none);
    if (__any_sync(0xffffffffu, tw != 0u))
      tile_redo(S, tw, P0, redo[warp], a.k, a.p, a.filter, m);
    uint32_t f = 0;
#pragma unroll
    for (int i = 0; i < TL_W; i++)
      if (m[i] % mod == 0u) f |= 1u << i;
    f &= vw;
    const uint32_t other = __shfl_down_sync(0xffffffffu, f, 1);
    if (TL_W * lane < strip && !(lane & 1)) sel[tile * SUB_WORDS + (P >> 5)] = f | (other << 16);
    const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(f));
    if (lane == 0) cnt[warp] = c;
    __syncthreads();  // also before the next tile's bases
    if (threadIdx.x == 0) {
      uint32_t s = 0;
      for (int x = 0; x < TL_WARPS; x++) s += cnt[x];
      tile_cnt[tile] = s;
    }
  }
}

// The 2k bits of the k bases from tile base l on (a byte that is no base
// counts as T, as in the packed superkmers).
template <typename K>
GKC_DEV K tile_kmer(const TileBases &S, int l, int k) {
  const int j = l >> 4;
  const uint32_t sh = 2 * (uint32_t)(l & 15);
  uint32_t w[sizeof(K) / 4 + 1];
#pragma unroll
  for (int t = 0; t <= (int)sizeof(K) / 4; t++) w[t] = S.pk[j + t].x;
  K x = 0;
#pragma unroll
  for (int t = 0; t < (int)sizeof(K) / 4; t++) x = (x << 32) | (K)__funnelshift_l(w[t + 1], w[t], sh);
  return x >> (8 * (int)sizeof(K) - 2 * k);
}

// Writes (canonical key, window start) of the selected windows in window
// order: a warp lists the selected windows of its words of the tile, then each
// lane takes the k-mer of one of them from the tile's packed bases, so that
// full warps cut and compare k-mers (13.9 M of 56 M windows at k 63: 171
// us; each lane its own window, a quarter of them selected, 203).
template <typename K>
__global__ void __launch_bounds__(SUB_NT) k_sub_write(WinArgs a, const uint32_t *sel, const uint64_t *tile_off,
                                                      K *keys, uint32_t *posv, uint64_t n_tiles) {
  __shared__ TileBases S;
  __shared__ uint32_t cnt[TL_WARPS];
  __shared__ uint16_t list[TL_NW_MAX];
  const int strip = a.strip, NW = TL_WARPS * strip, words = strip / 32;  // at most 15 words a warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w0 = warp * words;
  for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t G0 = (int64_t)(tile * NW);
    uint4 bytes = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < TL_GROUPS) bytes = tile_fetch(a.reads, a.n_bytes, a.aligned16, G0, threadIdx.x);
    const uint32_t mine = lane < words ? sel[tile * SUB_WORDS + w0 + lane] : 0u;
    tile_store(S, bytes, a.bits, a.bit_words, G0);
    const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(mine));
    if (lane == 0) cnt[warp] = c;
    __syncthreads();
    uint64_t o = tile_off[tile];
    for (int x = 0; x < warp; x++) o += cnt[x];
    uint16_t *L = list + 32 * w0;
    uint32_t n = 0;
    for (int r = 0; r < words; r++) {
      const uint32_t f = __shfl_sync(0xffffffffu, mine, r);
      if ((f >> lane) & 1u) L[n + __popc(f & ((1u << lane) - 1u))] = (uint16_t)(32 * (w0 + r) + lane);
      n += __popc(f);
    }
    __syncwarp();
    for (uint32_t i = lane; i < n; i += 32) {
      const int l = L[i];
      const K x = tile_kmer<K>(S, l, a.k), rc = revcomp_k<K>(x, a.k);
      keys[o + i] = x < rc ? x : rc;
      posv[o + i] = (uint32_t)(G0 + l);
    }
    __syncthreads();  // before the next tile's bases
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

static gkc_status check_window_args(gkc_ctx *c, const gkc_params *prm, const char *d_reads,
                                    uint64_t n_bytes, const uint64_t *d_offs, int kmax) {
  if (!c || !prm) return GKC_ERR_INVALID_ARG;
  if (prm->k < 1 || prm->k > kmax || prm->p < 3 || prm->p > 16 || prm->p > prm->k)
    return ctx_fail(c, GKC_ERR_INVALID_ARG, "need 3 <= p <= min(k, 16)");
  if (prm->hpc) return ctx_fail(c, GKC_ERR_INVALID_ARG, "run gkc_hpc_device first; hpc must be 0 here");
  if (n_bytes >= (1ull << 32)) return ctx_fail(c, GKC_ERR_INVALID_ARG, "positions are 32-bit");
  if (n_bytes && (!d_reads || !d_offs)) return ctx_fail(c, GKC_ERR_INVALID_ARG, "null input");
  return GKC_OK;
}

static gkc_status mark_starts(gkc_ctx *c, const uint64_t *d_offs, uint64_t n_reads, uint64_t n_bytes,
                              uint32_t **bits_out, uint32_t **err_out) {
  const uint64_t words = (n_bytes + 1) / 32 + 3;
  WS(bits, uint32_t, "win_bits", words);
  WS(err, uint32_t, "win_err", 4);
  CK(cudaMemsetAsync(bits, 0, words * 4, c->st));
  CK(cudaMemsetAsync(err, 0, 16, c->st));
  k_window_starts<<<(unsigned)std::min<uint64_t>((n_reads + 256) / 256, 65535), 256, 0, c->st>>>(
      d_offs, n_reads, n_bytes, bits, err);
  CK(cudaPeekAtLastError());
  *bits_out = bits;
  *err_out = err;
  return GKC_OK;
}

// Windows per warp: what a warp can take, less where that leaves SMs without a
// tile (15 kB of reads with 3% N, k 31: 112 us with full strips, 48 so).
static int window_strip(const gkc_ctx *c, const gkc_params *prm, uint64_t n_bytes) {
  int strip = tile_strip(prm->k - prm->p + 1);
  while (strip > 64 && n_bytes < (uint64_t)TL_WARPS * strip * c->n_sms) strip = strip / 2 & ~31;
  return strip;
}

static WinArgs win_args(const gkc_ctx *c, const gkc_params *prm, const uint8_t *reads, uint64_t n_bytes,
                        const uint64_t *offs, uint64_t n_reads, const uint32_t *bits) {
  return WinArgs{reads,  n_bytes, ((uintptr_t)reads % 16) == 0, offs,   n_reads, bits, (n_bytes + 1) / 32 + 3,
                 prm->k, prm->p,  c->filter, window_strip(c, prm, n_bytes)};
}

static gkc_status read_err(gkc_ctx *c, const uint32_t *err) {
  uint32_t e = 0;
  CK(cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  if (e & ERR_BAD_READ) return ctx_fail(c, GKC_ERR_INVALID_ARG, "read offsets decrease or pass n_bytes");
  if (e & ERR_SPIN_TIMEOUT) return ctx_fail(c, GKC_ERR_DEVICE_TIMEOUT, "sort look-back timed out");
  return GKC_OK;
}

gkc_status gkc_minimizers_device(gkc_ctx *c, const gkc_params *prm, const char *d_reads,
                                 uint64_t n_bytes, const uint64_t *d_offs, uint64_t n_reads,
                                 uint32_t *d_minimizer, uint8_t *d_pos, int8_t *d_strand) {
  gkc_status s = check_window_args(c, prm, d_reads, n_bytes, d_offs, 64);
  if (s != GKC_OK) return s;
  if (n_bytes == 0) return GKC_OK;
  if (!d_minimizer) return ctx_fail(c, GKC_ERR_INVALID_ARG, "null minimizer output");
  cudaSetDevice(c->dev);
  uint32_t *bits, *err;
  s = mark_starts(c, d_offs, n_reads, n_bytes, &bits, &err);
  if (s != GKC_OK) return s;
  const int nw = TL_WARPS * window_strip(c, prm, n_bytes);
  const uint64_t tiles = (n_bytes + nw - 1) / nw;
  const int aligned = (((uintptr_t)d_minimizer | (uintptr_t)d_pos | (uintptr_t)d_strand) & 15) == 0;
  k_window_minimizers<<<(unsigned)std::min<uint64_t>(tiles, (uint64_t)c->n_sms * 3), TL_NT, 0, c->st>>>(
      win_args(c, prm, reinterpret_cast<const uint8_t *>(d_reads), n_bytes, d_offs, n_reads, bits), d_minimizer, d_pos,
      d_strand, aligned);
  CK(cudaPeekAtLastError());
  return read_err(c, err);
}

template <typename K>
static gkc_status subsample_t(gkc_ctx *c, const gkc_params *prm, uint32_t mod, const uint8_t *reads,
                              uint64_t n_bytes, const uint64_t *d_offs, uint64_t n_reads,
                              gkc_poslist_view *out) {
  uint32_t *bits, *err;
  gkc_status s = mark_starts(c, d_offs, n_reads, n_bytes, &bits, &err);
  if (s != GKC_OK) return s;
  const int nw = TL_WARPS * window_strip(c, prm, n_bytes);
  const uint64_t tiles = (n_bytes + nw - 1) / nw;
  WS(sel, uint32_t, "win_sel", tiles * SUB_WORDS + 1);
  WS(tcnt, unsigned long long, "win_tile_cnt", tiles + 1);
  WS(toff, uint64_t, "win_tile_off", tiles + 2);
  WS(stmp, uint64_t, "win_scan_tmp", scan_u64_tmp_words(tiles + 1) + 8);
  k_sub_flags<<<(unsigned)std::min<uint64_t>(tiles, (uint64_t)c->n_sms * 4), SUB_NT, 0, c->st>>>(
      win_args(c, prm, reads, n_bytes, d_offs, n_reads, bits), mod, sel, tcnt, tiles);
  scan_u64(tcnt, toff, tiles, stmp, c->st);
  CK(cudaPeekAtLastError());
  uint64_t n = 0;
  CK(cudaMemcpyAsync(&n, toff + tiles, 8, cudaMemcpyDeviceToHost, c->st));
  s = read_err(c, err);  // synchronises
  if (s != GKC_OK) return s;
  WS(keys, K, "win_keys", n + 16);
  WS(alt, K, "win_keys_alt", n + 16);
  WS(pos, uint32_t, "win_pos", n + 16);
  WS(palt, uint32_t, "win_pos_alt", n + 16);
  WS(out_keys, K, "win_out_keys", n + 16);
  WS(pos_off, uint64_t, "win_pos_off", n + 2);
  if (n) {
    k_sub_write<K><<<(unsigned)std::min<uint64_t>(tiles, (uint64_t)c->n_sms * 8), SUB_NT, 0, c->st>>>(
        win_args(c, prm, reads, n_bytes, d_offs, n_reads, bits), sel, toff, keys, pos, tiles);
    CK(cudaPeekAtLastError());
    WS(os_hist, unsigned long long, "win_os_hist", 16 * 256);
    WS(os_lb, unsigned long long, "win_os_lookback", onesweep_lookback_words(n + 1));
    WS(os_ticket, unsigned long long, "win_os_ticket", 2);
    OnesweepScratch os{os_hist, os_lb, os_ticket, err, c->n_sms * 4};
    // the selected count, on the device, for the sort
    const uint64_t *n_dev = toff + tiles;
    uint32_t launches = 0;
    const PairsStatus r = sort_pairs<K>(keys, alt, pos, palt, n_dev, n, 2 * prm->k, os, c->st, &launches);
    int in_alt = r.result_in_alt;
    // distinct keys and their first indices (= the position-list offsets)
    const uint64_t nblk = rle_block_count(n);
    WS(rblk, unsigned long long, "win_rle_blk", nblk + 1);
    WS(roff, uint64_t, "win_rle_off", nblk + 2);
    WS(rtmp, uint64_t, "win_rle_tmp", scan_u64_tmp_words(nblk + 1) + 8);
    WS(cur, unsigned long long, "win_cursor", 2);
    uint64_t nd = 0;
    unsigned long long rest = 0;
    for (int pass = 0; pass < 2; pass++) {  // once more where long runs were left
      CK(cudaMemsetAsync(cur, 0, 16, c->st));
      rle_runs<K>(in_alt ? alt : keys, n, rblk, roff, rtmp, cur, out_keys, pos_off, c->st);
      CK(cudaPeekAtLastError());
      CK(cudaMemcpyAsync(&nd, roff + nblk, 8, cudaMemcpyDeviceToHost, c->st));
      if (r.partial && pass == 0) CK(cudaMemcpyAsync(&rest, os_lb, 8, cudaMemcpyDeviceToHost, c->st));
      s = read_err(c, err);
      if (s != GKC_OK) return s;
      if (!rest || pass) break;
      in_alt = sort_pairs_rest<K>(r, rest, keys, alt, pos, palt, n_dev, n, 2 * prm->k, os, c->st, &launches);
    }
    const uint32_t *sp = in_alt ? palt : pos;
    uint64_t nn = n;
    CK(cudaMemcpyAsync(pos_off + nd, &nn, 8, cudaMemcpyHostToDevice, c->st));
    CK(cudaStreamSynchronize(c->st));
    out->n_distinct = nd;
    out->positions = sp;
  } else {
    uint64_t zero = 0;
    CK(cudaMemcpyAsync(pos_off, &zero, 8, cudaMemcpyHostToDevice, c->st));
    CK(cudaStreamSynchronize(c->st));
    out->n_distinct = 0;
    out->positions = pos;
  }
  out->n_positions = n;
  out->key_words = sizeof(K) / 8;
  out->keys = reinterpret_cast<const uint64_t *>(out_keys);
  out->pos_off = pos_off;
  return GKC_OK;
}

gkc_status gkc_subsample_positions_device(gkc_ctx *c, const gkc_params *prm, uint32_t mod,
                                          const char *d_reads, uint64_t n_bytes,
                                          const uint64_t *d_offs, uint64_t n_reads,
                                          gkc_poslist_view *out) {
  gkc_status s = check_window_args(c, prm, d_reads, n_bytes, d_offs, 64);
  if (s != GKC_OK) return s;
  if (!out || mod == 0) return ctx_fail(c, GKC_ERR_INVALID_ARG, "need mod >= 1 and an output view");
  memset(out, 0, sizeof(*out));
  out->key_words = prm->k <= 32 ? 1 : 2;
  if (n_bytes == 0) return GKC_OK;
  cudaSetDevice(c->dev);
  const uint8_t *reads = reinterpret_cast<const uint8_t *>(d_reads);
  if (prm->k <= 32) return subsample_t<uint64_t>(c, prm, mod, reads, n_bytes, d_offs, n_reads, out);
  return subsample_t<u128>(c, prm, mod, reads, n_bytes, d_offs, n_reads, out);
}
