// Superkmer partitioning on the device.
//
// Semantics follow the reference's GPU_GenMinimizer / GPU_GenSKM /
// SKMStore::add_skms (gkc_cuda.cu:234-324, superkmers.hpp:167-186):
//   * every k-window of a read gets a canonical minimizer: the smallest
//     forward or reverse-complement p-mer that passes the filter, else 4^p-1;
//     windows touching a byte outside ACGTU follow the reference's exact
//     per-window update rule (including its 255-code smear);
//   * a superkmer is a maximal run of windows with equal minimizer value; its
//     bases are packed 2 bits per base, MSB first, N as T, byte aligned;
//   * its bin is minimizer % nbins.
// Reads shorter than k produce nothing.
//
// The fused kernel is persistent and tiled over the concatenated read bytes:
// the minimizers of a tile's windows stay in registers (tile.cuh), breaks are
// bitmaps of 32 windows a word, superkmers are compacted from them, and the
// packed bytes are written as coalesced 16-byte words.
#include "common.cuh"
#include "kernels.h"
#include "minimizer.cuh"
#include "tile.cuh"

namespace gkc {

constexpr int PT_NT = TL_NT;
constexpr int PT_PRE = 32;                       // local index of the first core window
constexpr int PT_HALO = 224;                     // windows after the core, to find superkmer ends
constexpr int PT_TMAX = TL_NW_MAX - PT_PRE - PT_HALO;  // core windows per tile (fewer where omega > 33)
constexpr int PT_STG = 6144;                     // packed bytes of a tile staged in shared memory
static_assert(PT_TMAX % 32 == 0 && kPartThreads == TL_NT, "whole words");
static_assert(kPartTile == TL_WARPS * 28 * TL_W - PT_PRE - PT_HALO, "the smallest tile");

struct PartSmem {
  TileBases t;
  uint32_t brkw[TL_NW_MAX / 32];   // bit i: window i starts a superkmer or lies in none
  union {
    struct {
      uint32_t smm[PT_TMAX];       // minimizer of each core superkmer
      uint32_t boff[PT_TMAX];      // its byte offset in the tile
      uint16_t spos[PT_TMAX];      // its first window
      uint16_t send[PT_TMAX];      // its end window (PT_EXT: ext_end)
    };
    RedoArea redo[TL_WARPS];       // before them
  };
  alignas(16) uint8_t stg[PT_STG]; // the tile's packed superkmers before they are written out (read as uint4)
  uint32_t scan_tmp[64];
  uint32_t lastmm[TL_WARPS], lastv[TL_WARPS], wcnt[TL_WARPS];
  int ext_end;                     // local end window of an extended last superkmer
  int halo;                        // a break lies in the halo
  unsigned long long base_skm, base_byte;
};
constexpr uint32_t PT_EXT = 0xFFFFu;

// Bound by instruction issue and the barriers between its phases: 256 threads
// and 64 registers, so that four CTAs on an SM overlap, the next tile's bytes
// loaded while this one is worked on.  900 M bases of 150 b reads (k 31, p 11)
// on a B200: 4.4 ms (ALU pipe 66 % of its cycles, 110 instructions for 32
// bases); every window searched from its bytes 8.7.
__global__ void __launch_bounds__(PT_NT, 4) k_partition(PartArgs a) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  PartSmem &S = *reinterpret_cast<PartSmem *>(smem_raw);
  stamp_now(a.stamp);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int k = a.k, p = a.p, omega = a.k - a.p + 1;
  if (a.nbytes_dev) a.nbytes = *a.nbytes_dev;
  const int strip = tile_strip(omega), NW = TL_WARPS * strip, T = NW - PT_PRE - PT_HALO;
  const uint64_t n_tiles = (a.nbytes + T - 1) / T;

  // per-CTA bin histograms (small bin counts only): superkmers, k-mers
  uint32_t *h_skm = reinterpret_cast<uint32_t *>(smem_raw + sizeof(PartSmem));
  uint32_t *h_km = h_skm + a.nbins_smem;
  for (int i = tid; i < 2 * a.nbins_smem; i += PT_NT) h_skm[i] = 0;

  uint4 bytes = make_uint4(0u, 0u, 0u, 0u);
  if (blockIdx.x < n_tiles && tid < TL_GROUPS)
    bytes = tile_fetch(a.reads, a.nbytes, a.aligned16, (int64_t)blockIdx.x * T - PT_PRE, tid);
  for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t G0 = (int64_t)(tile * T) - PT_PRE;  // global position of local 0 (32-aligned)
    tile_store(S.t, bytes, a.rs_bits, a.rs_words, G0);
    if (tid == 0) {
      S.ext_end = -1;
      S.halo = 0;
    }
    __syncthreads();
    if (tile + gridDim.x < n_tiles && tid < TL_GROUPS)
      bytes = tile_fetch(a.reads, a.nbytes, a.aligned16, (int64_t)((tile + gridDim.x) * T) - PT_PRE, tid);

    // ---- minimizers: lane l holds windows P .. P + 15 ----
    const int P0 = warp * strip, P = P0 + TL_W * lane;
    const bool own = TL_W * lane < strip;  // the strip's last lanes only feed the others
    uint32_t vw = 0, tw = 0;               // bit i: window P + i lies in a read; touches a byte that is no base
    if (own) {
      tile_valid(S.t, P >> 5, G0, 0, (int64_t)a.nbytes, k, &vw, &tw);
      vw = (vw >> (P & 31)) & 0xFFFFu;
      tw = (tw >> (P & 31)) & vw;
    }
    uint32_t m[TL_W], none[1];
    tile_minima<false>(S.t, P0, k, p, a.filter, m, none);
    if (__any_sync(0xffffffffu, tw != 0u))
      tile_redo(S.t, tw, P0, S.redo[warp], k, p, a.filter, m);
    if (P + TL_W == P0 + strip) {
      S.lastmm[warp] = m[TL_W - 1];
      S.lastv[warp] = vw >> 15;
    }
    __syncthreads();

    // ---- breaks and superkmer starts, 16 windows a lane ----
    uint32_t st;
    {
      uint32_t before = __shfl_up_sync(0xffffffffu, m[TL_W - 1], 1), pv = __shfl_up_sync(0xffffffffu, vw, 1) >> 15;
      if (lane == 0) {
        before = warp ? S.lastmm[warp - 1] : 0u;
        pv = warp ? S.lastv[warp - 1] : 0u;
      }
      uint32_t diff = 0;
#pragma unroll
      for (int i = 0; i < TL_W; i++) {
        if (m[i] != before) diff |= 1u << i;
        before = m[i];
      }
      const uint32_t rs = own ? S.t.rsw[P >> 5] >> (P & 31) : 0u;
      st = vw & (rs | diff | ~((vw << 1) | pv));
      const uint32_t brk = (st | ~vw) & 0xFFFFu;
      const uint32_t other = __shfl_down_sync(0xffffffffu, brk, 1);
      if (own && !(lane & 1)) S.brkw[P >> 5] = brk | (other << 16);
      if (own && P >= PT_PRE + T && brk) S.halo = 1;
    }
    if (P < PT_PRE || P >= PT_PRE + T) st = 0;  // core windows only (PT_PRE and T are multiples of 16)
    uint32_t wtot = __popc(st), at = wtot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, at, d);
      if (lane >= d) at += y;
    }
    at -= wtot;
    wtot = __shfl_sync(0xffffffffu, at + wtot, 31);
    if (lane == 0) S.wcnt[warp] = wtot;
    __syncthreads();
    uint32_t n_skm = 0;
#pragma unroll
    for (int x = 0; x < TL_WARPS; x++) {
      const uint32_t c = S.wcnt[x];
      if (x < warp) at += c;
      n_skm += c;
    }
#pragma unroll
    for (int i = 0; i < TL_W; i++)
      if ((st >> i) & 1u) {
        S.spos[at] = (uint16_t)(P + i);
        S.smm[at] = m[i];
        at++;
      }
    __syncthreads();

    // ---- the last superkmer runs past the tile where nothing breaks in the
    //      halo: the block looks for its end, a window a thread (16 M bases of
    //      8 kbp reads with a run of 1000 bases every 4000, k 31: 0.28 ms, with
    //      one thread going window by window 12.6; without such runs 0.15) ----
    if (!S.halo && n_skm > 0) {  // the same in every thread
      const uint32_t mv = S.smm[n_skm - 1];
      uint64_t x0 = (uint64_t)(G0 + NW);
      // a superkmer of more than 2^24 - 1 bases is refused wherever it ends
      const uint64_t most = (uint64_t)(G0 + S.spos[n_skm - 1]) + 0x1000000u;
      while (true) {
        const uint64_t x = x0 + tid;
        bool out = x >= a.nbytes || x >= most;
        if (!out) out = global_rs(a.rs_bits, x) || !global_window_valid(a.rs_bits, a.nbytes, x, k) ||
                        exact_window_minimizer([&](int u) { return global_code(a.reads, a.nbytes, (int64_t)x + u); }, k, p,
                                               a.filter) != mv;
        const uint32_t any = __ballot_sync(0xffffffffu, out);
        if (lane == 0) S.scan_tmp[warp] = any;
        __syncthreads();
        int first = -1;
#pragma unroll
        for (int w = TL_WARPS - 1; w >= 0; w--)
          if (S.scan_tmp[w]) first = 32 * w + __ffs((int)S.scan_tmp[w]) - 1;
        __syncthreads();  // before the words are written again
        if (first >= 0) {
          if (tid == 0) S.ext_end = (int)((int64_t)(x0 + first) - G0);
          break;
        }
        x0 += PT_NT;
      }
      __syncthreads();
    }

    // ---- ends, byte offsets: consecutive superkmers per thread ----
    const uint32_t per = (n_skm + PT_NT - 1) / PT_NT, i0 = min(tid * per, n_skm), i1 = min(i0 + per, n_skm);
    uint32_t my_bytes = 0;
    for (uint32_t i = i0; i < i1; i++) {
      const uint32_t l = S.spos[i];
      int w = (int)(l >> 5);
      uint32_t bits = S.brkw[w] & (0xFFFFFFFEu << (l & 31));
      while (!bits && ++w < NW / 32) bits = S.brkw[w];
      const uint32_t e = bits ? 32 * (uint32_t)w + __ffs((int)bits) - 1 : PT_EXT;
      const uint32_t end = bits ? e : (uint32_t)S.ext_end;
      S.send[i] = (uint16_t)e;
      const uint32_t nb = (end - l + k - 1 + 3) / 4;
      S.boff[i] = my_bytes;  // relative to the thread's first
      my_bytes += nb;
    }
    uint32_t tile_bytes;
    const uint32_t off0 = block_exclusive_scan<PT_NT>(my_bytes, S.scan_tmp, &tile_bytes);
    for (uint32_t i = i0; i < i1; i++) S.boff[i] += off0;
    const uint32_t rounded = (tile_bytes + 15u) & ~15u;
    if (tid == 0) {
      const unsigned long long bs = n_skm ? atomicAdd(a.cursors + 0, (unsigned long long)n_skm) : 0ull;
      const unsigned long long bb = rounded ? atomicAdd(a.cursors + 1, (unsigned long long)rounded) : 0ull;
      S.base_skm = bs;
      S.base_byte = bb;
      if (bs + n_skm > a.cap_skm || bb + rounded > a.cap_bytes) atomicOr(a.err, ERR_CAPACITY);
    }
    __syncthreads();
    const int ext_end = S.ext_end;
    // the staged packing needs every superkmer's bases in the tile's data
    const bool use_stg = rounded <= (uint32_t)PT_STG && (ext_end < 0 || ext_end + k - 1 <= 32 * TL_BWORDS);
    const unsigned long long base_skm = S.base_skm, base_byte = S.base_byte;
    const bool fits = base_skm + n_skm <= a.cap_skm && base_byte + rounded <= a.cap_bytes;

    // ---- descriptors, bin histograms; each superkmer's bases cut from the
    //      tile's 2-bit words into the staging area ----
    for (uint32_t i = tid; i < n_skm; i += PT_NT) {
      const uint32_t l = S.spos[i];
      const uint32_t e = S.send[i] == PT_EXT ? (uint32_t)ext_end : S.send[i];
      const uint32_t nk = e - l, len = nk + k - 1, mv = S.smm[i], bin = mv % (uint32_t)a.nbins;
      if (len > 0xFFFFFFu) atomicOr(a.err, ERR_BAD_READ);
      if (fits && len <= 0xFFFFFFu) {
        a.skm_desc[base_skm + i] = ((base_byte + S.boff[i]) << 24) | (uint64_t)len;
        a.skm_mm[base_skm + i] = mv;
        if (a.skm_gpos) a.skm_gpos[base_skm + i] = (uint64_t)(G0 + l);
      }
      if (bin < (uint32_t)a.nbins_smem) {
        atomicAdd(&h_skm[bin], 1u);
        atomicAdd(&h_km[bin], nk);
      } else {
        atomicAdd(&a.bin_nskm[bin], 1ull);
        atomicAdd(&a.bin_nkmers[bin], (unsigned long long)nk);
      }
      if (fits && use_stg) {
        const uint32_t nb = (len + 3) / 4;
        uint8_t *dst = S.stg + S.boff[i];
        for (uint32_t x = 0; 16 * x < len; x++) {
          const uint32_t B = l + 16 * x, w = B >> 4;
          uint32_t v = __funnelshift_l(S.t.pk[w + 1].x, S.t.pk[w].x, 2 * (B & 15u));
          const uint32_t rem = len - 16 * x;
          if (rem < 16) v &= 0xFFFFFFFFu << (32 - 2 * rem);  // zero padding after the last base
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (4 * x + u < nb) dst[4 * x + u] = (uint8_t)(v >> (24 - 8 * u));
        }
      }
    }
    if (fits && use_stg) {
      if (tid < 16 && tile_bytes + tid < rounded) S.stg[tile_bytes + tid] = 0;
      __syncthreads();
      uint4 *dst16 = reinterpret_cast<uint4 *>(a.packed + base_byte);
      const uint4 *src16 = reinterpret_cast<const uint4 *>(S.stg);
      for (uint32_t v = tid; v < rounded / 16; v += PT_NT) dst16[v] = src16[v];
    } else if (fits) {
      const uint32_t nwords = (tile_bytes + 3) / 4;
      uint32_t *dst = reinterpret_cast<uint32_t *>(a.packed + base_byte);
      for (uint32_t w = tid; w < nwords; w += PT_NT) {
        uint32_t word = 0;
        // superkmer holding the word's first byte: last i with boff[i] <= 4w
        int lo = 0, hi = (int)n_skm - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (S.boff[mid] <= w * 4) lo = mid; else hi = mid - 1;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint32_t q = w * 4 + u;
          if (q >= tile_bytes) break;
          while (lo + 1 < (int)n_skm && S.boff[lo + 1] <= q) lo++;
          const uint32_t l = S.spos[lo];
          const uint32_t e = S.send[lo] == PT_EXT ? (uint32_t)ext_end : S.send[lo];
          const uint32_t len = e - l + k - 1, bb = q - S.boff[lo];
          uint32_t byte = 0;
#pragma unroll
          for (int t = 0; t < 4; t++) {
            const uint32_t bi = bb * 4 + t;
            uint32_t c = 0;
            if (bi < len) {
              const uint32_t lp = l + bi;
              c = lp < 32u * TL_BWORDS ? tile_code(S.t, (int)lp) & 3u
                                       : global_code(a.reads, a.nbytes, G0 + (int64_t)lp) & 3u;
            }
            byte = (byte << 2) | c;
          }
          word |= byte << (8 * u);
        }
        dst[w] = word;
      }
    }
    __syncthreads();
  }

  // flush bin histograms
  __syncthreads();
  for (int i = tid; i < a.nbins_smem; i += PT_NT) {
    if (h_skm[i]) atomicAdd(&a.bin_nskm[i], (unsigned long long)h_skm[i]);
    if (h_km[i]) atomicAdd(&a.bin_nkmers[i], (unsigned long long)h_km[i]);
  }
}

size_t partition_smem_bytes(int nbins_smem) {
  return sizeof(PartSmem) + (size_t)nbins_smem * 2 * sizeof(uint32_t) + 16;
}

__global__ void k_partition_clear(ClearArgs a) {
  stamp_now(a.stamp);
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, nt = (uint64_t)gridDim.x * blockDim.x;
  if (t < 4) {
    a.cursors[t] = 0;
    a.err[t] = 0;
  }
  for (uint64_t i = t; i <= a.nbins; i += nt) a.bin_nskm[i] = a.bin_nkmers[i] = 0;
  for (uint64_t i = t; i < a.rs_words; i += nt) a.rs_bits[i] = 0;
}

// Read-start bitmap: bit offs[r]-offs[0] for every read, plus bit nbytes as
// the end-of-data sentinel.
__global__ void k_read_start_bits(const uint64_t *offs, uint64_t n_reads, uint32_t *bits) {
  uint64_t base = offs[0];
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r <= n_reads;
       r += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t pos = offs[r] - base;
    atomicOr(&bits[pos >> 5], 1u << (pos & 31));
  }
}

// Counting sort of superkmer descriptors by bin, with warp-aggregated atomics
// on the per-bin fill counters.
__global__ void k_bin_scatter(const unsigned long long *n_skm_ptr, const uint64_t *desc,
                              const uint32_t *mm, uint32_t nbins, const uint64_t *bin_start,
                              unsigned long long *bin_fill, uint64_t *out_desc, uint32_t *out_mm,
                              const uint64_t *gpos, uint64_t *out_gpos, const uint32_t *err) {
  if (*err & (ERR_CAPACITY | ERR_BAD_READ)) return;  // outputs incomplete: the host re-runs
  const uint64_t n = *n_skm_ptr;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x; i0 < n; i0 += stride) {
    uint64_t i = i0 + threadIdx.x;
    bool act = i < n;
    uint32_t active = __ballot_sync(0xffffffffu, act);
    if (!act) continue;
    uint32_t m = mm[i];
    uint32_t b = m % nbins;
    uint32_t peers = __match_any_sync(active, b);
    int leader = __ffs(peers) - 1;
    uint32_t rank = __popc(peers & ((1u << lane_id()) - 1u));
    unsigned long long base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(&bin_fill[b], (unsigned long long)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    uint64_t slot = bin_start[b] + base + rank;
    out_desc[slot] = desc[i];
    out_mm[slot] = m;
    if (gpos) out_gpos[slot] = gpos[i];
  }
}

// Bin placement without global atomics, for nbins <= kBinPlaceMaxBins.
// k_bin_count: superkmers per (bin, chunk of superkmers), stored
// bin-major (mat[b * nch_cap + c]) so that one exclusive scan gives every
// (bin, chunk) its first slot in bin order; k_bin_place then moves each
// chunk's superkmers with shared-memory cursors per bin.
__global__ void k_bin_count(const unsigned long long *n_skm_ptr, const uint32_t *mm, uint32_t nbins, uint32_t chunk,
                            uint64_t nch_cap, unsigned long long *mat, const uint32_t *err) {
  extern __shared__ uint32_t hcnt[];
  if (*err & (ERR_CAPACITY | ERR_BAD_READ)) return;
  const uint64_t n = *n_skm_ptr;
  for (uint64_t c = blockIdx.x; c < nch_cap; c += gridDim.x) {
    for (uint32_t b = threadIdx.x; b < nbins; b += blockDim.x) hcnt[b] = 0;
    __syncthreads();
    const uint64_t i1 = min(n, (c + 1) * (uint64_t)chunk);
    for (uint64_t i = c * (uint64_t)chunk + threadIdx.x; i < i1; i += blockDim.x)
      atomicAdd(&hcnt[mm[i] % nbins], 1u);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nbins; b += blockDim.x) mat[(uint64_t)b * nch_cap + c] = hcnt[b];
    __syncthreads();
  }
}

// Each chunk is placed in sub-rounds of kBinRound superkmers: counted per
// bin in shared memory, grouped by bin there, then written out so that each
// bin's superkmers leave as a run of consecutive slots.
__global__ void __launch_bounds__(kBinPlaceThreads, 2) k_bin_place(const unsigned long long *n_skm_ptr,
                                                                const uint64_t *desc, const uint32_t *mm,
                                                                uint32_t nbins, uint32_t chunk, uint64_t nch_cap,
                                                                const uint64_t *off, uint64_t *out_desc,
                                                                uint32_t *out_mm, const uint32_t *err) {
  extern __shared__ __align__(16) uint8_t bp_raw[];
  uint64_t *st_desc = reinterpret_cast<uint64_t *>(bp_raw);               // kBinRound
  uint32_t *st_mm = reinterpret_cast<uint32_t *>(st_desc + kBinRound);   // kBinRound
  uint64_t *cur = reinterpret_cast<uint64_t *>(st_mm + kBinRound);       // nbins: next global slot
  uint32_t *cnt = reinterpret_cast<uint32_t *>(cur + nbins);             // nbins: counts, then cursors
  uint32_t *lst = cnt + nbins;                                            // nbins: starts in the round
  __shared__ uint32_t tmp[64];
  if (*err & (ERR_CAPACITY | ERR_BAD_READ)) return;
  const uint64_t n = *n_skm_ptr;
  const uint64_t nch = min(nch_cap, (n + chunk - 1) / chunk);
  const int tid = threadIdx.x;
  for (uint64_t c = blockIdx.x; c < nch; c += gridDim.x) {
    for (uint32_t b = tid; b < nbins; b += kBinPlaceThreads) cur[b] = off[(uint64_t)b * nch_cap + c];
    const uint64_t c1 = min(n, (c + 1) * (uint64_t)chunk);
    for (uint64_t r0 = c * (uint64_t)chunk; r0 < c1; r0 += kBinRound) {
      const uint32_t m = (uint32_t)min((uint64_t)kBinRound, c1 - r0);
      for (uint32_t b = tid; b < nbins; b += kBinPlaceThreads) cnt[b] = 0;
      __syncthreads();
      constexpr int PER = kBinRound / kBinPlaceThreads;
      uint64_t dv[PER];
      uint32_t mv[PER], rk[PER];
#pragma unroll
      for (int u = 0; u < PER; u++) {
        const uint32_t i = u * kBinPlaceThreads + tid;
        if (i < m) {
          dv[u] = desc[r0 + i];
          mv[u] = mm[r0 + i];
          rk[u] = atomicAdd(&cnt[mv[u] % nbins], 1u);
        }
      }
      __syncthreads();
      // exclusive scan of the bin counts (thread-contiguous groups)
      {
        const uint32_t per = (nbins + kBinPlaceThreads - 1) / kBinPlaceThreads, b0 = tid * per;
        uint32_t s = 0;
        for (uint32_t b = b0; b < b0 + per && b < nbins; b++) s += cnt[b];
        uint32_t tot;
        uint32_t run = block_exclusive_scan<kBinPlaceThreads>(s, tmp, &tot);
        for (uint32_t b = b0; b < b0 + per && b < nbins; b++) {
          lst[b] = run;
          run += cnt[b];
        }
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PER; u++) {
        const uint32_t i = u * kBinPlaceThreads + tid;
        if (i < m) {
          const uint32_t p = lst[mv[u] % nbins] + rk[u];
          st_desc[p] = dv[u];
          st_mm[p] = mv[u];
        }
      }
      __syncthreads();
      for (uint32_t i = tid; i < m; i += kBinPlaceThreads) {
        const uint32_t v = st_mm[i], b = v % nbins;
        const uint64_t slot = cur[b] + (i - lst[b]);
        out_desc[slot] = st_desc[i];
        out_mm[slot] = v;
      }
      __syncthreads();
      for (uint32_t b = tid; b < nbins; b += kBinPlaceThreads) cur[b] += cnt[b];
      __syncthreads();
    }
  }
}

size_t bin_place_smem_bytes(uint32_t nbins) {
  return (size_t)kBinRound * 12 + (size_t)nbins * 16;
}

// Exclusive scans of the per-bin counters, one CTA (one thread alone took 22-25
// us at 256 bins).
__global__ void __launch_bounds__(kBinPrefixThreads) k_bin_prefix(const unsigned long long *bin_nskm,
                                                                  const unsigned long long *bin_nkmers, uint32_t nbins,
                                                                  uint64_t *bin_start, uint64_t *bin_kstart, unsigned long long *stamp) {
  stamp_now(stamp);
  constexpr int NT = kBinPrefixThreads;
  __shared__ uint64_t tmp[32];
  uint64_t cs = 0, ck = 0;
  for (uint32_t b0 = 0; b0 < nbins; b0 += NT) {
    const uint32_t b = b0 + threadIdx.x;
    uint64_t ts, tk;
    const uint64_t s = block_exclusive_scan_u64<NT>(b < nbins ? bin_nskm[b] : 0ull, tmp, &ts);
    const uint64_t kk = block_exclusive_scan_u64<NT>(b < nbins ? bin_nkmers[b] : 0ull, tmp, &tk);
    if (b < nbins) {
      bin_start[b] = cs + s;
      bin_kstart[b] = ck + kk;
    }
    cs += ts;
    ck += tk;
  }
  if (threadIdx.x == 0) {
    bin_start[nbins] = cs;
    bin_kstart[nbins] = ck;
  }
}

}  // namespace gkc
