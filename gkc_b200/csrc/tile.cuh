// Minimizers of a tile of windows, shared by the partition and the per-window
// kernels.
//
// A CTA takes a tile of consecutive windows of the concatenated reads, each
// warp a strip of them and each lane 16.  The tile's bases are held as 16-base
// words, each beside its reverse complement, so that any p-mer and its reverse
// complement are one funnel shift each, by a constant: lane l needs two words
// for its 16 p-mers.  The minimum over the omega = k - p + 1 p-mers of a
// window is built by doubling (shifts by 1, 2, 4, .. positions): most shifted
// values are the lane's own registers, the rest come from the next lanes, so
// no p-mer goes through shared memory.  The strip's last lanes only feed the
// others: 30 lanes have windows of their own, 28 where omega > 33.
// What bounds it is instruction issue (the ALU pipe): about 25 instructions a
// window, against 50 with one window of every word per lane (each shift an
// exchange and a select) and 210 where p-mers rolled through bytes in shared
// memory and prefix and suffix minima were kept per position.
#pragma once
#include "common.cuh"
#include "minimizer.cuh"

namespace gkc {

constexpr int TL_NT = 256;
constexpr int TL_WARPS = TL_NT / 32;
constexpr int TL_W = 16;                         // windows per lane
constexpr int TL_BWORDS = 123;                   // 32-base words: the last strip's p-mers and windows reach 3936 bases
constexpr int TL_GROUPS = 2 * TL_BWORDS;         // 16-base groups
constexpr int TL_NW_MAX = TL_WARPS * 30 * TL_W;  // windows per tile
static_assert(TL_GROUPS <= TL_NT, "one 16-base group per thread");
GKC_HOST_DEV int tile_strip(int omega) { return omega > 33 ? 28 * TL_W : 30 * TL_W; }  // windows per warp

// Whether a 2p-bit p-mer value passes the filter (mm_filter for such values).
template <int FILT>
GKC_DEV bool tile_pass(uint32_t v, int p) {
  // AAA, ACA or AGA on top: first base A, second below T, third A
  if (FILT == FILTER_NEW2) return v >= (3u << (2 * p - 4)) || (v & (3u << (2 * p - 6))) != 0;
  return mm_filter(v, p, FILT);
}

struct TileBases {
  uint2 pk[TL_GROUPS + 2];   // 16 bases, 2 bits each, first base in the top bits; their reverse complement
  uint32_t badw[TL_BWORDS + 2];  // bit i: base i is not ACGTU
  uint32_t rsw[TL_BWORDS + 2];   // bit i: a read starts at base i
};

// 2-bit codes of 4 bytes (16 bases a register): A/U 0, C 1, G 2, T 3, any
// other byte 3 with its flag set in *bad (bit 7 of each byte).  The low three
// bits of a letter name it; PRMT looks up the letter they stand for and its
// code, four at a time.
GKC_DEV uint32_t codes4(uint32_t v, uint32_t *bad) {
  const uint32_t x = v & 0x07070707u, y = x | (x >> 4);
  const uint32_t sel = __byte_perm(y, 0, 0x4420);                 // four selectors of 4 bits
  // index 1 'A', 3 'C', 4 'T', 5 'U', 7 'G' (upper case); the others match no byte of their index
  const uint32_t want = __byte_perm(0x430041FFu, 0x47005554u, sel);
  const uint32_t z = (v & 0xDFDFDFDFu) ^ want;
  const uint32_t nz = (((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z) & 0x80808080u;
  *bad = nz;
  const uint32_t code = __byte_perm(0x01000000u, 0x02000003u, sel);
  return code | (nz >> 7) | (nz >> 6);                            // a bad byte counts as T (3)
}

// 16 bytes -> 16 codes packed (first base in the top bits) and a 16-bit bad mask.
GKC_DEV uint32_t pack16(uint4 v, uint32_t *bad16) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t pk = 0, bad = 0;
#pragma unroll
  for (int t = 0; t < 4; t++) {
    uint32_t nz;
    const uint32_t c = codes4(w[t], &nz);
    pk = (pk << 8) | ((c * 0x40100401u) >> 24);                   // first base of the four in the top bits
    bad |= (((nz >> 7) * 0x01020408u) >> 24) << (4 * t);          // first base in the lowest bit
  }
  *bad16 = bad;
  return pk;
}

// Reverse complement of 16 packed bases.
GKC_DEV uint32_t revcomp16(uint32_t x) {
  x = __brev(~x);
  return ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
}

// The 16 bytes of group q of the tile whose first base is at G0 (a multiple
// of 32); bytes outside [0, nbytes) read as 0, which is no base.
GKC_DEV uint4 tile_fetch(const uint8_t *reads, uint64_t nbytes, int aligned16, int64_t G0, int q) {
  const int64_t g = G0 + 16 * q;
  if (g >= 0 && (uint64_t)(g + 16) <= nbytes && aligned16) return __ldg(reinterpret_cast<const uint4 *>(reads + g));
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  for (int t = 0; t < 16; t++)
    if (g + t >= 0 && (uint64_t)(g + t) < nbytes) w[t >> 2] |= (uint32_t)reads[g + t] << (8 * (t & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Stores the thread's group of the tile and the read-start words (call by all
// threads; a barrier follows).
GKC_DEV void tile_store(TileBases &S, uint4 v, const uint32_t *rs_bits, uint64_t rs_words, int64_t G0) {
  const int q = threadIdx.x;
  uint32_t bad = 0;
  if (q < TL_GROUPS) {
    const uint32_t pk = pack16(v, &bad);
    S.pk[q] = make_uint2(pk, revcomp16(pk));
  }
  const uint32_t other = __shfl_xor_sync(0xffffffffu, bad, 1);
  if (q < TL_GROUPS && (q & 1) == 0) S.badw[q >> 1] = bad | (other << 16);
  if (q < 2) {
    S.pk[TL_GROUPS + q] = make_uint2(0u, 0u);
    S.badw[TL_BWORDS + q] = 0u;
    S.rsw[TL_BWORDS + q] = 0u;
  }
  if (q < TL_BWORDS) {
    const int64_t gw = (G0 >> 5) + q;
    S.rsw[q] = gw >= 0 && (uint64_t)gw < rs_words ? rs_bits[gw] : 0u;
  }
}

// Bit i (0..31) of the result = OR of bits i .. i+n-1 of the 96-bit value
// (x2:x1:x0), for 1 <= n <= 64: a sliding OR built by doubling shifts.
GKC_DEV uint32_t span_or(uint32_t x0, uint32_t x1, uint32_t x2, int n) {
  uint64_t lo = (uint64_t)x0 | ((uint64_t)x1 << 32);
  uint64_t hi = x2;
  int m = 1;
  while (2 * m <= n) {  // lo:hi now holds the OR over m consecutive bits
    lo |= (lo >> m) | (hi << (64 - m));
    hi |= hi >> m;
    m *= 2;
  }
  const int r = n - m;  // 0 <= r < m: cover the remaining bits with an overlapping shift
  if (r > 0) lo |= (lo >> r) | (hi << (64 - r));
  return (uint32_t)lo;
}

// Windows of word w that lie inside one read and inside the bytes [lo, hi)
// (*valid), and those that touch a byte that is no base.
GKC_DEV void tile_valid(const TileBases &S, int w, int64_t G0, int64_t lo, int64_t hi, int k, uint32_t *valid,
                        uint32_t *touch) {
  const uint32_t r0 = S.rsw[w], r1 = S.rsw[w + 1], r2 = S.rsw[w + 2];
  // read starts at window bytes 1 .. k-1: the span shifted by one
  const uint32_t hit = k > 1 ? span_or((r0 >> 1) | (r1 << 31), (r1 >> 1) | (r2 << 31), r2 >> 1, k - 1) : 0u;
  *touch = span_or(S.badw[w], S.badw[w + 1], S.badw[w + 2], k);
  const int64_t s0 = G0 + 32 * (int64_t)w;  // windows s0 + i with lo <= s0 + i <= hi - k
  const int64_t ilo = lo > s0 ? lo - s0 : 0, ihi = hi - k - s0;
  uint32_t range = 0u;
  if (ihi >= 0 && ilo <= 31 && ihi >= ilo) {
    const int a = (int)ilo, b = (int)(ihi > 31 ? 31 : ihi);
    range = (0xFFFFFFFFu >> (31 - b)) & (0xFFFFFFFFu << a);
  }
  *valid = ~hit & range;
}

// Code of tile base l as the exact rule wants it: 255 where it is no base.
GKC_DEV uint32_t tile_code(const TileBases &S, int l) {
  if ((S.badw[l >> 5] >> (l & 31)) & 1u) return 255u;
  return (S.pk[l >> 4].x >> (30 - 2 * (l & 15))) & 3u;
}

// The (up to) 64 bases from tile base l on, in registers.
struct WindowBases {
  uint64_t hi, lo, bad;  // bases 0 .. 31 and 32 .. 63, the first on top (no base: 3); bit i: base i is no base
};
GKC_DEV WindowBases window_bases(const TileBases &S, int l) {
  const int j = l >> 4, q = l >> 5;
  const uint32_t sh = 2 * (uint32_t)(l & 15), bs = (uint32_t)(l & 31);
  uint32_t w[5];
#pragma unroll
  for (int t = 0; t < 5; t++) w[t] = S.pk[j + t].x;
  WindowBases b;
  b.hi = (uint64_t)__funnelshift_l(w[1], w[0], sh) << 32 | __funnelshift_l(w[2], w[1], sh);
  b.lo = (uint64_t)__funnelshift_l(w[3], w[2], sh) << 32 | __funnelshift_l(w[4], w[3], sh);
  const uint32_t b1 = S.badw[q + 1];
  b.bad = (uint64_t)__funnelshift_r(b1, S.badw[q + 2], bs) << 32 | __funnelshift_r(S.badw[q], b1, bs);
  return b;
}
// The bases [j, k) in order, 16 taken from the registers at a time:
// step(code, whether it is no base) for each.
template <typename Step>
GKC_DEV void each_base(WindowBases b, int j, int k, Step &&step) {
  if (j > 0) {  // 0 < j <= 16
    b.hi = b.hi << (2 * j) | b.lo >> (64 - 2 * j);
    b.lo <<= 2 * j;
    b.bad >>= j;
  }
  for (; j < k; j += 16) {
    uint32_t w = (uint32_t)(b.hi >> 32), x = (uint32_t)b.bad;
    const int n = min(16, k - j);
#pragma unroll 4
    for (int t = 0; t < n; t++) {
      step(w >> 30, (x & 1u) != 0u);
      w <<= 2;
      x >>= 1;
    }
    b.hi = b.hi << 32 | b.lo >> 32;
    b.lo <<= 32;
    b.bad >>= 16;
  }
}

// exact_window_minimizer from the window's bases in registers (codes of bytes
// that are no base: 255, as there).  A window costs k + p codes, each some 25
// instructions; 15 M bases with 30% N, k 31: partition 0.67 ms, with every code
// read from shared memory and the filter chosen at each 1.36.
template <int FILT>
GKC_DEV uint32_t exact_minimizer(const WindowBases &b, int k, int p) {
  const uint32_t M = 0xFFFFFFFFu >> (32 - 2 * p);
  uint32_t f = 0, r = 0;
  each_base(b, 0, p, [&](uint32_t c, bool bad) { f = (f << 2) | (bad ? 255u : c); });
  uint32_t w = (uint32_t)(b.hi >> 32) >> (32 - 2 * p), x = (uint32_t)b.bad << (32 - p);
  for (int j = 0; j < p; j++) {  // from base p - 1 down
    r = (r << 2) | ((int32_t)x < 0 ? 255u : 3u - (w & 3u));
    w >>= 2;
    x <<= 1;
  }
  uint32_t best = min(mm_filter(f, p, FILT) ? f : M, mm_filter(r, p, FILT) ? r : M);
  each_base(b, p, k, [&](uint32_t c, bool bad) {
    f = ((f << 2) | (bad ? 255u : c)) & M;
    r = (r >> 2) | ((bad ? 255u : 3u - c) << (2 * p - 2));
    if (mm_filter(f, p, FILT)) best = min(best, f);
    if (mm_filter(r, p, FILT)) best = min(best, r);
  });
  return best;
}
GKC_DEV uint32_t exact_minimizer(const WindowBases &b, int k, int p, int filter) {
  switch (filter) {
    case FILTER_ALL: return exact_minimizer<FILTER_ALL>(b, k, p);
    case FILTER_NEW: return exact_minimizer<FILTER_NEW>(b, k, p);
    case FILTER_SIGNATURE: return exact_minimizer<FILTER_SIGNATURE>(b, k, p);
    default: return exact_minimizer<FILTER_NEW2>(b, k, p);
  }
}

// m[i], i < 16: the filtered minimum of the p-mer at tile base P + i, P =
// 16 (j0 + lane), and its reverse complement.  With POS q[i] holds 4 * (tile
// base) + the strand of the chosen one (0 forward, 1 reverse, 2 both).
template <int FILT, bool POS>
GKC_DEV void tile_pmers(const TileBases &S, int j0, int p, uint32_t (&m)[TL_W], uint32_t (&q)[POS ? TL_W : 1]) {
  const uint32_t M = 0xFFFFFFFFu >> (32 - 2 * p), lane = threadIdx.x & 31u;
  const uint2 a = S.pk[j0 + lane], b = S.pk[j0 + lane + 1];
#pragma unroll
  for (int i = 0; i < TL_W; i++) {
    const uint32_t f = __funnelshift_l(b.x, a.x, 2 * i) >> (32 - 2 * p);
    const uint32_t r = __funnelshift_r(a.y, b.y, 2 * i) & M;
    const uint32_t vf = tile_pass<FILT>(f, p) ? f : M;
    const uint32_t vr = tile_pass<FILT>(r, p) ? r : M;
    m[i] = min(vf, vr);
    if (POS) q[POS ? i : 0] = 4 * (16 * (uint32_t)(j0 + lane) + i) + (f == r ? 2u : (vr < vf ? 1u : 0u));
  }
}

// m[i] = min(m[i], the value 16 ls + T positions on); with POS the q of the
// later one where they are equal.
template <int T, bool POS>
GKC_DEV void tile_shift(uint32_t (&m)[TL_W], uint32_t (&q)[POS ? TL_W : 1], int ls) {
  uint32_t t[T > 0 ? T : 1], tq[POS && T > 0 ? T : 1];
#pragma unroll
  for (int j = 0; j < T; j++) {
    t[j] = __shfl_down_sync(0xffffffffu, m[j], ls + 1);
    if (POS) tq[POS ? j : 0] = __shfl_down_sync(0xffffffffu, q[POS ? j : 0], ls + 1);
  }
#pragma unroll
  for (int i = 0; i < TL_W; i++) {
    uint32_t y, yq = 0;
    if (i + T < TL_W) {
      const int x = i + T < TL_W ? i + T : 0;
      y = m[x];
      if (POS) yq = q[POS ? x : 0];
      if (ls) {
        y = __shfl_down_sync(0xffffffffu, y, ls);
        if (POS) yq = __shfl_down_sync(0xffffffffu, yq, ls);
      }
    } else {
      const int x = i + T >= TL_W ? i + T - TL_W : 0;
      y = t[T > 0 ? x : 0];
      if (POS) yq = tq[POS && T > 0 ? x : 0];
    }
    if (POS) {
      if (y <= m[i]) q[POS ? i : 0] = yq;
    }
    m[i] = min(m[i], y);
  }
}

// The minimum over omega positions from p-mer minima (and, with POS, the
// rightmost position that has it).
template <bool POS>
GKC_DEV void tile_slide(uint32_t (&m)[TL_W], uint32_t (&q)[POS ? TL_W : 1], int omega) {
  if (omega >= 2) tile_shift<1, POS>(m, q, 0);
  if (omega >= 4) tile_shift<2, POS>(m, q, 0);
  if (omega >= 8) tile_shift<4, POS>(m, q, 0);
  if (omega >= 16) tile_shift<8, POS>(m, q, 0);
  if (omega >= 32) tile_shift<0, POS>(m, q, 1);
  int done = 1;
  while (2 * done <= omega) done *= 2;
  const int s = omega - done;  // the last step overlaps; 0 .. 31
  switch (s & 15) {
    case 0: if (s) tile_shift<0, POS>(m, q, s >> 4); break;
    case 1: tile_shift<1, POS>(m, q, s >> 4); break;
    case 2: tile_shift<2, POS>(m, q, s >> 4); break;
    case 3: tile_shift<3, POS>(m, q, s >> 4); break;
    case 4: tile_shift<4, POS>(m, q, s >> 4); break;
    case 5: tile_shift<5, POS>(m, q, s >> 4); break;
    case 6: tile_shift<6, POS>(m, q, s >> 4); break;
    case 7: tile_shift<7, POS>(m, q, s >> 4); break;
    case 8: tile_shift<8, POS>(m, q, s >> 4); break;
    case 9: tile_shift<9, POS>(m, q, s >> 4); break;
    case 10: tile_shift<10, POS>(m, q, s >> 4); break;
    case 11: tile_shift<11, POS>(m, q, s >> 4); break;
    case 12: tile_shift<12, POS>(m, q, s >> 4); break;
    case 13: tile_shift<13, POS>(m, q, s >> 4); break;
    case 14: tile_shift<14, POS>(m, q, s >> 4); break;
    default: tile_shift<15, POS>(m, q, s >> 4); break;
  }
}

// Minimizers of the warp's strip from window P0 (a multiple of 32) on: lane
// l's m[i] is that of window P0 + 16 l + i.
template <bool POS>
GKC_DEV void tile_minima(const TileBases &S, int P0, int k, int p, int filter, uint32_t (&m)[TL_W],
                         uint32_t (&q)[POS ? TL_W : 1]) {
  switch (filter) {
    case FILTER_ALL: tile_pmers<FILTER_ALL, POS>(S, P0 >> 4, p, m, q); break;
    case FILTER_NEW: tile_pmers<FILTER_NEW, POS>(S, P0 >> 4, p, m, q); break;
    case FILTER_SIGNATURE: tile_pmers<FILTER_SIGNATURE, POS>(S, P0 >> 4, p, m, q); break;
    default: tile_pmers<FILTER_NEW2, POS>(S, P0 >> 4, p, m, q); break;
  }
  tile_slide<POS>(m, q, k - p + 1);
}

// The windows of `mask` (bit i: the lane's window i) listed for the whole warp,
// so that those that touch a byte that is no base are redone by the exact rule
// 32 at a time (a single such byte touches k windows in a row, which few lanes
// hold).  Returns their number; *rank: that of the lane's first one.
constexpr int TL_REDO = 30 * TL_W;  // windows a warp may have to redo
GKC_DEV uint32_t tile_list(uint32_t mask, int P0, uint16_t *list, uint32_t *rank) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t rk = __popc(mask);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, rk, d);
    if (lane >= (uint32_t)d) rk += y;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, rk, 31);
  rk -= __popc(mask);
  *rank = rk;
  for (uint32_t left = mask; left; left &= left - 1) list[rk++] = (uint16_t)(P0 + TL_W * lane + __ffs((int)left) - 1);
  __syncwarp();
  return total;
}
// Their minimizers: m[i] for the lane's window i of the mask.
struct RedoArea {
  uint32_t v[TL_REDO / 16 * 17];  // in the list's order, so that lanes 16 apart meet in no bank
  uint16_t list[TL_REDO];
};
GKC_DEV void tile_redo(const TileBases &S, uint32_t mask, int P0, RedoArea &R, int k, int p, int filter,
                       uint32_t (&m)[TL_W]) {
  uint32_t rank;
  const uint32_t total = tile_list(mask, P0, R.list, &rank);
  for (uint32_t r = threadIdx.x & 31u; r < total; r += 32)
    R.v[r + (r >> 4)] = exact_minimizer(window_bases(S, R.list[r]), k, p, filter);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < TL_W; i++)
    if ((mask >> i) & 1u) {
      m[i] = R.v[rank + (rank >> 4)];
      rank++;
    }
  __syncwarp();
}

}  // namespace gkc
