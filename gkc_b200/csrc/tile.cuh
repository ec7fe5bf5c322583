// Minimizers of a tile of windows, shared by the partition and the per-window
// kernels.
//
// A CTA of TL_NT threads takes TL_NW consecutive windows of the concatenated
// reads, every warp TL_TW words of 32.  The tile's bases are held as 16-base
// words, each beside its reverse complement, so that any p-mer and its reverse
// complement are one funnel shift each; lane l of a warp holds window (and
// p-mer position) l of every word, and the minimum over the omega = k - p + 1
// p-mers of a window is built in registers by doubling (shifts by 1, 2, 4, ..
// positions between lanes), so no p-mer goes through shared memory.
// What bounds it is instruction issue: about 50 instructions a window, against
// 210 where p-mers rolled through bytes in shared memory and prefix and suffix
// minima were kept per position.
#pragma once
#include "common.cuh"
#include "minimizer.cuh"

namespace gkc {

constexpr int TL_NT = 256;
constexpr int TL_WARPS = TL_NT / 32;
constexpr int TL_TW = 15;                        // window words per warp
constexpr int TL_WORDS = TL_WARPS * TL_TW;       // window words per tile
constexpr int TL_NW = 32 * TL_WORDS;             // windows per tile
constexpr int TL_BWORDS = TL_WORDS + 3;          // words with bases (k <= 64: a window reaches two words on)
constexpr int TL_GROUPS = 2 * TL_BWORDS;         // 16-base groups
static_assert(TL_GROUPS <= TL_NT, "one 16-base group per thread");

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

// Filtered minimum of the p-mer at base 32 w + lane and its reverse
// complement; with POS also, in *code, the strand of the chosen one (0
// forward, 1 reverse, 2 both).
template <int FILT, bool POS>
GKC_DEV uint32_t tile_pmer(const TileBases &S, int w, int p, uint32_t M, uint32_t *code) {
  const uint32_t lane = threadIdx.x & 31u, sh = 2 * (lane & 15u);
  const uint2 a = S.pk[2 * w + (lane >> 4)], b = S.pk[2 * w + (lane >> 4) + 1];
  const uint32_t f = __funnelshift_l(b.x, a.x, sh) >> (32 - 2 * p);
  const uint32_t r = __funnelshift_r(a.y, b.y, sh) & M;
  const uint32_t vf = mm_filter(f, p, FILT) ? f : M;
  const uint32_t vr = mm_filter(r, p, FILT) ? r : M;
  if (POS) *code = f == r ? 2u : (vr < vf ? 1u : 0u);
  return vf < vr ? vf : vr;
}

// m[r], r < TL_TW: the minimum over the omega p-mers of window 32 (w0 + r) +
// lane (the last two words of m only feed the others).  With POS q[r] holds
// 4 * (tile base of the rightmost p-mer with that value) + its strand code.
template <int FILT, bool POS>
GKC_DEV void tile_minima(const TileBases &S, int w0, int p, int omega, uint32_t (&m)[TL_TW + 2],
                         uint32_t (&q)[POS ? TL_TW + 2 : 1]) {
  const uint32_t M = 0xFFFFFFFFu >> (32 - 2 * p), lane = threadIdx.x & 31u;
  const bool far = omega > 33;  // windows reach a second word
#pragma unroll
  for (int r = 0; r < TL_TW + 2; r++) {
    uint32_t code = 0;
    m[r] = 0xFFFFFFFFu;
    if (r < TL_TW + 1 || far) m[r] = tile_pmer<FILT, POS>(S, w0 + r, p, M, &code);
    if (POS) q[POS ? r : 0] = 4 * (32 * (uint32_t)(w0 + r) + lane) + code;
  }
  int done = 1;
  while (done < omega) {
    // min over `done` positions -> over 2 * done, or (the last step) over omega
    const int s = min(done, omega - done);  // 1 .. 32
    const uint32_t from = (lane + (uint32_t)s) & 31u;
    const bool same = lane + (uint32_t)s < 32u;
    uint32_t t = __shfl_sync(0xffffffffu, m[0], from), tq = 0;
    if (POS) tq = __shfl_sync(0xffffffffu, q[0], from);
#pragma unroll
    for (int r = 0; r < TL_TW + 2; r++) {
      uint32_t tn = 0xFFFFFFFFu, tqn = 0;
      if (r + 1 < TL_TW + 2) {
        tn = __shfl_sync(0xffffffffu, m[r + 1], from);
        if (POS) tqn = __shfl_sync(0xffffffffu, q[POS ? r + 1 : 0], from);
      }
      const uint32_t y = same ? t : tn;
      if (POS) {
        const uint32_t yq = same ? tq : tqn;
        if (y <= m[r]) q[POS ? r : 0] = yq;  // the rightmost of equal ones
      }
      m[r] = y < m[r] ? y : m[r];
      t = tn;
      tq = tqn;
    }
    done += s;
  }
}

}  // namespace gkc
