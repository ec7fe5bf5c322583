// Canonical k-mer counting from bin-grouped superkmers (batched path).
//
// Semantics follow kmc_counting_GPU (kmer_counting.cu:95-191): every k-mer of
// every superkmer of a bin, canonicalised as min(x, revcomp(x)), sorted
// ascending, run-length counted (count clamped to 2^32-1), per bin.
//
// The keys of a bin are split into buckets of about 3 K keys: runs of digits, the digit being the top bits of an order-preserving map of
// the key (eq_map), so a bin's sorted list is the concatenation of its
// buckets' sorted lists.  Device stages:
//   1. k_bucket_hist    - expands every k-mer once and counts the digits of
//                         each chunk of a bin's k-mers.  A lane takes a piece
//                         of consecutive k-mers of a superkmer from one load
//                         of aligned words;
//   2. k_bucket_scan    - one CTA per bin packs the digits into buckets;
//                         k_bucket_offsets turns the (chunk, digit) counts
//                         into each chunk's write offset per bucket;
//   3. k_bucket_scatter - moves every key to its chunk's offset for its
//                         bucket plus its rank there;
//   4. k_bucket_sort    - persistent, buckets taken by ticket, each counted
//                         on its own (8-byte keys that mostly repeat: in a
//                         small hash table first): split into groups of about
//                         100 keys by splitters taken from its keys, the
//                         groups sorted by warps in registers and run-length
//                         encoded.  The runs are staged at the bucket's own
//                         key range and its distinct count recorded;
//                         k_compact_runs then moves them to the scan of the
//                         counts;
//      k_bucket_open    - the buckets too large for that, and those in which
//                         copies of one key fill a group: the keys aggregated
//                         in a shared-memory hash table and the distinct ones
//                         sorted by a sample sort.  A bucket with too many
//                         distinct keys is sorted by the digit that follows
//                         the common prefix of its smallest and largest key
//                         and cut into slices;
//      k_bucket_slices  - counts the slices; a digit larger than a slice is
//                         opened the same way, one prefix further on.
#include "common.cuh"
#include "kernels.h"

namespace gkc {

// ------------------------------------------------------------ key digits

// Top 32 bits of a 2k-bit key, left-aligned when the key is shorter.
GKC_DEV uint32_t key_top32(uint64_t x, int key_bits) {
  // (the clamping shift gives the high word at key_bits = 64)
  return key_bits >= 32 ? __funnelshift_rc((uint32_t)x, (uint32_t)(x >> 32), key_bits - 32)
                        : (uint32_t)x << (32 - key_bits);
}
GKC_DEV uint32_t key_top32(u128 x, int key_bits) { return (uint32_t)(x >> (key_bits - 32)); }  // k > 32

// Order-preserving map of a canonical key's top 32 bits t that spreads
// canonical keys evenly: the canonical key of a uniform k-mer is the smaller
// of two near-independent uniform values, whose distribution function is
// 1 - (1 - u)^2; v = 2^32 (1 - (1 - t / 2^32)^2), non-decreasing in t.
GKC_DEV uint32_t eq_map(uint32_t t) { return ~__umulhi(~t, ~t); }

GKC_DEV uint32_t coarse_of(uint32_t v, int cb) { return __funnelshift_rc(v, 0u, 32 - cb); }  // 0 at cb = 0

template <typename K>
GKC_DEV uint32_t coarse_digit(K x, int key_bits, int cb) {
  return coarse_of(eq_map(key_top32(x, key_bits)), cb);
}

// Bits of a key type, its leading zeros, and the sb bits that follow the
// first cp bits (keys of one bucket share their first cp bits, the common
// prefix of the bucket's smallest and largest key, so these digits order the
// bucket's keys by their first differing bits whatever the distribution).
template <typename K> constexpr int key_type_bits() { return 8 * (int)sizeof(K); }
GKC_DEV int key_clz(uint64_t x) { return __clzll((long long)x); }
GKC_DEV int key_clz(u128 x) {
  const uint64_t hi = (uint64_t)(x >> 64);
  return hi ? __clzll((long long)hi) : 64 + __clzll((long long)(uint64_t)x);
}
template <typename K>
GKC_DEV uint32_t prefix_digit(K x, int cp, int sb) {
  if (sb == 0) return 0u;  // sb <= key bits - cp, so cp < key bits here
  return (uint32_t)((K)(x << cp) >> (key_type_bits<K>() - sb));
}
// The sub-bucket bits of a bucket of m keys whose smallest and largest keys
// are lo and hi: about two sub-buckets per key, at most CC_SB_MAX bits, and
// no more than the bits below the common prefix.
template <typename K>
GKC_DEV void prefix_split(K lo, K hi, uint64_t m, int sb_max, int *cp, int *sb) {
  *cp = lo == hi ? key_type_bits<K>() : key_clz((K)(lo ^ hi));
  int b = 0;
  while (b < sb_max && ((uint64_t)1 << b) < 2 * m) b++;
  *sb = min(b, key_type_bits<K>() - *cp);
}

// Pulls the 128-byte line holding p into L2 (no register waits for it).
GKC_DEV void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ------------------------------------------------------------------ planning

// Digit bits of a bin of nk keys: none where one bucket holds them, else
// digits of about an eighth of a bucket (so that the buckets packed from them
// come out even although the digits do not), at most max_bits.
GKC_DEV uint32_t plan_bits(uint64_t nk, uint32_t bucket_keys, uint32_t max_bits, uint32_t key_bits) {
  uint32_t bits = 0;
  if (nk > bucket_keys)
    while (bits < max_bits && bits < key_bits && (nk >> bits) > bucket_keys / 8) bits++;
  return bits;
}
// One CTA: the digits and chunks of every bin and the chunks' prefixes
// (one bin per thread; one thread for all bins took 71-134 us at 256 bins).
// A bin that is too large is flagged here, before the kernels that return at
// the flag begin: threads of one block must not read it differently.
__global__ void __launch_bounds__(kCountPlanThreads) k_count_plan(CountPlan pl) {
  constexpr int NT = kCountPlanThreads;
  __shared__ uint64_t tmp[32];
  const bool dead = (*pl.err & (ERR_CAPACITY | ERR_BAD_READ)) != 0;
  uint64_t cb = 0, hb = 0;
  for (uint32_t b0 = 0; b0 < pl.nbins; b0 += NT) {
    const uint32_t b = b0 + threadIdx.x;
    const bool in = b < pl.nbins;
    const uint64_t nk = dead || !in ? 0 : pl.bin_kstart[b + 1] - pl.bin_kstart[b];
    if (nk >> 32) atomicOr(pl.err, ERR_BIN_TOO_LARGE);  // offsets in a bin are 32-bit
    const uint32_t bits = plan_bits(nk, pl.bucket_keys, pl.max_bits, 2 * pl.k);
    const uint64_t nch = (nk + pl.chunk_kmers - 1) / pl.chunk_kmers;
    uint64_t nc, nh;
    const uint64_t oc = block_exclusive_scan_u64<NT>(nch, tmp, &nc);
    const uint64_t oh = block_exclusive_scan_u64<NT>(nch << bits, tmp, &nh);
    if (in) {
      pl.bin_bits[b] = bits;
      pl.chunk_base[b] = cb + oc;
      pl.hist_base[b] = hb + oh;
    }
    cb += nc;
    hb += nh;
  }
  if (threadIdx.x < 8) pl.tickets[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    pl.chunk_base[pl.nbins] = cb;
    pl.hist_base[pl.nbins] = hb;
  }
}

// The last index i in [lo, hi] with a[i] <= x (a ascending, a[lo] <= x), by
// the whole warp: 32 probes a step, so that few dependent loads follow on
// another.
GKC_DEV uint64_t warp_last_le(const uint64_t *a, uint64_t lo, uint64_t hi, uint64_t x) {
  const uint32_t lane = threadIdx.x & 31u;
  while (lo < hi) {
    const uint64_t step = (hi - lo) / 32 + 1, at = lo + lane * step;
    const uint32_t le = __ballot_sync(0xffffffffu, at <= hi && __ldg(a + at) <= x);
    lo += (uint64_t)(__popc(le) - 1) * step;
    hi = min(hi, lo + step - 1);
  }
  return lo;
}

// First superkmer of every chunk: the last superkmer of the bin whose k-mer
// prefix is at most the chunk's first k-mer.  Clears the digit totals, too.
__global__ void k_chunk_first(ExpandArgs a) {
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, nt = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = t >> 5; b < a.nbins; b += nt >> 5) {  // a warp per bin, its digits only
    uint32_t *tot = a.digit_total + (b << a.max_bits);
    for (uint32_t d = threadIdx.x & 31u; d < 1u << a.bin_bits[b]; d += 32) tot[d] = 0;
  }
  const uint64_t n_chunks = a.chunk_base[a.nbins];
  for (uint64_t c = t >> 5; c < n_chunks; c += nt >> 5) {  // a warp per chunk
    const uint32_t b = (uint32_t)warp_last_le(a.chunk_base, 0, a.nbins - 1, c);
    const uint64_t q0 = a.bin_kstart[b] + (c - a.chunk_base[b]) * a.chunk_kmers;
    const uint64_t s = warp_last_le(a.koff, a.bin_start[b], a.bin_start[b + 1] - 1, q0);
    if ((threadIdx.x & 31u) == 0) a.chunk_s0[c] = s;
  }
}

// ------------------------------------------------------- k-mer runs

constexpr int KM_PIECE = 6;  // consecutive k-mers of a superkmer that a lane takes

// The bases of a piece as 32-bit words of the packed ones (2 bits per base,
// MSB first within a byte): its first base is in word 0, r bits below the top
// once the word's bytes are swapped.  All words are loaded, so reads end
// within 16 bytes past the last superkmer (every packed buffer has them).
template <typename K> struct PackedWords {
  static constexpr int N = sizeof(K) / 4 + 2;  // 2 k + 2 (KM_PIECE - 1) + 30 bits
  uint32_t w[N];
  uint32_t r, count;  // k-mers of the piece: 0 .. KM_PIECE
};
template <typename K>
GKC_DEV void load_packed(PackedWords<K> &p, const uint8_t *packed, uint64_t off, uint32_t o) {
  const uint64_t at = off + (o >> 2);
  const uint32_t *src = reinterpret_cast<const uint32_t *>(packed + (at & ~3ull));
  p.r = 8 * ((uint32_t)at & 3u) + 2 * (o & 3u);
#pragma unroll
  for (int t = 0; t < PackedWords<K>::N; t++) p.w[t] = p.count ? __ldg(src + t) : 0u;
}

// Reverse complement of 16 bases.
GKC_DEV uint32_t revcomp32(uint32_t x) {
  const uint32_t y = __brev(x);
  return 2 * (~y & 0x55555555u) + (~(y >> 1) & 0x55555555u);
}
// The canonical keys (the smaller of a k-mer and its reverse complement) of a
// piece, each to emit(key, valid).  The reverse complement of the piece's
// words is taken once: that of a k-mer lies in it, as the k-mer in the words,
// two bits further on for each k-mer.
template <typename K, typename Emit>
GKC_DEV void emit_piece(const PackedWords<K> &p, int k, Emit &&emit) {
  constexpr int KW = sizeof(K) / 4;
  uint32_t b[KW + 2], w[KW + 1], rc[KW + 1];
#pragma unroll
  for (int t = 0; t < KW + 2; t++) b[t] = __byte_perm(p.w[t], 0, 0x0123);
#pragma unroll
  for (int t = 0; t <= KW; t++) {
    w[t] = __funnelshift_l(b[t + 1], b[t], p.r);
    rc[t] = revcomp32(w[t]);
  }
  const int s = 8 * (int)sizeof(K) - 2 * k;  // 0 .. 62
  const uint32_t m0 = s < 32 ? 0xFFFFFFFFu >> s : 0u, m1 = s < 32 ? 0xFFFFFFFFu : 0xFFFFFFFFu >> (s - 32);
#pragma unroll
  for (int t = 0; t < KM_PIECE; t++) {
    uint32_t m[KW], c[KW];  // the words from the k-mer's first base on; its reverse complement (both: word 0 on top)
#pragma unroll
    for (int i = 0; i < KW; i++) {
      m[i] = __funnelshift_l(w[i + 1], w[i], 2 * t);
      c[KW - 1 - i] = __funnelshift_r(rc[i], rc[i + 1], 2 * t);
    }
    c[0] &= m0;
    c[1] &= m1;
    K x = 0, r = 0;
#pragma unroll
    for (int i = 0; i < KW; i++) {
      const uint32_t v = s < 32 ? __funnelshift_r(m[i], i > 0 ? m[i > 0 ? i - 1 : 0] : 0u, s)
                                : i == 0 ? 0u : __funnelshift_r(m[i > 0 ? i - 1 : 0], i > 1 ? m[i > 1 ? i - 2 : 0] : 0u, s - 32);
      x = (x << 32) | (K)v;
      r = (r << 32) | (K)c[i];
    }
    emit(x < r ? x : r, (uint32_t)t < p.count);
  }
}

GKC_DEV uint32_t warp_exclusive_scan(uint32_t c, uint32_t *total) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t inc = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= (uint32_t)d) inc += t;
  }
  *total = __shfl_sync(0xffffffffu, inc, 31);
  return inc - c;
}

// The k-mers [qa, qb) of one bin, taken by the calling warp: 32 superkmers,
// one per lane, are cut into pieces of KM_PIECE consecutive k-mers, and each
// round every lane takes a piece, found in a bitmap of the pieces that begin a
// superkmer.  Whole rounds only: the pieces left over come first in the next
// batch of superkmers, which begins with theirs.  The canonical keys go to
// emit(key, valid) (called by every lane), in no order that matters.  s0 is
// the superkmer holding k-mer qa, s_end the bin's end (k-mer offsets up to
// koff[s_end] are read).
//
// What bounds it is instruction issue and the latency of the packed bases,
// which lie in tile order: a lane's words, their bytes swapped, its place and
// its reverse complement serve several k-mers; positions are 32-bit, relative to
// qa; the next batch's ends and descriptors are loaded before this one's
// rounds, and a piece's words requested before the piece before it is emitted.
template <typename K, typename Emit>
GKC_DEV void warp_kmers(const ExpandArgs &a, uint64_t qa, uint64_t qb, uint64_t s0, uint64_t s_end, Emit &&emit) {
  constexpr uint32_t Q = KM_PIECE, FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  const int k = a.k;
  const uint32_t n = (uint32_t)(qb - qa);  // at most a chunk
  // superkmers are counted from s0; their k-mer offsets differ from qa by less
  // than 2^32 (a bin holds fewer k-mers), so the low words are enough
  const uint32_t *koff = reinterpret_cast<const uint32_t *>(a.koff + s0);
  const unsigned long long *desc = reinterpret_cast<const unsigned long long *>(a.desc + s0);
  const uint32_t ns = (uint32_t)(s_end - s0), qa32 = (uint32_t)qa;
  // end of superkmer base + lane, and its descriptor
  auto end_of = [&](uint32_t b) -> uint32_t { return b + lane < ns ? __ldg(koff + 2 * (b + lane) + 2) - qa32 : ~0u; };
  auto desc_of = [&](uint32_t b) -> uint64_t { return b + lane < ns ? __ldg(desc + b + lane) : 0ull; };
  uint32_t base = 0, pos0 = 0;             // first superkmer of the batch, next k-mer to take
  uint32_t kb = __ldg(koff) - qa32;        // start of superkmer base (modulo 2^32: at most its length before qa)
  uint32_t e = end_of(0);
  uint64_t ds = desc_of(0);
  const uint32_t upto = FULL >> (31 - lane);
  PackedWords<K> pw;
  bool have = false;
  while (pos0 < n) {
    const uint32_t ec = min(e, n), up = __shfl_up_sync(FULL, e, 1);
    const uint32_t ks = lane ? up : kb, st = lane ? max(up, pos0) : pos0;  // start, and first k-mer to take
    const uint32_t pieces = ec > st ? (ec - st + Q - 1) / Q : 0u;
    uint32_t P;
    const uint32_t S = warp_exclusive_scan(pieces, &P);
    const uint32_t nz = __ballot_sync(FULL, pieces > 0);
    const uint32_t all = __shfl_sync(FULL, ec, 31);  // the batch's k-mers end here
    // the rounds of this batch, and where the next one begins
    const uint32_t rounds = all == n || P < 32 ? (P + 31) / 32 : P / 32;
    const uint64_t off = ds >> 24;
    if (rounds * 32 >= P) {
      pos0 = all;
      base += 32;
      kb = __shfl_sync(FULL, e, 31);
    } else {
      const uint32_t j = 31 - __clz((int)__ballot_sync(FULL, pieces > 0 && S <= rounds * 32));
      pos0 = __shfl_sync(FULL, st + Q * (rounds * 32 - S), j);
      kb = __shfl_sync(FULL, ks, j);
      base += j;
    }
    e = end_of(base);
    ds = desc_of(base);
    const uint32_t first = nz ? __ffs((int)nz) - 1 : 0, run = nz >> first;
    const bool dense = (run & (run + 1)) == 0;  // superkmers without k-mers only before and after the others
    for (uint32_t r = 0; r < rounds; r++) {
      const uint32_t p = 32 * r + lane, rel = S - 32 * r;
      const uint32_t before = __popc(__ballot_sync(FULL, pieces > 0 && S < 32 * r));
      const uint32_t begins = __reduce_or_sync(FULL, pieces > 0 && rel < 32u ? 1u << rel : 0u);
      const uint32_t at = before + __popc(begins & upto) - 1;  // the piece's superkmer, of those with pieces
      const uint32_t j = dense ? first + at : __fns(nz, 0, (int)at + 1);
      const uint32_t pos = __shfl_sync(FULL, st - Q * S, j) + Q * p, end = __shfl_sync(FULL, ec, j);
      const uint32_t o = pos - __shfl_sync(FULL, ks, j);
      const uint64_t src = __shfl_sync(FULL, off, j);
      PackedWords<K> nw;
      nw.count = p < P ? min(Q, end - pos) : 0u;
      load_packed<K>(nw, a.packed, src, o);
      if (have) emit_piece<K>(pw, k, emit);
      pw = nw;
      have = true;
    }
  }
  if (have) emit_piece<K>(pw, k, emit);
}

// The k-mers of chunk c (bin b, j-th chunk of the bin) taken by warp w of W:
// [*qa, *qb) and the superkmer holding *qa.
GKC_DEV uint64_t warp_run(const ExpandArgs &a, uint64_t c, uint32_t b, uint64_t j, int w, int W, uint64_t *qa,
                          uint64_t *qb) {
  const uint64_t q0 = a.bin_kstart[b] + j * a.chunk_kmers;
  const uint64_t q1 = min(q0 + a.chunk_kmers, a.bin_kstart[b + 1]);
  const uint64_t per = ((q1 - q0 + W - 1) / W + 31) & ~31ull;
  *qa = min(q0 + per * w, q1);
  *qb = min(*qa + per, q1);
  const uint64_t lo = a.chunk_s0[c];
  const uint64_t hi = (c + 1 < a.chunk_base[b + 1]) ? a.chunk_s0[c + 1] : a.bin_start[b + 1] - 1;
  return warp_last_le(a.koff, lo, hi, *qa);
}

// ----------------------------------------------------------- 1. histogram

constexpr int HS_NT = 256;

// Expands every k-mer once (k-mer extraction and canonical form:
// kmer_counting.cu:99-112, 33-44) into `flat` and counts the coarse digits of
// each chunk of a bin's k-mers.  Each warp takes a contiguous share of the
// chunk and fills that share of `flat` front to back as its lanes emit keys,
// so the writes are coalesced; their order within it is of no use to anyone.
// 720 M 31-mers 5.9 -> 3.8 ms, 134.7 M 21-mers 1.02 -> 0.80, 112.8 M 63-mers 0.95 ->
// 0.68 against one k-mer a lane and round (pieces of 3, 4, 5, 8 k-mers: 4.10,
// 3.95, 3.85, 3.85 ms).
template <typename K>
__global__ void __launch_bounds__(HS_NT) k_bucket_hist(ExpandArgs a) {
  __shared__ uint32_t hist[1 << kCoarseMaxBits];
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  K *flat = reinterpret_cast<K *>(a.flat);
  const uint64_t n_chunks = a.chunk_base[a.nbins];
  const int key_bits = 2 * a.k;
  const int w = threadIdx.x >> 5;
  for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
    const uint32_t b = (uint32_t)warp_last_le(a.chunk_base, 0, a.nbins - 1, c);
    const uint64_t j = c - a.chunk_base[b];
    const int cb = (int)a.bin_bits[b];
    const uint32_t nd = 1u << cb;
    for (uint32_t d = threadIdx.x; d < nd; d += HS_NT) hist[d] = 0;
    __syncthreads();
    uint64_t qa, qb;
    const uint64_t s0 = warp_run(a, c, b, j, w, HS_NT / 32, &qa, &qb);
    if (qa < qb && qb <= a.keys_cap) {
      K *to = flat + qa;
      const uint32_t below = (1u << (threadIdx.x & 31u)) - 1u;
      warp_kmers<K>(a, qa, qb, s0, a.bin_start[b + 1], [&](K key, bool valid) {
        const uint32_t m = __ballot_sync(0xffffffffu, valid);
        if (valid) {
          to[__popc(m & below)] = key;
          atomicAdd(&hist[coarse_digit<K>(key, key_bits, cb)], 1u);
        }
        to += __popc(m);
      });
    } else if (qa < qb && (threadIdx.x & 31u) == 0) {
      atomicOr(a.err, ERR_CAPACITY);
    }
    __syncthreads();
    uint32_t *row = a.hist + a.hist_base[b] + j * nd;  // the chunk's row, digits contiguous
    uint32_t *tot = a.digit_total + ((uint64_t)b << a.max_bits);
    for (uint32_t d = threadIdx.x; d < nd; d += HS_NT) {
      const uint32_t v = hist[d];
      row[d] = v;
      if (v) atomicAdd(&tot[d], v);
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------------- 2. scan

// One CTA per bin: the exclusive scan of the bin's digit totals, and the digits
// packed into buckets: as many consecutive digits as hold at most bucket_keys
// keys, at least one.  So buckets are full although digits are uneven (the
// keys of a minimizer bin crowd at the minimizers' own values; with a bucket's
// bounds at multiples of a span, 22% of the keys of compressed long reads lay
// in buckets too large for k_bucket_sort).  Each digit's successor as the
// first of a bucket is found by a search, the firsts from digit 0 on by
// doubling.  The last CTA to finish adds up the bins' buckets.
constexpr int BS_NT = 1024;
__global__ void __launch_bounds__(BS_NT) k_bucket_scan(ExpandArgs a) {
  constexpr int DPT = (1 << kCoarseMaxBits) / BS_NT;
  __shared__ uint32_t tmp[64];
  __shared__ uint64_t tmp64[32];
  __shared__ uint32_t start[(1 << kCoarseMaxBits) + 1];
  __shared__ uint16_t jump[1 << kCoarseMaxBits];
  __shared__ uint8_t mark[(1 << kCoarseMaxBits) + 1];
  __shared__ bool done;
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  const int tid = threadIdx.x;
  for (uint32_t b = blockIdx.x; b < a.nbins; b += gridDim.x) {
    const uint32_t bits = a.bin_bits[b], nd = 1u << bits;
    // thread t holds the contiguous digits [t * DPT, t * DPT + DPT)
    const uint32_t d0 = tid * DPT;
    const uint32_t *total = a.digit_total + ((uint64_t)b << a.max_bits);
    uint32_t col[DPT], s = 0;
#pragma unroll
    for (int u = 0; u < DPT; u++) {
      col[u] = d0 + u < nd ? total[d0 + u] : 0u;
      s += col[u];
    }
    uint32_t tot;
    uint32_t at = block_exclusive_scan<BS_NT>(s, tmp, &tot);
#pragma unroll
    for (int u = 0; u < DPT; u++) {
      if (d0 + u < nd) {
        start[d0 + u] = at;
        mark[d0 + u] = d0 + u == 0;
      }
      at += col[u];
    }
    if (tid == 0) {
      start[nd] = tot;
      mark[nd] = 0;
    }
    __syncthreads();
    uint32_t next[DPT];
#pragma unroll
    for (int u = 0; u < DPT; u++) {
      const uint32_t d = d0 + u;
      next[u] = nd;
      if (d < nd) {
        uint32_t lo = d + 1, hi = nd;  // the last first digit of a next bucket that leaves this one small enough
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          if (start[mid] - start[d] <= a.bucket_keys) lo = mid; else hi = mid - 1;
        }
        next[u] = lo;
        jump[d] = (uint16_t)lo;
      }
    }
    __syncthreads();
    for (uint32_t r = 0; r < bits; r++) {  // marks after 2^r, .. jumps; next[u] = jump[d], nd stays nd
#pragma unroll
      for (int u = 0; u < DPT; u++)
        if (d0 + u < nd && mark[d0 + u]) mark[next[u]] = 1;
#pragma unroll
      for (int u = 0; u < DPT; u++)
        if (next[u] < nd) next[u] = jump[next[u]];
      __syncthreads();
#pragma unroll
      for (int u = 0; u < DPT; u++)
        if (d0 + u < nd) jump[d0 + u] = (uint16_t)next[u];
      __syncthreads();
    }
    uint32_t begins = 0;
#pragma unroll
    for (int u = 0; u < DPT; u++)
      if (d0 + u < nd && mark[d0 + u]) begins |= 1u << u;
    uint32_t n_units;
    uint32_t unit = block_exclusive_scan<BS_NT>(__popc(begins), tmp, &n_units);
#pragma unroll
    for (int u = 0; u < DPT; u++) {
      const uint32_t d = d0 + u;
      if (d < nd) {
        unit += (begins >> u) & 1u;
        a.lut[((uint64_t)b << a.max_bits) + d] = (uint16_t)(unit - 1);
        if ((begins >> u) & 1u) a.unit_start[((uint64_t)b << a.max_bits) + unit - 1] = start[d];
      }
    }
    if (tid == 0) a.bin_units[b] = n_units;
    __syncthreads();  // before the areas are written again
  }
  // the last CTA: first bucket of every bin
  if (tid == 0) {
    __threadfence();
    done = atomicAdd(a.scan_done, 1ull) == gridDim.x - 1;
  }
  __syncthreads();
  if (!done) return;
  __threadfence();
  uint64_t base = 0;
  for (uint32_t b0 = 0; b0 < a.nbins; b0 += BS_NT) {
    const uint32_t b = b0 + tid;
    uint64_t n;
    const uint64_t o = block_exclusive_scan_u64<BS_NT>(b < a.nbins ? *(volatile uint32_t *)(a.bin_units + b) : 0ull, tmp64, &n);
    if (b < a.nbins) a.bucket_base[b] = base + o;
    base += n;
  }
  if (tid == 0) a.bucket_base[a.nbins] = base;
}

// Each bucket's start and size, and every chunk's write offset per bucket,
// relative to the bin's first key: a warp per bucket adds up its digits in 32
// chunks at a time, one a lane, and leaves each offset at the count of the
// bucket's first digit.  (A thread per
// bucket walked hundreds of chunks of a large bin one after the other: 524 us
// where bins are uneven.)
__global__ void __launch_bounds__(kBucketOffsetThreads) k_bucket_offsets(ExpandArgs a, uint64_t *bucket_start,
                                                                         uint64_t *bucket_size) {
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  const uint64_t n_buckets = a.bucket_base[a.nbins];
  const uint32_t lane = threadIdx.x & 31u;
  for (uint64_t g = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; g < n_buckets;
       g += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t b = (uint32_t)warp_last_le(a.bucket_base, 0, a.nbins - 1, g);
    const uint32_t u = (uint32_t)(g - a.bucket_base[b]), nd = 1u << a.bin_bits[b];
    // the bucket's digits [lo, hi): a run in the ascending table
    const uint16_t *lut = a.lut + ((uint64_t)b << a.max_bits);
    uint32_t lo = 0, hi = nd;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (lut[mid] < u) lo = mid + 1; else hi = mid;
    }
    hi = lo;
    for (uint32_t h = nd; hi < h;) {
      const uint32_t mid = (hi + h) >> 1;
      if (lut[mid] <= u) hi = mid + 1; else h = mid;
    }
    const uint32_t *us = a.unit_start + ((uint64_t)b << a.max_bits) + u;
    uint32_t run = us[0];
    const uint64_t k0 = a.bin_kstart[b];
    const uint32_t end = u + 1 < a.bin_units[b] ? us[1] : (uint32_t)(a.bin_kstart[b + 1] - k0), size = end - run;
    if (lane == 0) {
      bucket_start[g] = k0 + run;
      bucket_size[g] = size;
      a.bucket_head[g] = 0;
      if (size >= a.big_min) a.big_list[atomicAdd(a.big_count, 1ull)] = (uint32_t)g;
    }
    if (size == 0) continue;
    const uint64_t nch = a.chunk_base[b + 1] - a.chunk_base[b];
    uint32_t *M = a.hist + a.hist_base[b];
    for (uint64_t j0 = 0; j0 < nch; j0 += 32) {
      const uint64_t jj = j0 + lane;
      uint32_t v = 0;
      if (jj < nch) {
#pragma unroll 4
        for (uint32_t d = lo; d < hi; d++) v += M[jj * nd + d];
      }
      uint32_t inc = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= (uint32_t)d) inc += t;
      }
      if (jj < nch) M[jj * nd + lo] = run + inc - v;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

// -------------------------------------------------------------- 3. scatter

// threads of a scatter CTA and keys of its tile: one or two CTAs' tiles and
// digit tables fill an SM's shared memory
__host__ __device__ constexpr int sc_threads(int ctas) { return 1024 / ctas; }
template <typename K> __host__ __device__ constexpr int sc_tile(int ctas) {
  return sizeof(K) == 16 ? 8192 : ctas == 1 ? 16384 : 7168;
}

// Moves every key of `flat` to its bucket.  Each CTA takes whole chunks, a
// tile of SC_TILE keys at a time: the tile is counting-sorted by bucket in
// shared memory (a key's rank within its bucket from a shared-memory atomic),
// then written out in that order, so the keys of one bucket leave as a
// contiguous run at the chunk's write offset for the bucket
// (from the scan) plus the bucket's keys of the chunk's earlier tiles.  Bound
// by the shared-memory accesses of phases that barriers separate, and by the
// partial sectors at both ends of a run: one CTA an SM with as large a tile as
// fits, or two that fill each other's gaps where runs stay long enough
// (kScatterPairBin).  A tile is loaded into the registers that the previous
// one's keys leave while that is written out.  720 M keys: 5.1 ms; 112.8 M of 16
// bytes: 1.17 -> 0.98 ms with two digit tables instead of three.
template <typename K, int CTAS>
__global__ void __launch_bounds__(sc_threads(CTAS), CTAS) k_bucket_scatter(ExpandArgs a) {
  constexpr int SC_THREADS = sc_threads(CTAS), SC_TILE = sc_tile<K>(CTAS), KPT = SC_TILE / SC_THREADS;
  constexpr int ND = 1 << kCoarseMaxBits;
  extern __shared__ __align__(16) uint8_t sc_smem[];
  K *S = reinterpret_cast<K *>(sc_smem);                      // the tile, by bucket
  uint32_t *gbase = reinterpret_cast<uint32_t *>(S + SC_TILE);  // next write offset of every bucket; in a tile less its start there
  uint32_t *toff = gbase + ND;                                // tile counts, then tile ends
  uint32_t *tmp = toff + ND;                                  // block scan
  uint16_t *Sd = reinterpret_cast<uint16_t *>(tmp + 64);      // buckets of S
  uint16_t *lut = Sd + SC_TILE;                               // bucket of every digit
  stamp_now(a.stamp);
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  K *keys = reinterpret_cast<K *>(a.keys);
  const K *flat = reinterpret_cast<const K *>(a.flat);
  const uint64_t n_chunks = a.chunk_base[a.nbins];
  const int key_bits = 2 * a.k;
  const int tid = threadIdx.x;
  for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
    const uint32_t b = (uint32_t)warp_last_le(a.chunk_base, 0, a.nbins - 1, c);
    const uint64_t j = c - a.chunk_base[b];
    const int cb = (int)a.bin_bits[b];
    const uint32_t nd = (uint32_t)(a.bucket_base[b + 1] - a.bucket_base[b]);  // buckets
    const uint64_t kbase = a.bin_kstart[b];
    const uint64_t q0 = kbase + j * a.chunk_kmers;
    const uint64_t q1 = min(q0 + a.chunk_kmers, a.bin_kstart[b + 1]);
    K xs[KPT];
    auto load = [&](uint64_t t0) {
#pragma unroll
      for (int u = 0; u < KPT; u++) {
        const uint64_t i = t0 + u * SC_THREADS + tid;
        if (i < q1) xs[u] = flat[i];
      }
    };
    load(q0);
    const uint32_t *row = a.hist + a.hist_base[b] + (j << cb);
    const uint16_t *glut = a.lut + ((uint64_t)b << a.max_bits);
    for (uint32_t d = tid; d < (1u << cb); d += SC_THREADS) {
      const uint16_t u = glut[d];
      lut[d] = u;
      if (d == 0 || glut[d - 1] != u) {  // the bucket's first digit holds its offset
        gbase[u] = row[d];
        toff[u] = 0;
      }
    }
    __syncthreads();
    for (uint64_t t0 = q0; t0 < q1; t0 += SC_TILE) {
      const uint32_t tn = (uint32_t)min((uint64_t)SC_TILE, q1 - t0);
      uint32_t rk[KPT];  // bucket << 16 | rank within it (< SC_TILE)
#pragma unroll
      for (int u = 0; u < KPT; u++) {
        if (u * SC_THREADS + tid < tn) {
          const uint32_t d = lut[coarse_digit<K>(xs[u], key_bits, cb)];
          rk[u] = (d << 16) | atomicAdd(&toff[d], 1u);
        }
      }
      __syncthreads();
      // inclusive scan of the tile counts, thread-contiguous buckets
      const uint32_t per = (nd + SC_THREADS - 1) / SC_THREADS, d0 = tid * per;
      uint32_t sum = 0;
      for (uint32_t d = d0; d < d0 + per && d < nd; d++) sum += toff[d];
      uint32_t total;
      uint32_t run = block_exclusive_scan<SC_THREADS>(sum, tmp, &total);
      for (uint32_t d = d0; d < d0 + per && d < nd; d++) {
        const uint32_t v = toff[d];
        gbase[d] -= run;
        run += v;
        toff[d] = run;
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < KPT; u++) {
        if (u * SC_THREADS + tid < tn) {
          const uint32_t d = rk[u] >> 16;
          const uint32_t at = toff[d] - 1u - (rk[u] & 0xFFFFu);
          S[at] = xs[u];
          Sd[at] = (uint16_t)d;
        }
      }
      __syncthreads();
      if (t0 + SC_TILE < q1) load(t0 + SC_TILE);
#pragma unroll 4
      for (uint32_t i = tid; i < tn; i += SC_THREADS) {
        const uint32_t d = Sd[i];
        const uint64_t slot = kbase + (uint32_t)(gbase[d] + i);
        if (slot < a.keys_cap) keys[slot] = S[i];
        else atomicOr(a.err, ERR_CAPACITY);
      }
      __syncthreads();
      for (uint32_t d = tid; d < nd; d += SC_THREADS) {  // for the next tile
        gbase[d] += toff[d];
        toff[d] = 0;
      }
      __syncthreads();  // also before the next chunk's tables
    }
  }
}

template <typename K> size_t bucket_scatter_smem_bytes(int ctas) {
  constexpr int ND = 1 << kCoarseMaxBits;
  static_assert(sc_tile<K>(1) % sc_threads(1) == 0 && sc_tile<K>(2) % sc_threads(2) == 0, "whole rounds");
  return (size_t)sc_tile<K>(ctas) * (sizeof(K) + 2) + 4 * (2 * ND + 64) + 2 * ND;
}
template size_t bucket_scatter_smem_bytes<uint64_t>(int);
template size_t bucket_scatter_smem_bytes<u128>(int);

// ---------------------------------------------------------------- 4. count

// CAP: the most distinct keys a bucket (or a slice of one) is counted with in
// shared memory; SLOTS: its hash table, at most two thirds full.
template <typename K> struct CountShape;
template <> struct CountShape<uint64_t> { static constexpr int NT = 512, CAP = 4096, SLOTS = 6144; };
template <> struct CountShape<u128> { static constexpr int NT = 512, CAP = 3072, SLOTS = 4608; };
constexpr int CC_SB_MAX = 12;        // sub-bucket bits of an oversized bucket
constexpr int CC_NSUB_MAX = 1 << CC_SB_MAX;
// k_bucket_sort: threads per CTA; a bucket is split into groups of at most
// GROUP keys on average, sorted by one warp with at most RMAX keys a lane.
template <typename K> struct SortShape;
template <> struct SortShape<uint64_t> { static constexpr int NT = 256, GROUP = 128, RMAX = 16, CTAS = 5; };
template <> struct SortShape<u128> { static constexpr int NT = 256, GROUP = 64, RMAX = 8, CTAS = 3; };
constexpr int CS_GROUPS = 64;       // most groups of a bucket
constexpr uint32_t CC_SPLIT_MAX = 512;  // groups of the sample sort (one per thread)
constexpr uint32_t CC_TICKETS = 4;     // buckets taken per ticket
constexpr int CC_LEVELS = 130;      // open levels of an oversized bucket: each one fixes at least a bit

// The hash table of a bucket and the areas of the sample sort of its distinct
// keys.  8-byte keys: the table holds the keys (claimed by compare-and-swap)
// and 16-bit counts beside them; an element's handle is its slot.
template <typename K> struct HashArea {
  static constexpr int CAP = CountShape<K>::CAP, SLOTS = CountShape<K>::SLOTS;
  K T[SLOTS];                  // keys; at the end the sorted keys
  uint32_t TC[SLOTS / 2];      // counts, two 16-bit halves a word; at the end the sorted counts
  union {
    uint64_t G[CAP];            // the distinct keys, group after group
    K spl[2 * CC_SPLIT_MAX];   // samples (runs of 32), then the sorted splitters
  } g;
  uint16_t L[CAP];             // handles of the distinct keys, then the group of every G entry
  uint16_t GC[CAP];            // counts in G order
};
// 16-byte keys (no 128-bit compare-and-swap in shared memory): the bucket's
// keys stay in shared memory and a slot holds (index of the key's first
// claimant + 1) and the count in one word; an element's handle is that index.
template <> struct HashArea<u128> {
  static constexpr int CAP = CountShape<u128>::CAP, SLOTS = CountShape<u128>::SLOTS;
  u128 A[CAP];                 // the bucket's keys
  uint32_t T[SLOTS];           // 0: free, else (index + 1) | count << 13
  union {
    struct {
      uint16_t G[CAP];         // handles of the distinct keys, group after group
      uint16_t GC[CAP];        // counts in G order
      uint16_t P[CAP];         // sorted order: G index of every output
    } m;
    u128 spl[2 * CC_SPLIT_MAX];
  } g;
  uint16_t L[CAP];             // slots of the distinct keys, then the group of every G entry
};
static_assert(CountShape<u128>::CAP < (1 << 13) - 1, "index + 1 fits 13 bits");

// A bucket split into groups by splitters taken from its keys.
template <typename K, int NT, int CAP_> struct SortArea {
  static constexpr int CAP = CAP_;
  K A[CAP];                             // keys, group after group; then each group's runs
  uint16_t C[CAP];                      // group of each key; then first position of each run in its sorted group
  K spl[CS_GROUPS];                     // splitters, in the order of a breadth-first search tree
  uint32_t gcnt[CS_GROUPS];             // keys per group
  uint32_t cur[CS_GROUPS];              // placement cursors
  uint16_t goff[NT / 32][CS_GROUPS + 2];  // group starts, a copy for every warp
  uint16_t gd[CS_GROUPS];               // runs per group
  uint32_t next, same;                  // next group to sort; one key fills too much of the bucket
};

// Hash table of k_bucket_sort, for buckets of few distinct 8-byte keys: small
// enough that five CTAs stay on an SM with the sort's areas for CAP keys.
struct DedupArea {
  static constexpr int SLOTS = 2560, CAP = 1280;
  uint64_t T[SLOTS];
  uint32_t TC[SLOTS / 2];               // counts, two 16-bit halves a word
  uint16_t L[CAP];                      // slots of the distinct keys
};

template <typename K>
struct CountSmem {
  static constexpr int CAP = CountShape<K>::CAP, NT = CountShape<K>::NT;
  union {
    HashArea<K> h;
    SortArea<K, CountShape<K>::NT, CountShape<K>::CAP> s;
    uint32_t sub[CC_NSUB_MAX];        // sub-bucket counts of an oversized bucket, then placement cursors
  } u;
  uint32_t goff[CC_SPLIT_MAX + 1];    // group counts, then starts
  uint32_t tmp[64];
  uint32_t hfill;
  int flag;
  uint64_t g, start, n;
  K red[64];                          // block min / max
  // open levels of an oversized bucket: keys up to `end` are in buffer `buf`,
  // in the order of the sb bits after the first cp
  uint64_t lend[CC_LEVELS];
  uint8_t lcp[CC_LEVELS], lsb[CC_LEVELS], lbuf[CC_LEVELS];
};
static_assert(sizeof(CountSmem<uint64_t>) <= 115712 && sizeof(CountSmem<u128>) <= 115712, "two CTAs per SM");

template <typename K> size_t bucket_count_smem_bytes() { return sizeof(CountSmem<K>); }
template <typename K> uint64_t bucket_count_cap() { return CountShape<K>::CAP; }
template uint64_t bucket_count_cap<uint64_t>();
template uint64_t bucket_count_cap<u128>();
template size_t bucket_count_smem_bytes<uint64_t>();
template size_t bucket_count_smem_bytes<u128>();

template <typename K> struct SortSmem {
  static constexpr int NT = SortShape<K>::NT;
  union {
    SortArea<K, NT, CountShape<K>::CAP> s;
    struct {
      DedupArea t;
      SortArea<K, NT, DedupArea::CAP> s;
    } d;                              // 8-byte keys only
  } u;
  uint32_t tmp[64];
  uint32_t hfill;
  int flag;
  uint64_t g, start;
  uint32_t n;
  uint64_t bg[CC_TICKETS], bstart[CC_TICKETS];  // the batch of buckets in hand
  uint32_t bn[CC_TICKETS];
  uint64_t pf_start;                  // the next bucket's keys, prefetched into L2
  uint32_t pf_n;
};
// an SM's 228 KB less 1 KB a CTA
template <typename K> constexpr size_t sort_smem_room() { return 228 * 1024 / SortShape<K>::CTAS - 1024; }
static_assert(sizeof(SortSmem<uint64_t>) <= sort_smem_room<uint64_t>() && sizeof(SortSmem<u128>) <= sort_smem_room<u128>(),
              "as many CTAs on an SM as the registers are shared out for");
template <typename K> size_t bucket_sort_smem_bytes() { return sizeof(SortSmem<K>); }
template size_t bucket_sort_smem_bytes<uint64_t>();
template size_t bucket_sort_smem_bytes<u128>();

// Exclusive scan of cnt[0, nsub) in place (thread-contiguous groups).
template <int NT>
GKC_DEV void scan_sub(uint32_t *cnt, uint32_t *tmp, uint32_t nsub) {
  const uint32_t per = (nsub + NT - 1) / NT, c0 = threadIdx.x * per;
  uint32_t s = 0;
  for (uint32_t jj = c0; jj < c0 + per && jj < nsub; jj++) s += cnt[jj];
  uint32_t tot;
  uint32_t run = block_exclusive_scan<NT>(s, tmp, &tot);
  for (uint32_t jj = c0; jj < c0 + per && jj < nsub; jj++) {
    const uint32_t v = cnt[jj];
    cnt[jj] = run;
    run += v;
  }
  __syncthreads();
}

template <typename K> GKC_DEV K shfl_xor_k(K v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
template <> GKC_DEV u128 shfl_xor_k<u128>(u128 v, int m) {
  const uint64_t lo = __shfl_xor_sync(0xffffffffu, (uint64_t)v, m);
  const uint64_t hi = __shfl_xor_sync(0xffffffffu, (uint64_t)(v >> 64), m);
  return ((u128)hi << 64) | lo;
}

// Smallest and largest of the block's (lo, hi) pairs, in every thread.
template <typename K, int NT>
GKC_DEV void block_minmax(CountSmem<K> &S, K &lo, K &hi) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    const K a = shfl_xor_k<K>(lo, m), b = shfl_xor_k<K>(hi, m);
    lo = a < lo ? a : lo;
    hi = b > hi ? b : hi;
  }
  if (lane == 0) {
    S.red[w] = lo;
    S.red[32 + w] = hi;
  }
  __syncthreads();
  lo = S.red[0];
  hi = S.red[32];
  for (int i = 1; i < NT / 32; i++) {
    lo = S.red[i] < lo ? S.red[i] : lo;
    hi = S.red[32 + i] > hi ? S.red[32 + i] : hi;
  }
  __syncthreads();
}

// ---- a bucket (or a slice of one) in shared memory: its keys aggregated in
// a hash table, so that only its distinct keys are sorted, then a sample sort
// of those.  Keys of a minimizer bin are far from uniform in their leading
// bases (those holding the minimizer near their start share them), so the
// sort takes its splitters from the keys: the table's slots are in hash
// order, which makes any fixed choice of them a random sample.

constexpr uint64_t HT_MAX_KEYS = 65535;  // counts are 16-bit (8-byte keys)
constexpr uint64_t HT_EMPTY = ~0ull;     // never a canonical key: the reverse complement of all-T is all-A

GKC_DEV uint32_t ht_slot(uint64_t x, uint32_t slots) {
  return __umulhi((uint32_t)((x * 0x9E3779B97F4A7C15ull) >> 32), slots);
}
GKC_DEV uint32_t ht_slot(u128 x, uint32_t slots) {
  const uint64_t y = (uint64_t)x * 0x9E3779B97F4A7C15ull + (uint64_t)(x >> 64) * 0xC2B2AE3D27D4EB4Full;
  return __umulhi((uint32_t)(y >> 32), slots);
}

// Slots for n keys: twice as many, whole rounds of the block.
template <typename K>
GKC_DEV uint32_t ht_slots(uint64_t n) {
  constexpr uint32_t NT = CountShape<K>::NT, SLOTS = CountShape<K>::SLOTS;
  return 2 * n >= SLOTS ? SLOTS : max(NT, ((uint32_t)(2 * n) + NT - 1) / NT * NT);
}

// Inserts the n keys into the table tab (S holds the fill counter and the
// flag); false when they hold more than CAP distinct ones (only possible for
// n > CAP).  A key whose first slot holds it is counted at once; the others
// (new ones, and those further down their chain) wait in the warp's queue
// until 32 of them are there, so that the chains' loop runs with full warps
// (720 M 31-mers at 30x: count stage 8.8 -> 8.1 ms).  A warp inserts at most 32
// keys between looks at the flag, so at most CAP + NT slots are ever taken and
// every probe chain ends at a free slot.
constexpr int TQ_ROWS = 4;                       // keys in flight per thread
constexpr uint32_t TQ_LEN = 32 * (TQ_ROWS + 1);  // a warp's queue: 31 keys left and a batch
template <int NT, uint32_t CAP, uint32_t SLOTS, typename SM>
GKC_DEV bool table_insert64(SM &S, uint64_t *tab, uint32_t *counts, uint64_t *queue, const uint64_t *src, uint64_t n,
                            uint32_t slots) {
  static_assert(CAP + NT < SLOTS, "a free slot is always left");
  const int tid = threadIdx.x;
  const uint32_t lane = tid & 31u, below = (1u << lane) - 1u;
  const bool limited = n > CAP;
  for (uint32_t i = tid; i < slots; i += NT) tab[i] = HT_EMPTY;
  for (uint32_t i = tid; i < slots / 2; i += NT) counts[i] = 0;
  if (tid == 0) {
    S.hfill = 0;
    S.flag = 0;
  }
  __syncthreads();
  volatile uint64_t *T = tab;
  uint64_t *Q = queue + TQ_LEN * (tid >> 5);
  uint32_t waiting = 0;  // the same in every lane
  auto given_up = [&] { return limited && __any_sync(0xffffffffu, *(volatile int *)&S.flag); };
  for (uint64_t i0 = 0; i0 < n && !given_up(); i0 += (uint64_t)TQ_ROWS * NT) {
    uint64_t xs[TQ_ROWS], cur[TQ_ROWS];
    uint32_t h[TQ_ROWS];
#pragma unroll
    for (int u = 0; u < TQ_ROWS; u++) {
      const uint64_t i = i0 + (uint64_t)u * NT + tid;
      xs[u] = i < n ? __ldcg(reinterpret_cast<const unsigned long long *>(src) + i) : HT_EMPTY;
    }
#pragma unroll
    for (int u = 0; u < TQ_ROWS; u++) {
      h[u] = ht_slot(xs[u], slots);
      cur[u] = T[h[u]];
    }
#pragma unroll
    for (int u = 0; u < TQ_ROWS; u++) {
      const bool have = xs[u] != HT_EMPTY, hit = cur[u] == xs[u];
      const uint32_t miss = __ballot_sync(0xffffffffu, have && !hit);
      if (have && hit) atomicAdd(&counts[h[u] >> 1], 1u << (16 * (h[u] & 1u)));
      if (have && !hit) Q[waiting + __popc(miss & below)] = xs[u];
      waiting += __popc(miss);
    }
    const bool last = i0 + (uint64_t)TQ_ROWS * NT >= n;
    while ((waiting >= 32 || (last && waiting > 0)) && !given_up()) {
      const uint32_t m = min(waiting, 32u);
      waiting -= m;
      __syncwarp();
      if (lane < m) {
        const uint64_t x = Q[waiting + lane];
        uint32_t s = ht_slot(x, slots);
        while (true) {
          uint64_t c = T[s];
          if (c == HT_EMPTY) {
            c = atomicCAS(reinterpret_cast<unsigned long long *>(tab + s), (unsigned long long)HT_EMPTY,
                          (unsigned long long)x);
            if (c == HT_EMPTY) {
              if (limited && atomicAdd(&S.hfill, 1u) + 1 > CAP) S.flag = 1;
              c = x;
            }
          }
          if (c == x) break;
          s = s + 1 == slots ? 0 : s + 1;
        }
        atomicAdd(&counts[s >> 1], 1u << (16 * (s & 1u)));
      }
      __syncwarp();
    }
  }
  __syncthreads();
  return !(limited && S.flag);
}
template <int NT>
GKC_DEV bool table_insert(CountSmem<uint64_t> &S, const uint64_t *src, uint64_t n, uint32_t slots) {
  static_assert(TQ_LEN * (NT / 32) <= CountShape<uint64_t>::CAP, "the groups' keys have room for the queues");
  return table_insert64<NT, CountShape<uint64_t>::CAP, CountShape<uint64_t>::SLOTS>(S, S.u.h.T, S.u.h.TC, S.u.h.g.G, src,
                                                                                  n, slots);
}
GKC_DEV bool slot_taken(const CountSmem<uint64_t> &S, uint32_t slot) { return S.u.h.T[slot] != HT_EMPTY; }
GKC_DEV uint64_t slot_key(const CountSmem<uint64_t> &S, uint32_t slot) { return S.u.h.T[slot]; }
GKC_DEV void put_member(CountSmem<uint64_t> &S, uint32_t at, uint32_t slot) {
  HashArea<uint64_t> &H = S.u.h;
  H.g.G[at] = H.T[slot];
  H.GC[at] = (uint16_t)(H.TC[slot >> 1] >> (16 * (slot & 1u)));
}
GKC_DEV uint64_t member_key(const CountSmem<uint64_t> &S, uint32_t i) { return S.u.h.g.G[i]; }
GKC_DEV void put_sorted(CountSmem<uint64_t> &S, uint32_t at, uint32_t i, uint64_t x) {
  HashArea<uint64_t> &H = S.u.h;  // the table is no longer read
  H.T[at] = x;
  reinterpret_cast<uint16_t *>(H.TC)[at] = H.GC[i];
}
GKC_DEV void get_sorted(const CountSmem<uint64_t> &S, uint32_t at, uint64_t &x, uint32_t &c) {
  x = S.u.h.T[at];
  c = reinterpret_cast<const uint16_t *>(S.u.h.TC)[at];
}

// 16-byte keys: n <= CAP, so they never hold too many distinct ones.
template <int NT>
GKC_DEV bool table_insert(CountSmem<u128> &S, const u128 *src, uint64_t n, uint32_t slots) {
  HashArea<u128> &H = S.u.h;
  const int tid = threadIdx.x;
  if (n > (uint64_t)CountShape<u128>::CAP) return false;
  constexpr int CAP = CountShape<u128>::CAP, EPT = CAP / NT;
  const uint32_t m = (uint32_t)n;
  {
    ulonglong2 v[EPT];
#pragma unroll
    for (int u = 0; u < EPT; u++)
      if (u * NT + tid < m) v[u] = __ldcg(reinterpret_cast<const ulonglong2 *>(src) + u * NT + tid);
    for (uint32_t i = tid; i < slots; i += NT) H.T[i] = 0;
#pragma unroll
    for (int u = 0; u < EPT; u++)
      if (u * NT + tid < m) H.A[u * NT + tid] = ((u128)v[u].y << 64) | v[u].x;
  }
  __syncthreads();
  volatile uint32_t *T = H.T;
  for (uint32_t i = tid; i < (uint32_t)n; i += NT) {
    const u128 x = H.A[i];
    uint32_t h = ht_slot(x, slots);
    while (true) {
      uint32_t cur = T[h];
      if (cur == 0) {
        cur = atomicCAS(&H.T[h], 0u, (i + 1) | (1u << 13));
        if (cur == 0) break;
      }
      if (H.A[(cur & 8191u) - 1] == x) {
        atomicAdd(&H.T[h], 1u << 13);
        break;
      }
      h = h + 1 == slots ? 0 : h + 1;
    }
  }
  __syncthreads();
  return true;
}
GKC_DEV bool slot_taken(const CountSmem<u128> &S, uint32_t slot) { return S.u.h.T[slot] != 0; }
GKC_DEV u128 slot_key(const CountSmem<u128> &S, uint32_t slot) { return S.u.h.A[(S.u.h.T[slot] & 8191u) - 1]; }
GKC_DEV void put_member(CountSmem<u128> &S, uint32_t at, uint32_t slot) {
  HashArea<u128> &H = S.u.h;
  const uint32_t t = H.T[slot];
  H.g.m.G[at] = (uint16_t)((t & 8191u) - 1);
  H.g.m.GC[at] = (uint16_t)(t >> 13);
}
GKC_DEV u128 member_key(const CountSmem<u128> &S, uint32_t i) { return S.u.h.A[S.u.h.g.m.G[i]]; }
GKC_DEV void put_sorted(CountSmem<u128> &S, uint32_t at, uint32_t i, u128) { S.u.h.g.m.P[at] = (uint16_t)i; }
GKC_DEV void get_sorted(const CountSmem<u128> &S, uint32_t at, u128 &x, uint32_t &c) {
  const uint32_t i = S.u.h.g.m.P[at];
  x = member_key(S, i);
  c = S.u.h.g.m.GC[i];
}

// Counts the n keys src[0, n) through the table and writes their sorted runs
// to the staging arrays at `out_at`; their number is left in S.hfill.
// Returns false, with nothing written, when there are more than CAP distinct
// keys (the caller then splits them).  Not inlined: it is called for whole
// buckets and for the slices of large ones.
template <typename K, int NT>
__device__ __noinline__ bool hash_count(CountSmem<K> &S, const SortCountArgs &a, const K *src, uint64_t n,
                                        uint64_t out_at) {
  constexpr int CAP = CountShape<K>::CAP;
  constexpr int EPT = CAP / NT;                     // elements per thread
  constexpr int SPT = CountShape<K>::SLOTS / NT;    // slots per thread
  static_assert(CAP % NT == 0 && CountShape<K>::SLOTS % NT == 0 && CC_SPLIT_MAX == NT, "whole rounds");
  static_assert(CountShape<K>::SLOTS <= 8192 && SPT <= 32, "13-bit slots, one mask per thread");
  const int tid = threadIdx.x, lane = tid & 31;
  HashArea<K> &H = S.u.h;
  const uint32_t slots = ht_slots<K>(n);
  if (!table_insert<NT>(S, src, n, slots)) {
    __syncthreads();
    return false;
  }
  // the taken slots, listed
  uint32_t mask = 0;
#pragma unroll
  for (int q = 0; q < SPT; q++) {
    const uint32_t slot = q * NT + tid;
    if (slot < slots && slot_taken(S, slot)) mask |= 1u << q;
  }
  uint32_t D;
  {
    uint32_t pos = block_exclusive_scan<NT>(__popc(mask), S.tmp, &D);
    while (mask) {
      const int q = __ffs(mask) - 1;
      mask &= mask - 1;
      H.L[pos++] = (uint16_t)(q * NT + tid);
    }
  }
  S.goff[tid] = 0;
  __syncthreads();
  // ns - 1 splitters, so groups of about D / ns in (4, 8] keys: ns samples,
  // runs of 32 sorted by warps, then ranked against every other run
  uint32_t ns = 1;
  while (8 * ns < D && ns < CC_SPLIT_MAX) ns <<= 1;
  if (ns > 1) {
    K x = ~(K)0;
    const uint32_t nw = max(ns, 32u);
    if ((uint32_t)tid < nw) {
      if ((uint32_t)tid < ns) x = slot_key(S, H.L[(uint32_t)tid * D / ns]);
#pragma unroll
      for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          const K y = shfl_xor_k<K>(x, stride);
          const bool keep_min = ((lane & stride) == 0) == ((lane & size) == 0);
          x = keep_min ? (y < x ? y : x) : (x < y ? y : x);
        }
      }
      H.g.spl[tid] = x;
    }
    __syncthreads();
    if ((uint32_t)tid < ns) {
      uint32_t rank = lane;
      for (uint32_t r = 0; r < ns; r += 32) {
        if (r == (uint32_t)(tid & ~31)) continue;
        const K *R = H.g.spl + r;
        uint32_t p = 0;
#pragma unroll
        for (uint32_t st = 16; st > 0; st >>= 1)
          if (R[p + st - 1] < x) p += st;
        rank += p + (R[p] < x ? 1u : 0u);
      }
      H.g.spl[CC_SPLIT_MAX + rank] = x;
    }
    __syncthreads();
  }
  // each key's group (the splitters below it) and place in the group
  uint32_t es[EPT], er[EPT];  // slot | group << 13; place
  const K *spl = H.g.spl + CC_SPLIT_MAX;
#pragma unroll
  for (int u = 0; u < EPT; u++) {
    const uint32_t i = u * NT + tid;
    if (i < D) {
      const uint32_t slot = H.L[i];
      const K x = slot_key(S, slot);
      uint32_t p = 0;
      for (uint32_t st = ns >> 1; st > 0; st >>= 1)
        if (spl[p + st - 1] < x) p += st;
      es[u] = slot | (p << 13);
      er[u] = atomicAdd(&S.goff[p], 1u);
    }
  }
  __syncthreads();
  {
    const uint32_t c = S.goff[tid];
    uint32_t tot;
    const uint32_t o = block_exclusive_scan<NT>(c, S.tmp, &tot);
    S.goff[tid] = o;
    if (tid == 0) S.goff[NT] = tot;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < EPT; u++) {
    const uint32_t i = u * NT + tid;
    if (i < D) {
      const uint32_t p = es[u] >> 13, at = S.goff[p] + er[u];
      put_member(S, at, es[u] & 8191u);
      H.L[at] = (uint16_t)p;  // the list of slots is no longer read
    }
  }
  __syncthreads();
  // rank within the group
  for (uint32_t i = tid; i < D; i += NT) {
    const uint32_t p = H.L[i], b0 = S.goff[p], b1 = S.goff[p + 1];
    const K x = member_key(S, i);
    uint32_t at = b0;
    for (uint32_t j = b0; j < b1; j++) at += member_key(S, j) < x ? 1u : 0u;
    put_sorted(S, at, i, x);
  }
  __syncthreads();
  K *out = reinterpret_cast<K *>(a.stage_keys);
  for (uint32_t i = tid; i < D; i += NT) {
    if (out_at + i < a.stage_cap) {
      K x;
      uint32_t c;
      get_sorted(S, i, x, c);
      out[out_at + i] = x;
      a.stage_counts[out_at + i] = c;
    } else {
      atomicOr(a.err, ERR_CAPACITY);
    }
  }
  if (tid == 0) S.hfill = D;
  __syncthreads();
  return true;
}


// ---- a bucket (or a slice of one) sorted without a table: split into groups
// of about 100 keys by splitters taken from its keys, each group sorted by a
// warp in registers.

template <typename K> GKC_DEV K shfl_up_k(K v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
template <typename K> GKC_DEV K shfl_k(K v, int l) { return __shfl_sync(0xffffffffu, v, l); }
template <> GKC_DEV u128 shfl_k<u128>(u128 v, int l) {
  const uint64_t lo = __shfl_sync(0xffffffffu, (uint64_t)v, l);
  const uint64_t hi = __shfl_sync(0xffffffffu, (uint64_t)(v >> 64), l);
  return ((u128)hi << 64) | lo;
}
// A key read once (L2 only: the staged runs overwrite it).
GKC_DEV uint64_t load_key(const uint64_t *p) { return __ldcg(reinterpret_cast<const unsigned long long *>(p)); }
GKC_DEV u128 load_key(const u128 *p) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(p));
  return ((u128)v.y << 64) | v.x;
}
template <> GKC_DEV u128 shfl_up_k<u128>(u128 v, int d) {
  const uint64_t lo = __shfl_up_sync(0xffffffffu, (uint64_t)v, d);
  const uint64_t hi = __shfl_up_sync(0xffffffffu, (uint64_t)(v >> 64), d);
  return ((u128)hi << 64) | lo;
}

// Orders x and y (ascending if asc), and the smaller or the larger of two keys.
template <typename K>
GKC_DEV void compare_exchange(K &x, K &y, bool asc) {
  const bool sw = (y < x) == asc;
  const K a = sw ? y : x;
  y = sw ? x : y;
  x = a;
}
GKC_DEV void compare_exchange(uint32_t &x, uint32_t &y, bool asc) {
  const uint32_t lo = min(x, y), hi = max(x, y);
  x = asc ? lo : hi;
  y = asc ? hi : lo;
}
template <typename K>
GKC_DEV K pick(K x, K y, bool smaller) { return (y < x) == smaller ? y : x; }
GKC_DEV uint32_t pick(uint32_t x, uint32_t y, bool smaller) { return smaller ? min(x, y) : max(x, y); }

// Bitonic merge of each lane's R keys (ascending if asc).
template <typename K, int R>
GKC_DEV void lane_merge(K (&v)[R], bool asc) {
#pragma unroll
  for (int stride = R / 2; stride > 0; stride >>= 1) {
#pragma unroll
    for (int r = 0; r < R; r++)
      if ((r & stride) == 0) compare_exchange(v[r], v[r + stride], asc);
  }
}

// Sorts the warp's 32 R keys ascending, sorted position e in lane e / R,
// register e % R: a bitonic network whose strides below R stay in a lane, so
// that only 15 of its steps exchange keys between lanes, whatever R.  The
// steps between lanes are a loop, not unrolled: straight-line networks of
// several sizes are more code than the instruction cache holds, and their
// fetches cost more than the network (count stage of 135 M keys: 7.1 ms
// unrolled, 3.4 ms with one size left).
template <typename K, int R>
GKC_DEV void warp_bitonic(K (&v)[R]) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int size = 2; size <= R; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll
      for (int r = 0; r < R; r++)
        if ((r & stride) == 0) compare_exchange(v[r], v[r + stride], size < R ? (r & size) == 0 : (lane & 1u) == 0);
    }
  }
#pragma unroll 1
  for (uint32_t lsize = 2; lsize <= 32; lsize <<= 1) {
    const bool asc = (lane & lsize) == 0;
#pragma unroll 1
    for (uint32_t lm = lsize >> 1; lm > 0; lm >>= 1) {
      const bool keep_min = ((lane & lm) == 0) == asc;
#pragma unroll
      for (int r = 0; r < R; r++) {
        v[r] = pick(v[r], shfl_xor_k<K>(v[r], (int)lm), keep_min);
      }
    }
    lane_merge<K, R>(v, asc);
  }
}

// The runs of the warp's sorted values (position e in lane e / R, register
// e % R; the first n): the distinct keys, made of the values by `key`, to A,
// the first position of each to C.  Returns their number.
template <typename K, typename V, int R, typename F>
GKC_DEV uint32_t warp_runs(const V (&v)[R], K *A, uint16_t *C, uint32_t b0, uint32_t n, F key) {
  const uint32_t lane = threadIdx.x & 31u;
  const V before = shfl_up_k<V>(v[R - 1], 1);
  uint32_t hb = 0;  // run heads among the first n positions
#pragma unroll
  for (int r = 0; r < R; r++) {
    const uint32_t e = lane * R + r;
    const V p = r == 0 ? before : v[r > 0 ? r - 1 : 0];
    if (e < n && (e == 0 || p != v[r])) hb |= 1u << r;
  }
  uint32_t D;
  uint32_t rank = b0 + warp_exclusive_scan(__popc(hb), &D);
#pragma unroll
  for (int r = 0; r < R; r++)
    if ((hb >> r) & 1u) {
      A[rank] = key(v[r]);
      C[rank] = (uint16_t)(lane * R + r);
      rank++;
    }
  __syncwarp();
  return D;
}

// Sorts A[b0, b0 + n), n <= 32 R, with the calling warp and leaves its runs
// there: the distinct keys in A, the first position of each in C.  Returns
// their number.  NARROW: 8-byte keys that share their upper word, as a group's
// keys do where k is small, are sorted by the lower one, a third of the
// network's instructions (count stage of 134.7 M distinct 21-mers 3.1 -> 2.6
// ms; both networks in the kernel cost 25-mers, whose groups seldom qualify,
// 3.9 -> 4.2, so the caller decides by k: narrow_groups).
template <typename K, int R, bool NARROW>
GKC_DEV uint32_t warp_sort_runs(K *A, uint16_t *C, uint32_t b0, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  K v[R];
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = r * 32 + lane < n ? A[b0 + r * 32 + lane] : ~(K)0;
  if constexpr (NARROW) {
    const uint32_t upper = (uint32_t)(A[b0] >> 32);
    uint32_t diff = 0;
#pragma unroll
    for (int r = 0; r < R; r++)
      if (r * 32 + lane < n) diff |= (uint32_t)(v[r] >> 32) ^ upper;
    if (!__any_sync(0xffffffffu, diff)) {
      uint32_t u[R];
#pragma unroll
      for (int r = 0; r < R; r++) u[r] = (uint32_t)v[r];
      warp_bitonic<uint32_t, R>(u);
      return warp_runs<K>(u, A, C, b0, n, [upper](uint32_t x) { return (K)upper << 32 | x; });
    }
  }
  warp_bitonic<K, R>(v);
  return warp_runs<K>(v, A, C, b0, n, [](K x) { return x; });
}

constexpr uint32_t SORT_REJECTED = ~0u;

// Counts the n <= CAP keys src[0, n) and writes their sorted runs to the
// staging arrays at `out_at`; returns their number, or SORT_REJECTED with
// nothing written when a group is too large for a warp (copies of one key
// cannot be split): the caller takes the hash table then.
//
// What bounds it is instruction issue and the shared-memory port, so it keeps
// the keys in registers where it can: 128 samples are sorted by one warp and
// every second to fourth (fewer groups: more) becomes a splitter, which keeps
// groups even whatever the keys' distribution; a key's group is found in a
// breadth-first tree (the nodes of a level are neighbours, so the lanes'
// loads meet in few banks); the groups' network needs 15 exchanges between
// lanes at any size.
// Keys in global memory: a run's count is its length.
template <typename K> struct GlobalKeys {
  const K *p;
  GKC_DEV K key(uint32_t i) const { return load_key(p + i); }
  GKC_DEV uint32_t count(K, uint32_t run) const { return run; }
};
// The distinct keys of the table: a key's count is found in its slot.
struct TableKeys {
  const DedupArea &t;
  GKC_DEV uint64_t key(uint32_t i) const { return t.T[t.L[i]]; }
  GKC_DEV uint32_t count(uint64_t x, uint32_t) const {
    uint32_t h = ht_slot(x, DedupArea::SLOTS);
    while (t.T[h] != x) h = h + 1 == DedupArea::SLOTS ? 0 : h + 1;  // x is in the table
    return (t.TC[h >> 1] >> (16 * (h & 1u))) & 0xFFFFu;
  }
};

template <typename K, int NT, bool NARROW, typename Src, typename Area>
GKC_DEV uint32_t sort_count(Area &S, const SortCountArgs &a, const Src &src, uint32_t n, uint64_t out_at) {
  constexpr int CAP = Area::CAP, W = NT / 32, RMAX = SortShape<K>::RMAX;
  static_assert(CAP <= 65535 && (CS_GROUPS * SortShape<K>::GROUP) >= CAP, "16-bit positions");
  const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
  int lg = 0;
  while (((uint32_t)SortShape<K>::GROUP << lg) < n || (lg < 3 && (32u << lg) < n)) lg++;  // few keys: a group for every warp
  const uint32_t G = 1u << lg;  // <= CS_GROUPS
  if (tid < CS_GROUPS) S.gcnt[tid] = lg == 0 && tid == 0 ? n : 0u;
  if (tid == NT - 1) {
    S.next = 0;
    if (lg == 0) S.same = 0;
  }
  if (lg > 0) {
    // splitter j (1 .. G - 1) is sample j * (samples / G) in order; as a node
    // of the tree it is number j >> (t + 1) of its level, t its trailing zero bits
    auto put = [&](uint32_t j, K x) {
      const int t = __ffs((int)j) - 1;
      S.spl[(1u << (lg - 1 - t)) + (j >> (t + 1))] = x;
    };
    if (G <= 8) {  // n > 32 here: 32 samples, each ranked by a few threads (the block waits for them)
      constexpr uint32_t T = NT / 32;
      if (tid < 32) S.A[tid] = src.key(tid * n / 32);
      if (tid == 0) S.same = 0;
      __syncthreads();
      const uint32_t i = tid / T;
      const K x = S.A[i];
      uint32_t r = 0;
#pragma unroll
      for (uint32_t j = tid % T; j < 32; j += T) {
        const K y = S.A[j];
        r += y < x || (y == x && j < i) ? 1u : 0u;
      }
#pragma unroll
      for (int d = 1; d < (int)T; d <<= 1) r += __shfl_xor_sync(0xffffffffu, r, d);
      if (tid % T == 0 && r > 0 && r * G % 32 == 0) put(r * G / 32, x);
    } else if (w == 0) {
      K v[4];
#pragma unroll
      for (int r = 0; r < 4; r++) v[r] = src.key((uint32_t)(r * 32 + lane) * n / 128);
      warp_bitonic<K, 4>(v);
      const uint32_t j = lane * 4 * G / 128;  // G <= 32: every (128 / G)th sample is a lane's first
#pragma unroll
      for (int r = 0; r < 4; r += 2) {        // G = 64: every second one
        const uint32_t e = lane * 4 + r, jj = r ? e * G / 128 : j;
        if (jj > 0 && jj * 128 == e * G) put(jj, v[r]);
      }
      // 32 equal samples: one key fills about a quarter of the bucket
      const K far = shfl_k<K>(v[0], min(lane + 8, 31u));
      const uint32_t any = __any_sync(0xffffffffu, lane < 24 && v[0] == far && n > 4u * 32 * RMAX);
      if (lane == 0) S.same = any;
    }
  }
  __syncthreads();
  if (S.same) {
    __syncthreads();
    return SORT_REJECTED;
  }
  // groups counted, each key's group kept in C
  if (lg > 0) {
#pragma unroll 4
    for (uint32_t i = tid; i < n; i += NT) {
      const K x = src.key(i);
      uint32_t node = 1;
      for (int l = 0; l < lg; l++) node = 2 * node + (x < S.spl[node] ? 0u : 1u);
      S.C[i] = (uint16_t)(node - G);
      atomicAdd(&S.gcnt[node - G], 1u);
    }
  }
  __syncthreads();
  uint16_t *goff = S.goff[w];
  {
    const uint32_t c0 = S.gcnt[2 * lane], c1 = S.gcnt[2 * lane + 1];
    uint32_t tot;
    const uint32_t o = warp_exclusive_scan(c0 + c1, &tot);
    goff[2 * lane] = (uint16_t)o;
    goff[2 * lane + 1] = (uint16_t)(o + c0);
    if (lane == 31) goff[CS_GROUPS] = (uint16_t)tot;
    if (w == 0) {
      S.cur[2 * lane] = o;
      S.cur[2 * lane + 1] = o + c0;
    }
    const bool large = __reduce_max_sync(0xffffffffu, max(c0, c1)) > 32u * RMAX;  // the same in every warp
    __syncthreads();
    if (large) return SORT_REJECTED;
  }
  if (lg > 0) {
#pragma unroll 4
    for (uint32_t i = tid; i < n; i += NT) S.A[atomicAdd(&S.cur[S.C[i]], 1u)] = src.key(i);
  } else {
    for (uint32_t i = tid; i < n; i += NT) S.A[i] = src.key(i);
  }
  __syncthreads();
  while (true) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(&S.next, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= G) break;
    const uint32_t b0 = goff[t], m = goff[t + 1] - b0;
    uint32_t d;
    if (m <= 64) d = warp_sort_runs<K, 2, NARROW>(S.A, S.C, b0, m);
    else if (m <= 128) d = warp_sort_runs<K, 4, NARROW>(S.A, S.C, b0, m);
    else if (RMAX <= 8 || m <= 256) d = warp_sort_runs<K, 8, NARROW>(S.A, S.C, b0, m);
    else d = warp_sort_runs<K, RMAX, NARROW>(S.A, S.C, b0, m);
    if (lane == 0) S.gd[t] = (uint16_t)d;
  }
  __syncthreads();
  const uint32_t d0 = 2 * lane < G ? S.gd[2 * lane] : 0u, d1 = 2 * lane + 1 < G ? S.gd[2 * lane + 1] : 0u;
  uint32_t D;
  const uint32_t o = warp_exclusive_scan(d0 + d1, &D);
  K *out = reinterpret_cast<K *>(a.stage_keys);
  const bool fits = out_at + n <= a.stage_cap;
  if (!fits && tid == 0) atomicOr(a.err, ERR_CAPACITY);
  for (uint32_t t = w; t < G; t += W) {
    const uint32_t at = __shfl_sync(0xffffffffu, o, t >> 1) + (t & 1u ? __shfl_sync(0xffffffffu, d0, t >> 1) : 0u);
    const uint32_t d = __shfl_sync(0xffffffffu, t & 1u ? d1 : d0, t >> 1);
    const uint32_t b0 = goff[t], m = goff[t + 1] - b0;
    for (uint32_t i = lane; i < d && fits; i += 32) {
      const uint32_t e = i + 1 < d ? S.C[b0 + i + 1] : m;
      const K x = S.A[b0 + i];
      out[out_at + at + i] = x;
      a.stage_counts[out_at + at + i] = src.count(x, e - S.C[b0 + i]);
    }
  }
  __syncthreads();
  return D;
}

// A bucket of n <= 65535 8-byte keys, its distinct keys (their number is
// returned; SORT_REJECTED when there are more than the table takes or sorted
// groups are too large) aggregated in the table first and then sorted.
template <int NT, bool NARROW>
__device__ __noinline__ uint32_t dedup_count(SortSmem<uint64_t> &S, const SortCountArgs &a, const uint64_t *src,
                                             uint32_t n, uint64_t out_at) {
  DedupArea &H = S.u.d.t;
  constexpr int SPT = DedupArea::SLOTS / NT;
  static_assert(DedupArea::SLOTS % NT == 0 && SPT <= 32, "one mask per thread");
  static_assert(TQ_LEN * (NT / 32) <= DedupArea::CAP, "the sort's keys have room for the queues");
  if (!table_insert64<NT, DedupArea::CAP, DedupArea::SLOTS>(S, H.T, H.TC, S.u.d.s.A, src, n, DedupArea::SLOTS)) {
    __syncthreads();
    return SORT_REJECTED;
  }
  uint32_t mask = 0;
#pragma unroll
  for (int q = 0; q < SPT; q++)
    if (H.T[q * NT + threadIdx.x] != HT_EMPTY) mask |= 1u << q;
  uint32_t D;
  uint32_t pos = block_exclusive_scan<NT>(__popc(mask), S.tmp, &D);
  while (mask) {
    const int q = __ffs(mask) - 1;
    mask &= mask - 1;
    H.L[pos++] = (uint16_t)(q * NT + threadIdx.x);
  }
  __syncthreads();
  return sort_count<uint64_t, NT, NARROW>(S.u.d.s, a, TableKeys{H}, D, out_at);
}
template <int NT, bool NARROW>
GKC_DEV uint32_t dedup_count(SortSmem<u128> &, const SortCountArgs &, const u128 *, uint32_t, uint64_t) {
  return SORT_REJECTED;
}

template <typename K, int NT>
__device__ __noinline__ uint32_t slice_count(SortArea<K, NT, CountShape<K>::CAP> &S, const SortCountArgs &a,
                                             const K *src, uint32_t n, uint64_t out_at) {
  return sort_count<K, NT, false>(S, a, GlobalKeys<K>{src}, n, out_at);
}

// Buckets of at most CAP keys, persistent, taken by ticket.  Those that
// sort_count rejects join the list of large ones (k_bucket_open).  256
// threads and 45 KB (58 KB), so that five CTAs (three for 16-byte keys) on an SM hide
// each other's barriers.  Count stage (with the two kernels below) on a
// B200, against counting each bucket in a 4096-slot hash table with a merge
// sort, or by insertion and warp sorts of 4096 fixed digits: 720 M 31-mers at
// 30x 8.1 ms (14.7), 134.7 M mostly distinct 21-mers 2.7 ms (10.6), 150.9 M
// 25-mers of compressed long reads 3.8 ms (14.8), 112.8 M 63-mers 2.8 ms (9.9).
template <typename K, bool NARROW>
__global__ void __launch_bounds__(SortShape<K>::NT, SortShape<K>::CTAS) k_bucket_sort(SortCountArgs a) {
  constexpr int NT = SortShape<K>::NT;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  SortSmem<K> &S = *reinterpret_cast<SortSmem<K> *>(smem_raw);
  const K *keys = reinterpret_cast<const K *>(a.keys);
  const int tid = threadIdx.x;
  stamp_now(a.stamp);
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  const uint64_t n_buckets = a.bucket_base[a.nbins];
  // several buckets per ticket only where every CTA gets many: with few, a
  // batch would leave CTAs without any
  const uint32_t batch = n_buckets >= 16ull * CC_TICKETS * gridDim.x ? CC_TICKETS : 1;
  uint32_t bi = 0, bm = 0;          // thread 0: next and end of its batch of buckets
  uint32_t repeats = 0;             // 8-byte keys: the same in every thread of the block
  uint32_t skip = 0;                // thread 0, 16-byte keys: buckets to list before one is sorted again
  uint32_t often = 0;               // thread 0, 16-byte keys: how many were listed last (0: the last one sorted held few repeats)
  while (true) {
    if (tid == 0) while (true) {
      while (bi == bm) {  // a new batch, without the large ones
        const uint64_t t0 = atomicAdd(a.ticket, (unsigned long long)batch);
        bi = bm = 0;
        if (t0 >= n_buckets) {
          S.bg[0] = n_buckets;
          S.bn[0] = 0;
          S.bstart[0] = 0;
          bm = 1;
          break;
        }
        uint64_t sz[CC_TICKETS], st[CC_TICKETS];
#pragma unroll
        for (uint32_t j = 0; j < CC_TICKETS; j++) {
          const bool in = j < batch && t0 + j < n_buckets;
          sz[j] = in ? a.bucket_size[t0 + j] : ~0ull;
          st[j] = in ? a.bucket_start[t0 + j] : 0;
        }
#pragma unroll
        for (uint32_t j = 0; j < CC_TICKETS; j++)
          if (sz[j] == 0) {
            a.bucket_d[t0 + j] = 0;
          } else if (sz[j] < a.big_min) {
            S.bg[bm] = t0 + j;
            S.bstart[bm] = st[j];
            S.bn[bm] = (uint32_t)sz[j];
            bm++;
          }
      }
      if (sizeof(K) == 8 || skip == 0 || S.bg[bi] >= n_buckets) break;
      a.big_list[atomicAdd(a.big_count, 1ull)] = (uint32_t)S.bg[bi++];
      skip--;
    }
    if (tid == 0) {
      S.g = S.bg[bi];
      S.start = S.bstart[bi];
      S.n = S.bn[bi];
      bi++;
      S.pf_n = bi < bm && !often ? S.bn[bi] : 0;
      S.pf_start = bi < bm ? S.bstart[bi] : 0;
    }
    __syncthreads();
    const uint64_t g = S.g, start = S.start;
    const uint32_t n = S.n;
    if (g >= n_buckets) break;
    {
      constexpr int KPL = 128 / (int)sizeof(K);
      const uint64_t ps = S.pf_start, pe = ps + S.pf_n;
      for (uint64_t i = ps + (uint64_t)tid * KPL; i < pe; i += (uint64_t)NT * KPL) prefetch_l2(keys + i);
    }
    // Which way is faster depends on how often keys repeat, which changes
    // little from bucket to bucket: the last bucket's share decides.  8-byte
    // keys: the table first where two keys in three or more are repeats.
    // 16-byte keys have no table here: the next 15 buckets go to the list,
    // unseen, then one is sorted again; 31 and 63 while that holds repeats
    // too (count stage of 112.8 M 63-mers 2.84 ms with 15 each time, 2.71 so).
    uint32_t D = SORT_REJECTED;
    if (sizeof(K) == 8 && repeats) D = dedup_count<NT, NARROW>(S, a, keys + start, n, start);
    if (D == SORT_REJECTED) D = sort_count<K, NT, NARROW>(S.u.s, a, GlobalKeys<K>{keys + start}, n, start);
    const bool most = D != SORT_REJECTED && 3 * D <= n;
    if (sizeof(K) == 8) repeats = most;
    if (tid == 0) {  // sort_count's barriers lie between the reads of S.g and the next bucket's
      if (D != SORT_REJECTED) a.bucket_d[g] = D;
      else a.big_list[atomicAdd(a.big_count, 1ull)] = (uint32_t)g;
      if (sizeof(K) == 16) {
        often = most ? min(max(2 * often + 1, 15u), 63u) : 0;
        skip = often;
      }
    }
  }
}

// What open_level found: the digit's place; the only key (where there is just
// one); the keys left, and the copies left out of them and of which key.
template <typename K> struct Opened {
  int cp, sb;
  K key, crowd;
  uint64_t kept;
  uint32_t extra;
};

// A key that fills a quarter of [b, e) or more, by 32 samples: in S.red[0],
// S.flag tells whether there may be one.  Barriers around it are the caller's.
template <typename K>
GKC_DEV void crowd_sample(CountSmem<K> &S, const K *from, uint64_t b, uint64_t e) {
  if (threadIdx.x >= 32) return;
  const uint32_t lane = threadIdx.x;
  const K x = load_key(from + b + (e - b) * lane / 32);
  uint32_t same = 0;
#pragma unroll 4
  for (int l = 0; l < 32; l++) same += shfl_k<K>(x, l) == x ? 1u : 0u;
  const uint32_t most = __reduce_max_sync(0xffffffffu, same << 5 | lane);
  if (lane == (most & 31u)) {
    S.red[0] = x;
    S.flag = (most >> 5) >= 8;
    S.tmp[0] = 0;
  }
}

// Opens the keys [b, e) of an oversized bucket (`from`: its keys, `to`: the
// same range of the other buffer): sorted into `to` by the up to 12 bits after
// their common prefix, so that at least the first differing bit is among
// them.  Returns false when all keys are equal (o->key), nothing moved then.
// Buckets grow large because keys crowd, often at one key, whose copies would
// be moved from level to level by one CTA: of a key that is a quarter of them or
// more one copy is left in, and the caller adds the others to its run (15 M
// bases, 98.5% A: k 21 in 31 bins 34.6 -> 15.6 ms, k 31 in 256 51.8 -> 18.4).
template <typename K, int NT>
__device__ __noinline__ bool open_level(CountSmem<K> &S, const K *from, K *to, uint64_t b, uint64_t e, Opened<K> *o) {
  constexpr int U = sizeof(K) == 8 ? 8 : 4;  // keys in flight per thread
  const int tid = threadIdx.x;
  uint32_t *sub = S.u.sub;
  bool crowded = false;  // the same in every thread
  K crowd = 0;
  if (e - b > 4 * (uint64_t)CountShape<K>::CAP) {
    crowd_sample<K>(S, from, b, e);
    __syncthreads();
    crowded = S.flag;
    crowd = S.red[0];
    __syncthreads();
  }
  K lo = ~(K)0, hi = 0;
  uint32_t copies = 0;
#pragma unroll U
  for (uint64_t i = b + tid; i < e; i += NT) {
    const K x = load_key(from + i);
    lo = x < lo ? x : lo;
    hi = x > hi ? x : hi;
    copies += x == crowd ? 1u : 0u;
  }
  if (crowded) {
    copies = __reduce_add_sync(0xffffffffu, copies);
    if ((tid & 31) == 0) atomicAdd(&S.tmp[0], copies);
  }
  block_minmax<K, NT>(S, lo, hi);
  o->key = lo;
  if (lo == hi) return false;
  copies = crowded ? S.tmp[0] : 0u;
  crowded = copies >= (e - b) / 4 && copies > 16;
  int cp, sb;
  prefix_split<K>(lo, hi, e - b, CC_SB_MAX, &cp, &sb);
  const uint32_t nsub = 1u << sb;
  for (uint32_t jj = tid; jj < nsub; jj += NT) sub[jj] = 0;
  __syncthreads();
  if (crowded && tid == 0) atomicAdd(&sub[prefix_digit<K>(crowd, cp, sb)], 1u);
#pragma unroll U
  for (uint64_t i = b + tid; i < e; i += NT) {
    const K x = load_key(from + i);
    if (!crowded || x != crowd) atomicAdd(&sub[prefix_digit<K>(x, cp, sb)], 1u);
  }
  __syncthreads();
  scan_sub<NT>(sub, S.tmp, nsub);
  if (crowded && tid == 0) to[b + atomicAdd(&sub[prefix_digit<K>(crowd, cp, sb)], 1u)] = crowd;
#pragma unroll U
  for (uint64_t i = b + tid; i < e; i += NT) {
    const K x = load_key(from + i);
    if (!crowded || x != crowd) to[b + atomicAdd(&sub[prefix_digit<K>(x, cp, sb)], 1u)] = x;
  }
  __syncthreads();
  o->cp = cp;
  o->sb = sb;
  o->crowd = crowd;
  o->extra = crowded ? copies - 1 : 0u;
  o->kept = e - b - o->extra;
  return true;
}

// Adds the copies left out of key x to its run, one of the staged runs [lo, hi).
// By one thread.
template <typename K>
GKC_DEV void add_copies(const SortCountArgs &a, uint64_t lo, uint64_t hi, K x, uint32_t extra) {
  const K *keys = reinterpret_cast<const K *>(a.stage_keys);
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (load_key(keys + mid) < x) lo = mid + 1; else hi = mid;
  }
  if (lo < a.stage_cap && load_key(keys + lo) == x) a.stage_counts[lo] = __ldcg(a.stage_counts + lo) + extra;
  else atomicOr(a.err, ERR_BOUNDS);  // not possible: one copy was left in
}

// Counts the keys [pos, end) of an oversized bucket (offsets from its key range
// `start`; `from`: the buffer that holds them) and stages their runs from
// start + pos on; returns their number.  The keys are sorted by digit into the
// other buffer, then counted in slices of at most CAP keys in key order; a
// digit of more keys is opened in turn, back into the first buffer.  Buffer 0
// is the bucket's own key range, buffer 1 the same range of the scratch array
// (the result's key array, written only after the count).  The staged runs
// never pass the keys already counted.
template <typename K>
__device__ __noinline__ uint64_t count_range(CountSmem<K> &S, const SortCountArgs &a, uint64_t start, uint64_t pos,
                                             uint64_t end, int from) {
  constexpr int NT = CountShape<K>::NT, CAP = CountShape<K>::CAP;
  const int tid = threadIdx.x;
  K *const buf[2] = {reinterpret_cast<K *>(a.keys) + start, reinterpret_cast<K *>(a.scratch) + start};
  start += pos;          // of the staged runs
  uint64_t run = 0;      // [pos, end): what is opened next; the same in every thread
  int level = 0;
  while (true) {
    Opened<K> o;
    if (open_level<K, NT>(S, buf[from], buf[from ^ 1], pos, end, &o)) {
      if (level == CC_LEVELS) {  // not possible: every level fixes a bit of the key
        if (tid == 0) atomicOr(a.err, ERR_BOUNDS);
        break;
      }
      if (tid == 0) {
        S.lend[level] = pos + o.kept;
        S.lcp[level] = (uint8_t)o.cp;
        S.lsb[level] = (uint8_t)o.sb;
        S.lbuf[level] = (uint8_t)((from ^ 1) | (o.extra ? 2 : 0));
        if (o.extra) {  // more than 16, so there is room where the copies were
          K *x = buf[from ^ 1] + pos + o.kept;
          x[0] = o.crowd;
          x[1] = (K)o.extra;
          x[2] = (K)run;
          x[3] = (K)end;
        }
      }
      level++;
    } else {  // one key
      if (tid == 0) {
        if (start + run < a.stage_cap) {
          reinterpret_cast<K *>(a.stage_keys)[start + run] = o.key;
          a.stage_counts[start + run] = (uint32_t)(end - pos);
        } else {
          atomicOr(a.err, ERR_CAPACITY);
        }
      }
      run++;
      pos = end;
    }
    __syncthreads();
    // slices of the innermost open level, until one has to be opened
    bool open = false;
    while (level > 0 && !open) {
      const uint64_t lend = S.lend[level - 1];
      if (pos == lend) {
        level--;
        const uint32_t lb = S.lbuf[level];
        if (lb & 2u) {
          const K *x = buf[lb & 1u] + lend;
          if (tid == 0) add_copies<K>(a, start + (uint64_t)load_key(x + 2), start + run, load_key(x), (uint32_t)load_key(x + 1));
          pos = (uint64_t)load_key(x + 3);
        }
        continue;
      }
      const int lcp = S.lcp[level - 1], lsb = S.lsb[level - 1];
      from = S.lbuf[level - 1] & 1;
      const K *src = buf[from];
      end = lend;
      if (lend - pos > (uint64_t)CAP) {
        // the digit of the first key that does not fit ends the slice
        const uint32_t d = prefix_digit<K>(load_key(src + pos + CAP), lcp, lsb);
        uint64_t l = pos, h = pos + CAP;  // first key of digit d
        while (l < h) {
          const uint64_t mid = (l + h) >> 1;
          if (prefix_digit<K>(load_key(src + mid), lcp, lsb) < d) l = mid + 1; else h = mid;
        }
        end = l;
        if (l == pos) {  // digit d alone is larger than a slice
          l = pos + CAP + 1;
          h = lend;
          while (l < h) {
            const uint64_t mid = (l + h) >> 1;
            if (prefix_digit<K>(load_key(src + mid), lcp, lsb) <= d) l = mid + 1; else h = mid;
          }
          end = l;
          open = true;
          break;
        }
      }
      const uint32_t ns = (uint32_t)(end - pos);
      uint32_t D = slice_count<K, NT>(S.u.s, a, src + pos, ns, start + run);
      if (D == SORT_REJECTED) {
        hash_count<K, NT>(S, a, src + pos, ns, start + run);  // at most CAP keys: never too many
        D = S.hfill;
        __syncthreads();
      }
      run += D;
      pos = end;
    }
    if (!open) break;
    __syncthreads();  // the level's parameters are read before a new one is written
  }
  return run;
}

// The listed buckets: larger than CAP, or rejected by k_bucket_sort.  A bucket
// that the table takes is counted here; another is sorted by digit into the
// scratch array and its slices of at most CAP keys (and each digit of more)
// become tasks of k_bucket_slices, so that a large bucket is counted by many
// CTAs (by one, the largest of 150.9 M 25-mers kept the chip waiting: 1.9 ms).
template <typename K>
__global__ void __launch_bounds__(CountShape<K>::NT, 2) k_bucket_open(SortCountArgs a) {
  constexpr int NT = CountShape<K>::NT, CAP = CountShape<K>::CAP;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  CountSmem<K> &S = *reinterpret_cast<CountSmem<K> *>(smem_raw);
  K *keys = reinterpret_cast<K *>(a.keys);
  const int tid = threadIdx.x;
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  const uint64_t n_big = *a.big_count;
  int hash_skip = 0;                // the same in every thread of the block
  while (true) {
    if (tid == 0) {
      const uint64_t t = atomicAdd(a.big_ticket, 1ull);
      S.g = t < n_big ? a.big_list[t] : ~0ull;
      if (t < n_big) {
        S.start = a.bucket_start[S.g];
        S.n = a.bucket_size[S.g];
      }
    }
    __syncthreads();
    const uint64_t g = S.g;
    if (g == ~0ull) break;
    const uint64_t start = S.start, n = S.n;
    // the whole bucket through the table: always possible up to CAP keys,
    // else tried unless the last larger one had too many distinct keys
    bool done = false;
    if (n <= (uint64_t)CAP) {
      done = hash_count<K, NT>(S, a, keys + start, n, start);
    } else if (sizeof(K) == 8 && n <= HT_MAX_KEYS) {
      if (hash_skip == 0) {
        done = hash_count<K, NT>(S, a, keys + start, n, start);
        if (!done) hash_skip = 8;
      } else {
        hash_skip--;
      }
    }
    if (done) {
      if (tid == 0) a.bucket_d[g] = S.hfill;
      __syncthreads();
      continue;
    }
    Opened<K> o;
    if (!open_level<K, NT>(S, keys + start, reinterpret_cast<K *>(a.scratch) + start, 0, n, &o)) {
      if (tid == 0) {  // one key
        reinterpret_cast<K *>(a.stage_keys)[start] = o.key;  // start + n <= stage_cap: the keys were there
        a.stage_counts[start] = (uint32_t)n;
        a.bucket_d[g] = 1;
      }
      __syncthreads();
      continue;
    }
    // S.u.sub[d] is now the end of digit d: as many digits a task as fit CAP
    // keys, at least one; the first digits of the tasks are listed
    uint16_t *first = reinterpret_cast<uint16_t *>(S.u.sub + CC_NSUB_MAX);
    static_assert(sizeof(S.u) >= CC_NSUB_MAX * 6, "the list fits after the digits");
    if (tid == 0) {
      const uint32_t nsub = 1u << o.sb;
      uint32_t m = 0, d = 0, s0 = 0;
      while (d < nsub) {
        uint32_t lo = d + 1, hi = nsub;
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          if (S.u.sub[mid - 1] - s0 <= (uint32_t)CAP) lo = mid; else hi = mid - 1;
        }
        if (S.u.sub[lo - 1] != s0) first[m++] = (uint16_t)d;
        s0 = S.u.sub[lo - 1];
        d = lo;
      }
      S.hfill = m;
      S.n = atomicAdd(a.task_count, (unsigned long long)m);
      a.bucket_d[g] = 0;
      if (S.n + m > a.task_cap) atomicOr(a.err, ERR_BOUNDS);  // not possible: at most 3 n / CAP + 1 tasks
      else a.bucket_head[g] = (uint32_t)S.n + 1;
    }
    __syncthreads();
    const uint32_t m = S.hfill;
    const uint64_t t0 = S.n;
    for (uint32_t i = tid; i < m && t0 + m <= a.task_cap; i += NT) {
      const uint32_t b = first[i] ? S.u.sub[first[i] - 1] : 0u;
      const uint32_t e = i + 1 < m ? S.u.sub[first[i + 1] - 1] : (uint32_t)o.kept;
      // the slice with the key whose copies were left out: it and they, behind the bucket's keys
      const uint32_t d = o.extra ? prefix_digit<K>(o.crowd, o.cp, o.sb) : 0u;
      const bool crowd = o.extra && first[i] <= d && (i + 1 == m || d < first[i + 1]);
      if (crowd) {
        K *x = reinterpret_cast<K *>(a.scratch) + start + n;
        x[-1] = o.crowd;
        x[-2] = (K)o.extra;
      }
      a.tasks[t0 + i] = make_uint4((uint32_t)g, b, e - b, crowd ? 1u : 0u);
    }
    __syncthreads();
  }
}

// The tasks of k_bucket_open: slices of an opened bucket, each staged over its
// own keys; k_compact_runs puts them together.
template <typename K>
__global__ void __launch_bounds__(CountShape<K>::NT, 2) k_bucket_slices(SortCountArgs a) {
  constexpr int NT = CountShape<K>::NT, CAP = CountShape<K>::CAP;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  CountSmem<K> &S = *reinterpret_cast<CountSmem<K> *>(smem_raw);
  if (*a.err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE | ERR_BOUNDS)) return;
  const uint64_t n_tasks = *a.task_count;
  while (true) {
    if (threadIdx.x == 0) S.g = atomicAdd(a.task_ticket, 1ull);
    __syncthreads();
    const uint64_t t = S.g;
    if (t >= n_tasks) break;
    const uint4 task = a.tasks[t];
    const uint64_t start = a.bucket_start[task.x];
    uint64_t D;
    if (task.z <= (uint32_t)CAP) {
      const K *src = reinterpret_cast<const K *>(a.scratch) + start + task.y;
      const uint32_t d = slice_count<K, NT>(S.u.s, a, src, task.z, start + task.y);
      if (d != SORT_REJECTED) {
        D = d;
      } else {
        hash_count<K, NT>(S, a, src, task.z, start + task.y);  // at most CAP keys: never too many
        D = S.hfill;
      }
    } else {
      D = count_range<K>(S, a, start, task.y, (uint64_t)task.y + task.z, 1);
    }
    __syncthreads();  // S.g and S.hfill are read
    if (threadIdx.x == 0) {
      if (task.w) {
        const K *x = reinterpret_cast<const K *>(a.scratch) + start + a.bucket_size[task.x];
        add_copies<K>(a, start + task.y, start + task.y + D, load_key(x - 1), (uint32_t)load_key(x - 2));
      }
      a.tasks[t].w = (uint32_t)D;
      atomicAdd(&a.bucket_d[task.x], (unsigned long long)D);
    }
  }
}

// Moves each bucket's staged runs to its final offset (the exclusive scan of
// the buckets' distinct counts); bin_out[b] is the offset of the bin's first
// bucket.  A warp per bucket where there are buckets for every warp, else
// several warps share one; four entries a lane in flight.  An opened bucket's
// runs lie task by task.
template <typename K>
__global__ void k_compact_runs(const K *stage_keys, const uint32_t *stage_counts, const uint64_t *bucket_start,
                               const unsigned long long *bucket_d, const uint64_t *bucket_out,
                               const uint64_t *bucket_base, uint32_t nbins, K *out_keys, uint32_t *out_counts,
                               uint64_t *bin_out, const uint32_t *bucket_head, const uint4 *tasks,
                               const unsigned long long *task_count, const uint32_t *err) {
  if (*err & (ERR_CAPACITY | ERR_BAD_READ | ERR_BIN_TOO_LARGE)) return;
  constexpr int U = 4;
  const uint64_t nb = bucket_base[nbins];
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = t; b <= nbins; b += nt) bin_out[b] = bucket_out[bucket_base[b]];
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warps = nt >> 5;
  const uint32_t parts = nb == 0 || nb >= warps ? 1 : (uint32_t)min(warps / nb, (uint64_t)32);
  for (uint64_t x = t >> 5; x < nb * parts; x += warps) {
    const uint64_t g = x / parts;
    uint64_t s = bucket_start[g], d = bucket_d[g], o = bucket_out[g];
    const uint64_t start = s;
    uint64_t t = bucket_head[g];  // first task + 1, 0: none
    const uint64_t nt2 = t ? *task_count : 0;
    while (true) {
      if (t) {
        if (t > nt2 || tasks[t - 1].x != (uint32_t)g) break;
        s = start + tasks[t - 1].y;
        d = tasks[t - 1].w;
        t++;
      }
      for (uint64_t i0 = (x - g * parts) * 32 * U + lane; i0 < d; i0 += (uint64_t)parts * 32 * U) {
        K kv[U];
        uint32_t cv[U];
#pragma unroll
        for (int u = 0; u < U; u++)
          if (i0 + 32 * u < d) {
            kv[u] = stage_keys[s + i0 + 32 * u];
            cv[u] = stage_counts[s + i0 + 32 * u];
          }
#pragma unroll
        for (int u = 0; u < U; u++)
          if (i0 + 32 * u < d) {
            out_keys[o + i0 + 32 * u] = kv[u];
            out_counts[o + i0 + 32 * u] = cv[u];
          }
      }
      if (!t) break;
      o += d;
    }
  }
}

template __global__ void k_compact_runs<uint64_t>(const uint64_t *, const uint32_t *, const uint64_t *,
                                                  const unsigned long long *, const uint64_t *, const uint64_t *,
                                                  uint32_t, uint64_t *, uint32_t *, uint64_t *, const uint32_t *,
                                                  const uint4 *, const unsigned long long *, const uint32_t *);
template __global__ void k_compact_runs<u128>(const u128 *, const uint32_t *, const uint64_t *,
                                              const unsigned long long *, const uint64_t *, const uint64_t *,
                                              uint32_t, u128 *, uint32_t *, uint64_t *, const uint32_t *,
                                              const uint4 *, const unsigned long long *, const uint32_t *);
template __global__ void k_bucket_hist<uint64_t>(ExpandArgs);
template __global__ void k_bucket_hist<u128>(ExpandArgs);
template __global__ void k_bucket_scatter<uint64_t, 1>(ExpandArgs);
template __global__ void k_bucket_scatter<uint64_t, 2>(ExpandArgs);
template __global__ void k_bucket_scatter<u128, 1>(ExpandArgs);
template __global__ void k_bucket_sort<uint64_t, false>(SortCountArgs);
template __global__ void k_bucket_sort<uint64_t, true>(SortCountArgs);
template __global__ void k_bucket_sort<u128, false>(SortCountArgs);
template __global__ void k_bucket_open<uint64_t>(SortCountArgs);
template __global__ void k_bucket_open<u128>(SortCountArgs);
template __global__ void k_bucket_slices<uint64_t>(SortCountArgs);
template __global__ void k_bucket_slices<u128>(SortCountArgs);

}  // namespace gkc
