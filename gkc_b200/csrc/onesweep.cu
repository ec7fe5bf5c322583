// Device-wide LSD radix sort, onesweep form (Adinets & Merrill, "Onesweep: a
// faster least significant digit radix sort for GPUs", 2022): one upfront
// pass histograms every digit position, then each digit pass is a single
// kernel in which a tile ranks its keys stably, publishes its per-digit
// counts, and finds the counts of all earlier tiles by a decoupled
// look-back, so keys are scattered in one read and one write per pass.
//
// Keys: uint64 or unsigned __int128, sorted on their low `key_bits` bits,
// 8-bit digits.  Every wait on another tile is bounded.  Long keys with values
// (sort_pairs) take passes over their leading bits only; a kernel of its own
// orders the runs that these leave.
#include <algorithm>
#include <utility>
#include <vector>

#include "common.cuh"
#include "onesweep.h"

namespace gkc {

constexpr int OS_NT = 256;
constexpr int OS_WARPS = OS_NT / 32;
constexpr int OS_RADIX = 256;
// Keys per thread: a tile's keys are put in digit order in shared memory
// before they are written.  8 leave three CTAs on an SM (16 8-byte keys: two,
// and the merged list of 60 M bases took 4.5 ms, not 4.3).
constexpr int OS_ITEMS = 8;
constexpr int OS_TILE = OS_NT * OS_ITEMS;
constexpr int OS_WINDOW = 4;  // earlier tiles looked at together

constexpr unsigned long long OS_AGG = 1ull << 62, OS_PRE = 2ull << 62;
constexpr unsigned long long OS_VAL = (1ull << 62) - 1;

// Tile entries carry all that is read through them, so no order with other
// memory is needed: relaxed accesses, several in flight.
GKC_DEV unsigned long long os_ld(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
GKC_DEV void os_st(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

template <typename K>
GKC_DEV uint32_t os_digit(K x, int shift) {
  return (uint32_t)(x >> shift) & 0xFFu;
}

// The lanes whose digit equals this one's, among those with `in`: eight
// ballots (a MATCH takes 31 cycles a warp here, these about 12).
GKC_DEV uint32_t os_peers(uint32_t d, bool in) {
  uint32_t peers = __ballot_sync(0xffffffffu, in);
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool bit = (d >> b) & 1u;
    const uint32_t v = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? v : ~v;
  }
  return peers;
}

// hist[pass][digit] over all keys, for every pass (digits from bit `bit0` on).
template <typename K>
__global__ void __launch_bounds__(OS_NT) k_os_histogram(const K *keys, const uint64_t *n_dev,
                                                        int passes, int bit0, unsigned long long *hist) {
  __shared__ uint32_t h[16][OS_RADIX];
  const uint64_t n = *n_dev;
  for (int i = threadIdx.x; i < passes * OS_RADIX; i += OS_NT) h[i / OS_RADIX][i % OS_RADIX] = 0;
  __syncthreads();
  for (uint64_t i = blockIdx.x * (uint64_t)OS_NT + threadIdx.x; i < n; i += (uint64_t)gridDim.x * OS_NT) {
    K x = keys[i];
    for (int p = 0; p < passes; p++) atomicAdd(&h[p][os_digit<K>(x, bit0 + 8 * p)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * OS_RADIX; i += OS_NT) {
    uint32_t v = h[i / OS_RADIX][i % OS_RADIX];
    if (v) atomicAdd(&hist[i], (unsigned long long)v);
  }
}

// exclusive scan of each pass's 256 digit counts (one CTA, one warp per pass)
__global__ void k_os_digit_offsets(unsigned long long *hist, int passes) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int p = warp; p < passes; p += blockDim.x / 32) {
    unsigned long long carry = 0;
    for (int d0 = 0; d0 < OS_RADIX; d0 += 32) {
      unsigned long long v = hist[p * OS_RADIX + d0 + lane], x = v;
      for (int s = 1; s < 32; s <<= 1) {
        unsigned long long y = __shfl_up_sync(0xffffffffu, x, s);
        if (lane >= s) x += y;
      }
      hist[p * OS_RADIX + d0 + lane] = carry + x - v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
  }
}

// One digit pass.  With KV, a uint32 value moves with each key (vin -> vout).
// A tile is put in digit order in shared memory, so that each digit's keys
// leave as one run; a tile's counts are published before that, and the
// earlier tiles' are added up after it, four a step.  (Keys written straight
// from registers and one earlier tile a step: 424 us a pass of 13.9 M 16-byte
// keys with values.)
template <typename K, bool KV>
__global__ void __launch_bounds__(OS_NT, 3) k_os_pass(const K *in, K *out, const uint32_t *vin,
                                                                           uint32_t *vout, const uint64_t *n_dev,
                                                                           int shift, const unsigned long long *digit_base,
                                                                           unsigned long long *lookback,
                                                                           unsigned long long *ticket, uint32_t *err) {
  constexpr int ITEMS = OS_ITEMS, TILE = OS_TILE;
  __shared__ __align__(16) uint8_t sbuf[TILE * sizeof(K)];
  __shared__ uint8_t D[TILE];
  __shared__ uint32_t warp_cnt[OS_WARPS][OS_RADIX];
  __shared__ uint32_t toff[OS_RADIX];               // first tile position of each digit
  __shared__ uint64_t gbase[OS_RADIX];              // where tile position 0 of each digit would go
  __shared__ uint32_t tmp[64];
  __shared__ uint64_t s_tile;
  K *S = reinterpret_cast<K *>(sbuf);               // the tile in digit order, D its digits
  uint32_t *V = &warp_cnt[0][0];                    // and its values, once every rank is known
  static_assert(TILE == OS_WARPS * OS_RADIX, "a value for every counter");
  const uint64_t n = *n_dev;
  const uint64_t n_tiles = (n + TILE - 1) / TILE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  while (true) {
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1ull);
    for (int i = threadIdx.x; i < OS_WARPS * OS_RADIX; i += OS_NT) (&warp_cnt[0][0])[i] = 0;
    __syncthreads();
    const uint64_t tile = s_tile;
    if (tile >= n_tiles) break;
    const uint32_t tn = (uint32_t)min((uint64_t)TILE, n - tile * TILE);
    // each warp owns a contiguous segment of 32 * ITEMS keys; round r, lane l
    // takes key r*32 + l of that segment, so (round, lane) order is the input
    // order and the ranks below are stable
    const uint64_t seg = tile * TILE + (uint64_t)warp * 32 * ITEMS;
    K key[ITEMS];
    uint32_t val[KV ? ITEMS : 1];
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
      const uint64_t i = seg + (uint64_t)r * 32 + lane;
      key[r] = i < n ? in[i] : (K)0;
      if (KV) val[KV ? r : 0] = i < n ? vin[i] : 0u;
    }
    uint32_t rank[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
      const bool v = seg + (uint64_t)r * 32 + lane < n;
      const uint32_t d = os_digit<K>(key[r], shift);
      const uint32_t peers = os_peers(d, v);
      const uint32_t below = __popc(peers & ((1u << lane) - 1u));
      uint32_t base = 0;
      if (v) base = warp_cnt[warp][d];
      __syncwarp();
      rank[r] = d << 16 | (base + below);
      // the highest peer advances the warp's counter for this digit
      if (v && (peers >> lane) == 1u) warp_cnt[warp][d] = base + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    // per digit: tile count, warp prefixes; publish
    const int d = threadIdx.x;  // OS_NT == OS_RADIX
    unsigned long long *lb = lookback + tile * OS_RADIX + d;
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < OS_WARPS; w++) {
      const uint32_t c = warp_cnt[w][d];
      warp_cnt[w][d] = run;
      run += c;
    }
    os_st(lb, (tile == 0 ? OS_PRE : OS_AGG) | run);
    uint32_t total;
    const uint32_t first = block_exclusive_scan<OS_NT>(run, tmp, &total);
    toff[d] = first;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; r++)
      if (seg + (uint64_t)r * 32 + lane < n) {
        const uint32_t x = rank[r] >> 16;
        rank[r] = (rank[r] & 0xFFFFu) + toff[x] + warp_cnt[warp][x];
        S[rank[r]] = key[r];
        D[rank[r]] = (uint8_t)x;
      }
    if (KV) {
      __syncthreads();
#pragma unroll
      for (int r = 0; r < ITEMS; r++)
        if (seg + (uint64_t)r * 32 + lane < n) V[rank[r]] = val[KV ? r : 0];
    }
    // the earlier tiles' keys of this digit
    uint64_t excl = 0, j = tile;  // tiles [j, tile) are added up
    uint32_t it = 0;
    bool found = tile == 0;
    while (!found) {
      unsigned long long v[OS_WINDOW];
#pragma unroll
      for (int i = 0; i < OS_WINDOW; i++)
        v[i] = j > (uint64_t)i ? os_ld(lookback + (j - 1 - i) * OS_RADIX + d) : OS_PRE;
      uint32_t used = 0;
      bool more = true;
#pragma unroll
      for (int i = 0; i < OS_WINDOW; i++) {
        more = more && (v[i] & ~OS_VAL) != 0;
        if (more) {
          excl += v[i] & OS_VAL;
          used++;
          if ((v[i] & ~OS_VAL) == OS_PRE) {
            found = true;
            more = false;
          }
        }
      }
      if (!found) {
        j -= used;
        if (used == 0) {
          if (++it > (1u << 24)) {
            atomicOr(err, ERR_SPIN_TIMEOUT);
            break;
          }
          nanosleep_backoff(it);
        }
      }
    }
    if (tile != 0) os_st(lb, OS_PRE | (excl + run));
    gbase[d] = digit_base[d] + excl - first;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < tn; i += OS_NT) {
      const uint64_t at = gbase[D[i]] + i;
      out[at] = S[i];
      if (KV) vout[at] = V[i];
    }
    __syncthreads();
  }
}

template <typename K, bool KV>
static OnesweepStatus onesweep_run(K *keys, K *alt, uint32_t *vals, uint32_t *valt, const uint64_t *n_dev,
                                   uint64_t n_max, int bit0, int key_bits, OnesweepScratch s, cudaStream_t st,
                                   uint32_t *launches) {
  const int passes = (key_bits - bit0 + 7) / 8;
  const uint64_t tiles = (n_max + OS_TILE - 1) / OS_TILE;
  cudaMemsetAsync(s.hist, 0, sizeof(unsigned long long) * 16 * OS_RADIX, st);
  unsigned grid_h = (unsigned)std::min<uint64_t>(std::max<uint64_t>(1, (n_max + OS_NT * 8 - 1) / (OS_NT * 8)), 148 * 16);
  k_os_histogram<K><<<grid_h, OS_NT, 0, st>>>(keys, n_dev, passes, bit0, s.hist);
  k_os_digit_offsets<<<1, 32 * 8, 0, st>>>(s.hist, passes);
  *launches += 2;
  K *src = keys, *dst = alt;
  uint32_t *vsrc = vals, *vdst = valt;
  for (int p = 0; p < passes; p++) {
    cudaMemsetAsync(s.lookback, 0, sizeof(unsigned long long) * (tiles + 1) * OS_RADIX, st);
    cudaMemsetAsync(s.ticket, 0, sizeof(unsigned long long), st);
    unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)s.max_ctas));
    k_os_pass<K, KV><<<grid, OS_NT, 0, st>>>(src, dst, vsrc, vdst, n_dev, bit0 + 8 * p, s.hist + p * OS_RADIX, s.lookback,
                                              s.ticket, s.err);
    *launches += 1;
    K *t = src;
    src = dst;
    dst = t;
    uint32_t *vt = vsrc;
    vsrc = vdst;
    vdst = vt;
  }
  return OnesweepStatus{src == keys ? 0 : 1};
}

template <typename K>
OnesweepStatus onesweep_sort(K *keys, K *alt, const uint64_t *n_dev, uint64_t n_max, int key_bits,
                             OnesweepScratch s, cudaStream_t st, uint32_t *launches) {
  return onesweep_run<K, false>(keys, alt, nullptr, nullptr, n_dev, n_max, 0, key_bits, s, st, launches);
}

// ---- pairs by their leading bits, then the rest run by run ----

// Of n keys whose leading bits spread them well, few share some log2(n) + 5
// leading bits with another one: passes over those bits leave runs of equal
// leading bits, short ones, which one more kernel puts in order.  So a sort of
// 126-bit keys takes four or five passes over memory, not 16.
constexpr int OF_NT = 256;
constexpr uint32_t OF_TILE = 1024;  // a tile's runs begin in it
constexpr uint32_t OF_RUN = 512;    // and are ranked in shared memory up to this length
constexpr uint32_t OF_LOAD = OF_TILE + OF_RUN;

// 1 where y at place j comes before x at place i (equal keys in their order):
// the borrow of y - x less that of j - i, one subtraction a word.
GKC_DEV uint32_t os_before(uint64_t y, uint32_t j, uint64_t x, uint32_t i) {
  uint32_t t;
  asm("{\n\t"
      ".reg .u32 d;\n\t"
      "sub.cc.u32 d, %1, %2;\n\t"
      "subc.cc.u32 d, %3, %4;\n\t"
      "subc.cc.u32 d, %5, %6;\n\t"
      "subc.u32 %0, 0, 0;\n\t"
      "}"
      : "=r"(t)
      : "r"(j), "r"(i), "r"((uint32_t)y), "r"((uint32_t)x), "r"((uint32_t)(y >> 32)), "r"((uint32_t)(x >> 32)));
  return 0u - t;
}
GKC_DEV uint32_t os_before(u128 y, uint32_t j, u128 x, uint32_t i) {
  uint32_t t;
  asm("{\n\t"
      ".reg .u32 d;\n\t"
      "sub.cc.u32 d, %1, %2;\n\t"
      "subc.cc.u32 d, %3, %4;\n\t"
      "subc.cc.u32 d, %5, %6;\n\t"
      "subc.cc.u32 d, %7, %8;\n\t"
      "subc.cc.u32 d, %9, %10;\n\t"
      "subc.u32 %0, 0, 0;\n\t"
      "}"
      : "=r"(t)
      : "r"(j), "r"(i), "r"((uint32_t)y), "r"((uint32_t)x), "r"((uint32_t)(y >> 32)), "r"((uint32_t)(x >> 32)),
        "r"((uint32_t)(y >> 64)), "r"((uint32_t)(x >> 64)), "r"((uint32_t)(y >> 96)), "r"((uint32_t)(x >> 96)));
  return 0u - t;
}

// What k_os_fix leaves behind it, in the look-back words: the number of runs
// listed for the host, a word for every tile (whether the run that begins in it
// and goes on past it is listed), and the runs' [begin, end), each longer than
// OF_RUN, so at most n / OF_RUN.
struct FixLists {
  unsigned long long *count, *claimed, *runs;
};
static uint64_t fix_tiles(uint64_t n) { return (n + OF_TILE - 1) / OF_TILE; }
static FixLists fix_lists(unsigned long long *words, uint64_t n) {
  return FixLists{words, words + 2, words + 2 + fix_tiles(n)};
}

// The first place in [0, base) whose key has the leading bits `lead` (keys in
// their order, the last one of them has), by the calling warp.
template <typename K>
GKC_DEV uint64_t os_run_start(const K *in, uint64_t base, K lead, int bit0) {
  const uint32_t lane = threadIdx.x & 31u;
  uint64_t lo = 0, hi = base;
  while (lo < hi) {
    const uint64_t step = (hi - lo + 31) / 32, at = lo + lane * step;
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, at < hi && (in[at] >> bit0) < lead));
    hi = min(hi, lo + c * step);
    if (c) lo += (c - 1) * step + 1;
  }
  return lo;
}

// Pairs in the order of their bits from `bit0` up, to `out` in the order of
// all bits: each run of equal leading bits by ranking every key in it (equal
// keys keep their order).  A tile takes the runs that begin in it.  Longer ones
// than OF_RUN are copied as they are, each tile its own part; the first tile
// that sees keys of a run differ lists it for the host.  Bound by the comparisons, a run's length
// for each key (one subtraction a word: 0.48 -> 0.26 ms for 13.9 M 16-byte keys
// in runs of about 17; the twelve passes it stands for take 2.7.  8.7 M
// distinct 8-byte keys: 0.08, for passes of 0.47).  Reads of few letters, 12 M
// keys, most in one run: position lists 34.6 ms where one block copied a run, 2.6 so.
template <typename K>
__global__ void __launch_bounds__(OF_NT) k_os_fix(const K *in, K *out, const uint32_t *vin, uint32_t *vout,
                                                  const uint64_t *n_dev, int bit0, FixLists lists) {
  __shared__ __align__(16) K S[OF_LOAD];
  __shared__ uint32_t heads[OF_LOAD / 32];  // bit i: a run begins at S[i] (or the keys end there)
  __shared__ uint32_t n_long, long_s[4], long_e[4], before;  // before: end of a long run that goes on here
  constexpr uint32_t OPEN = ~0u;
  const uint64_t n = *n_dev;
  const uint32_t tid = threadIdx.x;
  for (uint64_t base = (uint64_t)blockIdx.x * OF_TILE; base < n; base += (uint64_t)gridDim.x * OF_TILE) {
    const uint32_t m = (uint32_t)min(n - base, (uint64_t)OF_LOAD);
    const bool closed = base + m == n;
    for (uint32_t i = tid; i < m; i += OF_NT) S[i] = in[base + i];
    if (tid == 0) {
      n_long = 0;
      before = 0;
    }
    __syncthreads();
    for (uint32_t i = tid; i < OF_LOAD; i += OF_NT) {  // OF_LOAD is whole rounds
      bool head = i == m;
      if (i < m) {
        const bool first = i == 0 && base == 0;
        head = first || ((i ? S[i - 1] : in[base - 1]) >> bit0) != (S[i] >> bit0);
      }
      const uint32_t w = __ballot_sync(0xffffffffu, head);
      if ((tid & 31u) == 0) heads[i >> 5] = w;
    }
    __syncthreads();
    if (tid == 0 && !(heads[0] & 1u)) {  // a run of an earlier tile goes on
      uint32_t w = 0;
      while (w + 1 < OF_LOAD / 32 && !heads[w]) w++;
      const uint32_t e = heads[w] ? 32 * w + __ffs(heads[w]) - 1 : closed ? m : OPEN;
      if (e == OPEN || (base + e > OF_RUN && (in[base + e - OF_RUN - 1] >> bit0) == (S[0] >> bit0)))
        before = e;
    }
    for (uint32_t i = tid; i < m; i += OF_NT) {
      const uint32_t b = i & 31u;
      uint32_t w = i >> 5, bits = heads[w] & (0xFFFFFFFFu >> (31 - b));
      while (!bits && w > 0) bits = heads[--w];
      if (!bits) continue;  // begins in an earlier tile
      const uint32_t s = 32 * w + 31 - __clz(bits);
      if (s >= OF_TILE) continue;  // in a later one
      w = i >> 5;
      bits = b == 31 ? 0u : heads[w] & (0xFFFFFFFFu << (b + 1));
      while (!bits && w + 1 < OF_LOAD / 32) bits = heads[++w];
      const uint32_t e = bits ? 32 * w + __ffs(bits) - 1 : closed ? m : OPEN;
      if (e == OPEN || e - s > OF_RUN) {
        if (i == s) {  // at most OF_TILE / OF_RUN + 1 of them
          const uint32_t at = atomicAdd(&n_long, 1u);
          long_s[at] = s;
          long_e[at] = e;
        }
        continue;
      }
      const K x = S[i];
      uint32_t at = s;
#pragma unroll 4
      for (uint32_t j = s; j < e; j++) at += os_before(S[j], j, x, i);
      out[base + at] = x;
      vout[base + at] = vin[base + i];
    }
    __syncthreads();
    // the tile's part of long runs: of the one from before, then of those that begin here
    for (uint32_t l = 0; l < n_long + 1; l++) {
      const uint32_t s = l ? long_s[l - 1] : 0u, e = l ? long_e[l - 1] : before, stop = min(e, min(m, OF_TILE));
      if (s >= stop) continue;  // the same in every thread
      bool differ = false;
      for (uint32_t i = s + tid; i < stop; i += OF_NT) {
        const K x = S[i];
        if (i > s || l == 0) differ = differ || x != (i ? S[i - 1] : in[base - 1]);
        out[base + i] = x;
        vout[base + i] = vin[base + i];
      }
      if (__syncthreads_or(differ) && tid < 32) {
        const uint64_t first = l ? base + s : os_run_start<K>(in, base, S[0] >> bit0, bit0);
        const bool whole = l && e <= OF_TILE;  // no other tile sees it
        if (tid == 0 && (whole || atomicExch(lists.claimed + first / OF_TILE, 1ull) == 0)) {
          uint64_t end = base + e;
          if (e == OPEN) {  // the first key after the loaded ones with other leading bits
            const K lead = S[s] >> bit0;
            end = base + m;
            for (uint64_t hi = n; end < hi;) {
              const uint64_t mid = (end + hi) >> 1;
              if ((in[mid] >> bit0) == lead) end = mid + 1;
              else hi = mid;
            }
          }
          const unsigned long long at = atomicAdd(lists.count, 1ull);
          lists.runs[2 * at] = first;
          lists.runs[2 * at + 1] = end;
        }
      }
    }
    __syncthreads();  // before the next tile's keys
  }
}

// The listed runs (begin, end, first place in the compact arrays) to the
// compact arrays, or back.
template <typename K>
__global__ void __launch_bounds__(OF_NT) k_os_runs(K *keys, uint32_t *vals, K *ck, uint32_t *cv,
                                                   const unsigned long long *runs, uint64_t n_runs, bool back) {
  for (uint64_t r = blockIdx.x; r < n_runs; r += gridDim.x) {
    const uint64_t s = runs[3 * r], n = runs[3 * r + 1] - s, at = runs[3 * r + 2];
    for (uint64_t i = threadIdx.x; i < n; i += OF_NT) {
      if (back) {
        keys[s + i] = ck[at + i];
        vals[s + i] = cv[at + i];
      } else {
        ck[at + i] = keys[s + i];
        cv[at + i] = vals[s + i];
      }
    }
  }
}

template <typename K>
PairsStatus sort_pairs(K *keys, K *alt, uint32_t *vals, uint32_t *valt, const uint64_t *n_dev, uint64_t n, int key_bits,
                       OnesweepScratch s, cudaStream_t st, uint32_t *launches) {
  int lead = 5;
  while (lead < 64 && (n >> (lead - 5))) lead++;
  lead = (lead + 7) / 8 * 8;
  if (lead + 8 >= key_bits)  // the last kernel would save a pass at most
    return PairsStatus{onesweep_run<K, true>(keys, alt, vals, valt, n_dev, n, 0, key_bits, s, st, launches).result_in_alt,
                       false};
  const int bit0 = key_bits - lead;
  const int in_alt = onesweep_run<K, true>(keys, alt, vals, valt, n_dev, n, bit0, key_bits, s, st, launches).result_in_alt;
  // the look-back entries are free now: the lists of long runs
  const FixLists lists = fix_lists(s.lookback, n);
  cudaMemsetAsync(lists.count, 0, 8 * (2 + fix_tiles(n)), st);
  const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + OF_TILE - 1) / OF_TILE, 1u << 20));
  k_os_fix<K><<<grid, OF_NT, 0, st>>>(in_alt ? alt : keys, in_alt ? keys : alt, in_alt ? valt : vals,
                                      in_alt ? vals : valt, n_dev, bit0, lists);
  *launches += 1;
  return PairsStatus{!in_alt, true};
}

template <typename K>
int sort_pairs_rest(PairsStatus done, uint64_t n_runs, K *keys, K *alt, uint32_t *vals, uint32_t *valt,
                    const uint64_t *n_dev, uint64_t n, int key_bits, OnesweepScratch s, cudaStream_t st,
                    uint32_t *launches) {
  K *from = done.result_in_alt ? alt : keys, *free_k = done.result_in_alt ? keys : alt;
  uint32_t *vfrom = done.result_in_alt ? valt : vals, *free_v = done.result_in_alt ? vals : valt;
  std::vector<unsigned long long> list(2 * n_runs), runs(3 * n_runs);
  cudaMemcpyAsync(list.data(), fix_lists(s.lookback, n).runs, 16 * n_runs, cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  std::vector<std::pair<unsigned long long, unsigned long long>> r(n_runs);
  for (uint64_t i = 0; i < n_runs; i++) r[i] = {list[2 * i], list[2 * i + 1]};
  std::sort(r.begin(), r.end());
  uint64_t u = 0;
  for (uint64_t i = 0; i < n_runs; i++) {
    runs[3 * i] = r[i].first;
    runs[3 * i + 1] = r[i].second;
    runs[3 * i + 2] = u;
    u += r[i].second - r[i].first;
  }
  const uint64_t lb = onesweep_lookback_words(u);
  if (2 * u > n || lb + 3 * n_runs + 1 > onesweep_lookback_words(n)) {
    // no room for them beside their sort: all pairs (equal keys are in order, and stay so)
    const int moved = onesweep_run<K, true>(from, free_k, vfrom, free_v, n_dev, n, 0, key_bits, s, st, launches).result_in_alt;
    return moved ? !done.result_in_alt : done.result_in_alt;
  }
  // the runs compacted into the free buffer, sorted there (they keep their
  // order among each other), and put back.  Their table lies behind the place
  // of this sort's look-back entries.
  unsigned long long *tab = s.lookback + lb;
  runs.push_back(u);
  cudaMemcpyAsync(tab, runs.data(), 8 * runs.size(), cudaMemcpyHostToDevice, st);
  cudaStreamSynchronize(st);  // `runs` ends with this call
  const unsigned grid = (unsigned)std::min<uint64_t>(n_runs, 148 * 8);
  k_os_runs<K><<<grid, OF_NT, 0, st>>>(from, vfrom, free_k, free_v, tab, n_runs, false);
  const int moved = onesweep_run<K, true>(free_k, free_k + u, free_v, free_v + u,
                                          reinterpret_cast<const uint64_t *>(tab + 3 * n_runs), u, 0, key_bits, s, st,
                                          launches).result_in_alt;
  k_os_runs<K><<<grid, OF_NT, 0, st>>>(from, vfrom, free_k + (moved ? u : 0), free_v + (moved ? u : 0), tab, n_runs, true);
  *launches += 2;
  return done.result_in_alt;
}

size_t onesweep_lookback_words(uint64_t n_max) {
  return ((n_max + OS_TILE - 1) / OS_TILE + 1) * OS_RADIX;
}

template OnesweepStatus onesweep_sort<uint64_t>(uint64_t *, uint64_t *, const uint64_t *, uint64_t,
                                                int, OnesweepScratch, cudaStream_t, uint32_t *);
template OnesweepStatus onesweep_sort<u128>(u128 *, u128 *, const uint64_t *, uint64_t, int,
                                            OnesweepScratch, cudaStream_t, uint32_t *);
template PairsStatus sort_pairs<uint64_t>(uint64_t *, uint64_t *, uint32_t *, uint32_t *, const uint64_t *, uint64_t, int,
                                          OnesweepScratch, cudaStream_t, uint32_t *);
template PairsStatus sort_pairs<u128>(u128 *, u128 *, uint32_t *, uint32_t *, const uint64_t *, uint64_t, int,
                                      OnesweepScratch, cudaStream_t, uint32_t *);
template int sort_pairs_rest<uint64_t>(PairsStatus, uint64_t, uint64_t *, uint64_t *, uint32_t *, uint32_t *,
                                       const uint64_t *, uint64_t, int, OnesweepScratch, cudaStream_t, uint32_t *);
template int sort_pairs_rest<u128>(PairsStatus, uint64_t, u128 *, u128 *, uint32_t *, uint32_t *, const uint64_t *,
                                   uint64_t, int, OnesweepScratch, cudaStream_t, uint32_t *);

}  // namespace gkc
