// Device-wide exclusive scan of 64-bit counters: out[i] = sum(in[0, i)),
// out[n] = total.  Small lists: one CTA, one launch (each launch of the three
// costs 2-4 us whatever its size).  Others: reduce -> scan of the tile sums
// -> apply.
#include "common.cuh"
#include "kernels.h"

namespace gkc {

constexpr int SCAN_NT = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_NT * SCAN_ITEMS;
constexpr int SCAN_ONE_NT = 1024;
// up to here one CTA: three rounds of 8192 take about as long as the three launches (the 54 K cells of a 3 M base
// job took 12 us longer in one CTA)
constexpr uint64_t SCAN_ONE_MAX = 24576;

// What is scanned: an array, or the k-mers of superkmer descriptors.
struct ScanArray {
  const unsigned long long *p;
  GKC_DEV uint64_t operator()(uint64_t i) const { return p[i]; }
};
struct ScanKmers {
  const unsigned long long *desc;
  int k;
  GKC_DEV uint64_t operator()(uint64_t i) const {
    const uint32_t len = (uint32_t)(desc[i] & 0xFFFFFFu);
    return len >= (uint32_t)k ? len - k + 1 : 0;
  }
};

// packed bytes of superkmers given by length, or by descriptor (its low 24 bits)
struct ScanLenBytes {
  const uint32_t *len;
  GKC_DEV uint64_t operator()(uint64_t i) const { return ((uint64_t)len[i] + 3) / 4; }
};
struct ScanDescBytes {
  const uint64_t *desc;
  GKC_DEV uint64_t operator()(uint64_t i) const { return ((desc[i] & 0xFFFFFFu) + 3) / 4; }
};

GKC_DEV uint64_t scan_len(uint64_t n_cap, const uint64_t *n_dev) { return n_dev ? min(n_cap, *n_dev) : n_cap; }

template <typename Src>
__global__ void __launch_bounds__(SCAN_ONE_NT) k_scan_one(Src in, uint64_t n_cap, const uint64_t *n_dev, uint64_t *out,
                                                           unsigned long long *stamp) {
  stamp_now(stamp);
  __shared__ uint64_t tmp[32];
  const uint64_t n = scan_len(n_cap, n_dev);
  uint64_t carry = 0;
  for (uint64_t b0 = 0; b0 < n; b0 += SCAN_ONE_NT * SCAN_ITEMS) {
    const uint64_t i0 = b0 + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint64_t v[SCAN_ITEMS], s = 0;
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; t++) {
      v[t] = i0 + t < n ? in(i0 + t) : 0;
      s += v[t];
    }
    uint64_t total;
    uint64_t run = carry + block_exclusive_scan_u64<SCAN_ONE_NT>(s, tmp, &total);
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; t++) {
      if (i0 + t < n) out[i0 + t] = run;
      run += v[t];
    }
    carry += total;
  }
  if (threadIdx.x == 0) out[n] = carry;
}

template <typename Src>
__global__ void __launch_bounds__(SCAN_NT) k_scan_reduce(Src in, uint64_t n_cap, const uint64_t *n_dev,
                                                         uint64_t *tile_sum, unsigned long long *stamp) {
  stamp_now(stamp);
  __shared__ uint64_t tmp[32];
  const uint64_t n = scan_len(n_cap, n_dev), base = (uint64_t)blockIdx.x * SCAN_TILE;
  if (base >= n) return;  // not read by the next kernels
  uint64_t s = 0;
#pragma unroll
  for (int t = 0; t < SCAN_ITEMS; t++) {
    const uint64_t i = base + (uint64_t)t * SCAN_NT + threadIdx.x;
    if (i < n) s += in(i);
  }
  s = block_sum_u64<SCAN_NT>(s, tmp);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = s;
}

// single CTA: exclusive scan of the tile sums in place, the total to out[n]
__global__ void __launch_bounds__(SCAN_ONE_NT) k_scan_tiles(uint64_t *tile_sum, uint64_t n_cap, const uint64_t *n_dev,
                                                            uint64_t *out) {
  __shared__ uint64_t tmp[32];
  const uint64_t n = scan_len(n_cap, n_dev), n_tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  uint64_t carry = 0;
  for (uint64_t b0 = 0; b0 < n_tiles; b0 += SCAN_ONE_NT * SCAN_ITEMS) {
    const uint64_t i0 = b0 + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint64_t v[SCAN_ITEMS], s = 0;
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; t++) {
      v[t] = i0 + t < n_tiles ? tile_sum[i0 + t] : 0;
      s += v[t];
    }
    uint64_t total;
    uint64_t run = carry + block_exclusive_scan_u64<SCAN_ONE_NT>(s, tmp, &total);
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; t++) {
      if (i0 + t < n_tiles) tile_sum[i0 + t] = run;
      run += v[t];
    }
    carry += total;
  }
  if (threadIdx.x == 0) out[n] = carry;
}

template <typename Src>
__global__ void __launch_bounds__(SCAN_NT) k_scan_apply(Src in, uint64_t n_cap, const uint64_t *n_dev,
                                                        const uint64_t *tile_sum, uint64_t *out) {
  __shared__ uint64_t tmp[32];
  const uint64_t n = scan_len(n_cap, n_dev), base = (uint64_t)blockIdx.x * SCAN_TILE;
  if (base >= n) return;
  // warp w holds 32 * SCAN_ITEMS consecutive items, round t its items t * 32 .. + 31
  const int lane = threadIdx.x & 31;
  const uint64_t i0 = base + (uint64_t)(threadIdx.x >> 5) * 32 * SCAN_ITEMS + lane;
  uint64_t v[SCAN_ITEMS], s = 0;
#pragma unroll
  for (int t = 0; t < SCAN_ITEMS; t++) v[t] = i0 + 32 * t < n ? in(i0 + 32 * t) : 0;
#pragma unroll
  for (int t = 0; t < SCAN_ITEMS; t++) {  // v[t]: exclusive within the warp's items
    uint64_t x = v[t];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    const uint64_t row = __shfl_sync(0xffffffffu, x, 31);
    v[t] = s + x - v[t];
    s += row;
  }
  // s: the warp's total, in every lane
  if (lane == 0) tmp[threadIdx.x >> 5] = s;
  __syncthreads();
  uint64_t run = tile_sum[blockIdx.x];
  for (int w = 0; w < (int)(threadIdx.x >> 5); w++) run += tmp[w];
#pragma unroll
  for (int t = 0; t < SCAN_ITEMS; t++)
    if (i0 + 32 * t < n) out[i0 + 32 * t] = run + v[t];
}

size_t scan_u64_tmp_words(uint64_t n) { return (n + SCAN_TILE - 1) / SCAN_TILE + 2; }

template <typename Src>
static uint32_t scan_any(Src in, uint64_t *out, uint64_t n_cap, const uint64_t *n_dev, uint64_t *block_tmp,
                         cudaStream_t st, unsigned long long *stamp = nullptr) {
  if (n_cap <= SCAN_ONE_MAX) {
    k_scan_one<Src><<<1, SCAN_ONE_NT, 0, st>>>(in, n_cap, n_dev, out, stamp);
    return 1;
  }
  const unsigned tiles = (unsigned)((n_cap + SCAN_TILE - 1) / SCAN_TILE);
  k_scan_reduce<Src><<<tiles, SCAN_NT, 0, st>>>(in, n_cap, n_dev, block_tmp, stamp);
  k_scan_tiles<<<1, SCAN_ONE_NT, 0, st>>>(block_tmp, n_cap, n_dev, out);
  k_scan_apply<Src><<<tiles, SCAN_NT, 0, st>>>(in, n_cap, n_dev, block_tmp, out);
  return 3;
}

uint32_t scan_u64_dev(const unsigned long long *in, uint64_t *out, uint64_t n_cap, const uint64_t *n_dev,
                      uint64_t *block_tmp, cudaStream_t st, unsigned long long *stamp) {
  return scan_any(ScanArray{in}, out, n_cap, n_dev, block_tmp, st, stamp);
}

uint32_t scan_u64(const unsigned long long *in, uint64_t *out, uint64_t n, uint64_t *block_tmp, cudaStream_t st) {
  return scan_any(ScanArray{in}, out, n, nullptr, block_tmp, st);
}

uint32_t scan_kmers_dev(const uint64_t *desc, int k, uint64_t *out, uint64_t n_cap, const uint64_t *n_dev,
                        uint64_t *block_tmp, cudaStream_t st, unsigned long long *stamp) {
  return scan_any(ScanKmers{reinterpret_cast<const unsigned long long *>(desc), k}, out, n_cap, n_dev, block_tmp, st, stamp);
}

uint32_t scan_len_bytes(const uint32_t *len, uint64_t *out, uint64_t n, uint64_t *block_tmp, cudaStream_t st) {
  return scan_any(ScanLenBytes{len}, out, n, nullptr, block_tmp, st);
}

uint32_t scan_desc_bytes(const uint64_t *desc, uint64_t *out, uint64_t n, uint64_t *block_tmp, cudaStream_t st) {
  return scan_any(ScanDescBytes{desc}, out, n, nullptr, block_tmp, st);
}

}  // namespace gkc
