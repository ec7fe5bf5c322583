// Kernel argument blocks and launch helpers shared by the .cu files.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

namespace gkc {

struct PartArgs {
  int filter;            // minimizer filter (FILTER_*)
  const uint8_t *reads;  // concatenated read bytes (CSR), offsets rebased to 0
  uint64_t nbytes;       // byte count (an upper bound when nbytes_dev is set)
  const uint64_t *nbytes_dev;  // optional: device-side byte count
  int aligned16;         // reads is 16-byte aligned
  const uint32_t *rs_bits;  // read-start bitmap, bit nbytes set
  uint64_t rs_words;
  int k, p, nbins, nbins_smem;
  uint64_t *skm_desc;    // (packed byte offset << 24) | length in bases
  uint32_t *skm_mm;      // minimizer of the superkmer
  uint64_t *skm_gpos;    // optional: global position of its first base
  uint8_t *packed;       // 2-bit packed superkmer bases
  unsigned long long *cursors;  // [0] superkmers, [1] packed bytes (16-byte rounded per tile)
  uint64_t cap_skm, cap_bytes;
  unsigned long long *bin_nskm, *bin_nkmers;
  uint32_t *err;
  unsigned long long *stamp;    // start time, or null
};

constexpr int kPartThreads = 256;
constexpr int kPartTile = 3328;  // windows of the smallest tile
size_t partition_smem_bytes(int nbins_smem);
__global__ void k_partition(PartArgs a);
constexpr int kBinChunk = 8192;          // superkmers per placement chunk (kBinRound where there are few)
constexpr int kBinRound = 2048;          // superkmers grouped by bin at a time
constexpr int kBinPlaceThreads = 512;
size_t bin_place_smem_bytes(uint32_t nbins);
constexpr int kBinPlaceMaxBins = 2048;   // larger bin counts use k_bin_scatter
__global__ void k_bin_count(const unsigned long long *n_skm_ptr, const uint32_t *mm, uint32_t nbins, uint32_t chunk,
                            uint64_t nch_cap, unsigned long long *mat, const uint32_t *err);
__global__ void k_bin_place(const unsigned long long *n_skm_ptr, const uint64_t *desc, const uint32_t *mm,
                            uint32_t nbins, uint32_t chunk, uint64_t nch_cap, const uint64_t *off, uint64_t *out_desc,
                            uint32_t *out_mm, const uint32_t *err);
// Zeroes the partition's counters and the read-start bitmap.
struct ClearArgs {
  unsigned long long *cursors;  // 4
  uint32_t *err;                // 4
  unsigned long long *bin_nskm, *bin_nkmers;  // nbins + 1
  uint32_t nbins;
  uint32_t *rs_bits;
  uint64_t rs_words;
  unsigned long long *stamp;  // start time, or null
};
__global__ void k_partition_clear(ClearArgs a);
__global__ void k_read_start_bits(const uint64_t *offs, uint64_t n_reads, uint32_t *bits);
__global__ void k_bin_scatter(const unsigned long long *n_skm_ptr, const uint64_t *desc,
                              const uint32_t *mm, uint32_t nbins, const uint64_t *bin_start,
                              unsigned long long *bin_fill, uint64_t *out_desc, uint32_t *out_mm,
                              const uint64_t *gpos, uint64_t *out_gpos, const uint32_t *err);
constexpr int kBinPrefixThreads = 1024;
__global__ void k_bin_prefix(const unsigned long long *bin_nskm,
                             const unsigned long long *bin_nkmers, uint32_t nbins,
                             uint64_t *bin_start, uint64_t *bin_kstart, unsigned long long *stamp);

// ---- counting ----
struct CountPlan {
  // inputs
  uint32_t nbins;
  const uint64_t *bin_start;   // superkmers per bin (exclusive prefix, nbins+1)
  const uint64_t *bin_kstart;  // k-mers per bin (exclusive prefix, nbins+1)
  uint32_t bucket_keys;        // most keys of a bucket of several digits
  uint32_t max_bits;           // digit bits cap (<= kCoarseMaxBits)
  uint64_t chunk_kmers;        // k-mers per expansion chunk
  int k;
  uint32_t *err;               // nothing is planned after an upstream overflow; flags a bin of 2^32 k-mers
  // outputs
  uint32_t *bin_bits;          // digit bits per bin
  uint64_t *chunk_base;        // first chunk of each bin (nbins+1)
  uint64_t *hist_base;         // first (digit, chunk) entry of each bin (nbins+1)
  unsigned long long *tickets; // 8, zeroed
};
__global__ void k_count_plan(CountPlan pl);
constexpr int kCountPlanThreads = 1024;

struct ExpandArgs {
  const uint64_t *desc;        // bin-ordered superkmer descriptors
  const uint64_t *koff;        // k-mer offset of each bin-ordered superkmer (n + 1)
  const uint8_t *packed;
  uint32_t nbins;
  const uint64_t *bin_start;
  const uint64_t *bin_kstart;
  const uint64_t *chunk_base;
  const uint64_t *hist_base;
  uint64_t *bucket_base;       // first bucket of each bin (written by the scan)
  const uint32_t *bin_bits;
  uint64_t chunk_kmers;
  int k;
  uint64_t *chunk_s0;          // first superkmer of each chunk
  uint32_t *hist;              // (bin, chunk, digit) counts, then write offsets in the bin per bucket
  uint32_t *digit_total;       // per (bin, digit), 1 << max_bits entries per bin
  uint16_t *lut;               // bucket (of its bin) of every digit, 1 << max_bits entries per bin
  uint32_t max_bits;
  uint32_t bucket_keys;
  void *keys;                  // scatter output (uint64 or u128)
  void *flat;                  // the keys in k-mer order (written by the histogram, read by the scatter)
  uint64_t keys_cap;          // of keys and flat
  uint32_t *big_list;          // buckets of at least big_min keys (listed by the scan, counted first)
  unsigned long long *big_count;  // zeroed
  uint64_t big_min;
  uint32_t *bucket_head;       // zeroed with the offsets
  uint32_t *unit_start;        // start of each bucket of a bin, 1 << max_bits entries per bin
  uint32_t *bin_units;         // buckets of each bin
  unsigned long long *scan_done;  // zeroed
  uint32_t *err;
  unsigned long long *stamp;   // start time of the scatter, or null
};
__global__ void k_chunk_first(ExpandArgs a);
template <typename K> __global__ void k_bucket_hist(ExpandArgs a);
__global__ void k_bucket_scan(ExpandArgs a);
__global__ void k_bucket_offsets(ExpandArgs a, uint64_t *bucket_start, uint64_t *bucket_size);
constexpr int kBucketOffsetThreads = 128;
template <typename K, int CTAS> __global__ void k_bucket_scatter(ExpandArgs a);
constexpr int kBucketScanThreads = 1024;
constexpr int kBucketHistThreads = 256;
template <typename K> size_t bucket_scatter_smem_bytes(int ctas);

struct SortCountArgs {
  uint32_t nbins;
  const uint64_t *bucket_base;    // buckets per bin (prefix, nbins + 1)
  const uint64_t *bucket_start;   // first key of each bucket
  const uint64_t *bucket_size;
  void *keys;                     // bucketed keys
  void *scratch;                  // second buffer of oversized buckets, at their own key range
  void *stage_keys;               // runs of bucket g at [bucket_start[g], + its distinct count)
  uint32_t *stage_counts;
  uint64_t stage_cap;
  unsigned long long *bucket_d;   // distinct keys of each bucket
  unsigned long long *ticket;     // zeroed
  uint32_t *big_list;             // buckets of at least big_min keys (from the scan), then rejected ones
  unsigned long long *big_count;
  unsigned long long *big_ticket;  // zeroed
  // slices of opened buckets: bucket, offset in it, keys, distinct keys (until
  // then: 1 where copies of a key are to be added); a bucket's tasks follow one another
  uint4 *tasks;
  uint64_t task_cap;
  unsigned long long *task_count, *task_ticket;  // zeroed
  uint32_t *bucket_head;           // first task + 1 of each bucket, 0: none (zeroed before)
  uint64_t big_min;
  uint32_t *err;
  unsigned long long *stamp;   // start time of k_bucket_sort, or null
};
template <typename K, bool NARROW> __global__ void k_bucket_sort(SortCountArgs a);
template <typename K> size_t bucket_sort_smem_bytes();
constexpr int kBucketSortThreads = 256;
template <typename K> __global__ void k_bucket_open(SortCountArgs a);
template <typename K> __global__ void k_bucket_slices(SortCountArgs a);
template <typename K> size_t bucket_count_smem_bytes();
template <typename K> uint64_t bucket_count_cap();  // largest bucket of k_bucket_sort
template <typename K>
__global__ void k_compact_runs(const K *stage_keys, const uint32_t *stage_counts, const uint64_t *bucket_start,
                               const unsigned long long *bucket_d, const uint64_t *bucket_out,
                               const uint64_t *bucket_base, uint32_t nbins, K *out_keys, uint32_t *out_counts,
                               uint64_t *bin_out, const uint32_t *bucket_head, const uint4 *tasks,
                               const unsigned long long *task_count, const uint32_t *err);
constexpr int kBucketCountThreads = 512;
constexpr uint32_t kCoarseTarget = 8192;
// Most keys of a bucket of several digits for a tuned target (an upper bound of
// the mean): at the default target 3584 8-byte or 3072 16-byte keys, of the
// 4096 (3072) that k_bucket_sort takes.  (900 M bases at k 31: 28.8 ms with
// 3072, 28.3 with 3584, 28.0 with 4096, but mostly distinct long reads 7.3 ms
// with 3584 and 7.4 with either; k 63: 7.1 ms with 2048, 6.8 with 2560, 6.7
// with 3072.)
template <typename K> constexpr uint32_t bucket_target(uint32_t target) {
  return sizeof(K) == 8 ? target / 16 * 7 : target / 8 * 3;
}
constexpr uint32_t kCoarseMaxBits = 12;
constexpr uint64_t kChunkKmers = 65536;
// Doubled where there are eight for each of the histogram's CTAs (eight an SM),
// which leaves four: fewer rows of digits (720 M k-mers in bins of 2.8 M, 9.3
// for each, 64 K / 128 K / 256 K: histogram + scatter 8.85 / 8.56 / 8.71 ms; 151 M,
// 1.9 for each: 2.00 / 2.04 / 2.19).  What lies between was not measured.  `keys`
// is the room for keys: the bases where a whole pipeline runs, the k-mers where a
// partition is counted.
// Halved down to this while there are fewer chunks than the histogram has CTAs
// (histogram + scatter, 64 K / 32 K / 16 K: 20 M bases 389 / 319 / 269 us, 60 M
// 718 / 684 / 678, 120 M 1331 / 1328 / 1387).
constexpr uint64_t kChunkKmersMin = 16384;
inline uint64_t default_chunk(uint64_t keys, int n_sms) {
  uint64_t chunk = keys / kChunkKmers >= 64 * (uint64_t)n_sms ? 2 * kChunkKmers : kChunkKmers;
  while (chunk > kChunkKmersMin && keys / chunk < 8 * (uint64_t)n_sms) chunk /= 2;
  return chunk;
}
// Largest mean bin (room for keys, as above) whose 8-byte keys are scattered by two CTAs an SM
// with tiles of 7168 keys rather than one with 16384: their phases overlap,
// but in larger bins a bucket's run of the smaller tile ends within few 32-byte
// sectors (134.7 M k-mers, one CTA / two: 256 bins 0.91 / 0.86 ms, 64 bins 0.98 /
// 0.95, 31 bins 1.06 / 1.27; 720 M in 1024 bins 4.72 / 4.26).  16-byte keys
// gain nothing from it (112.8 M in 128 bins: 1.02 / 1.09).
constexpr uint64_t kScatterPairBin = 2 << 20;

// device-wide exclusive scan of uint64 counters (n <= 2^31); out[n] = total.
// Returns the kernels launched.
uint32_t scan_u64(const unsigned long long *in, uint64_t *out, uint64_t n, uint64_t *block_tmp, cudaStream_t st);
size_t scan_u64_tmp_words(uint64_t n);
// the same over a device-side length min(*n_dev, n_cap)
uint32_t scan_u64_dev(const unsigned long long *in, uint64_t *out, uint64_t n_cap, const uint64_t *n_dev,
                      uint64_t *block_tmp, cudaStream_t st, unsigned long long *stamp = nullptr);
// the same over the k-mers of each superkmer
uint32_t scan_kmers_dev(const uint64_t *desc, int k, uint64_t *out, uint64_t n_cap, const uint64_t *n_dev,
                        uint64_t *block_tmp, cudaStream_t st, unsigned long long *stamp = nullptr);

}  // namespace gkc

namespace gkc {
// Run-length pass over sorted keys (distinct keys + first indices).
uint64_t rle_block_count(uint64_t n);
template <typename K>
void rle_runs(const K *sorted, uint64_t n, unsigned long long *blk, uint64_t *blk_off, uint64_t *tmp,
              const unsigned long long *cursor, K *out_keys, uint64_t *starts, cudaStream_t st);

// the same over the packed bytes of superkmers, given by length or by descriptor
uint32_t scan_len_bytes(const uint32_t *len, uint64_t *out, uint64_t n, uint64_t *block_tmp, cudaStream_t st);
uint32_t scan_desc_bytes(const uint64_t *desc, uint64_t *out, uint64_t n, uint64_t *block_tmp, cudaStream_t st);

}  // namespace gkc
