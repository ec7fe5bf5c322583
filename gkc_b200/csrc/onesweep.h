// Onesweep LSD radix sort (device-wide) interface.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

namespace gkc {

struct OnesweepScratch {
  unsigned long long *hist;      // 16 * 256
  unsigned long long *lookback;  // onesweep_lookback_words(n_max)
  unsigned long long *ticket;    // 1
  uint32_t *err;
  int max_ctas;
};
struct OnesweepStatus {
  int result_in_alt;  // 1 if the sorted keys ended in `alt`
};
size_t onesweep_lookback_words(uint64_t n_max);
template <typename K>
OnesweepStatus onesweep_sort(K *keys, K *alt, const uint64_t *n_dev, uint64_t n_max, int key_bits,
                             OnesweepScratch s, cudaStream_t st, uint32_t *launches);
// n pairs (key, uint32 value) sorted by key (n == *n_dev); equal keys keep
// their input order.  Where the keys are long, only their leading bits are
// sorted by passes and the runs of equal leading bits are put in order by one
// more kernel (`partial`), all but runs of more than a few hundred keys that
// are not all equal: lookback[0] counts those once the stream is done.
struct PairsStatus {
  int result_in_alt;  // 1 if the sorted pairs ended in `alt`
  bool partial;
};
template <typename K>
PairsStatus sort_pairs(K *keys, K *alt, uint32_t *vals, uint32_t *valt, const uint64_t *n_dev, uint64_t n, int key_bits,
                       OnesweepScratch s, cudaStream_t st, uint32_t *launches);
// Sorts the n_runs (> 0) counted ones; waits for the stream.  Returns 1 if the
// sorted pairs are in `alt` then.
template <typename K>
int sort_pairs_rest(PairsStatus done, uint64_t n_runs, K *keys, K *alt, uint32_t *vals, uint32_t *valt,
                    const uint64_t *n_dev, uint64_t n, int key_bits, OnesweepScratch s, cudaStream_t st,
                    uint32_t *launches);

}  // namespace gkc
