"""The scatter of k-mers to buckets at the edges of its tiles and chunks, on
both sides of the rule that takes one or two CTAs an SM (mean bins above 2 M
k-mers), against the oracle."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F
from gkc_b200 import synth

pytestmark = pytest.mark.gpu

# k-mers of one bin: a tile (7168, 8192 or 16384 keys) or a chunk (16384) more or less one; then the rule's two sides
SIZES = [7167, 7168, 7169, 8192, 8193, 16383, 16384, 16385, 33000, 2 << 20, (2 << 20) + 70000]


@pytest.mark.parametrize("k", [21, 45])
@pytest.mark.parametrize("n", SIZES)
def test_tile_and_chunk_edges(n, k):
    import torch
    length = 1000
    reads_n = (n + length - k) // (length - k + 1)
    reads, _ = synth.iid_reads(n % 97, reads_n, length, 0.0)
    last = n - (reads_n - 1) * (length - k + 1) + k - 1
    lens = [length] * (reads_n - 1) + [last]
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    reads = reads[:int(offs[-1])]
    skm = F.oracle_partition(reads, offs, k, 7, 0, 1)
    want = F.oracle_count_bins(skm, k, 1)
    assert int(want["counts"].astype(np.int64).sum()) == n
    d_reads, d_offs = torch.from_numpy(reads.copy()).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        _, cv = ctx.pipeline_device(d_reads, len(reads), d_offs, len(offs) - 1, G.params(k, 7, 1))
        _, keys, counts = ctx.count_copy_out(cv)
    assert np.array_equal(keys[:, 0], want["keys_lo"])
    if k > 32:
        assert np.array_equal(keys[:, 1], want["keys_hi"])
    assert np.array_equal(counts, want["counts"])
