"""The count filter at the edges of its tiles: entries around one and two
tiles, bins that end inside and on a tile, ranges that keep all, some and
nothing, against the oracle's list."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 2047, 2048, 2049, 4096, 5000])
@pytest.mark.parametrize("nbins", [1, 7, 300])
def test_ranges_and_tiles(n, nbins):
    import torch
    k, r = 21, np.random.default_rng(n + nbins)
    seq = np.frombuffer(b"ACGT", np.uint8)[r.integers(0, 4, n + k - 1)]
    again = [seq[i:i + 60] for i in r.integers(0, max(1, len(seq) - 60), n // 40)] * 2  # some k-mers three times
    parts = [seq] + [a for a in again if len(a) >= k]
    reads = np.concatenate(parts)
    offs = np.concatenate([[0], np.cumsum([len(x) for x in parts])]).astype(np.uint64)
    want = F.oracle_count_bins(F.oracle_partition(reads, offs, k, 7, 0, nbins), k, nbins)
    d_reads, d_offs = torch.from_numpy(reads.copy()).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        ctx.pipeline_device(d_reads, len(reads), d_offs, len(offs) - 1, G.params(k, 7, nbins))
        for lo, hi in ((1, 0xFFFFFFFF), (2, 0xFFFFFFFF), (1, 1), (2, 3), (1000, 2000)):
            keep = (want["counts"] >= lo) & (want["counts"] <= hi)
            places = np.concatenate([[0], np.cumsum(keep)])
            bin_off, keys, counts = ctx.count_output(lo, hi, nbins=nbins)
            assert np.array_equal(np.asarray(bin_off)[:nbins + 1], places[want["bin_off"].astype(np.int64)])
            assert np.array_equal(keys[:, 0], want["keys_lo"][keep])
            assert np.array_equal(counts, want["counts"][keep])
            _, mkeys, mcounts = ctx.count_output(lo, hi, merged=True)
            order = np.argsort(want["keys_lo"][keep])
            assert np.array_equal(mkeys[:, 0], want["keys_lo"][keep][order])
            assert np.array_equal(mcounts, want["counts"][keep][order])
