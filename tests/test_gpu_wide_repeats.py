"""16-byte keys that mostly repeat, in more buckets than there are CTAs, so
that buckets are listed for the table unseen; with a distinct part after or
before them, and in one or many bins, against the oracle."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu


def reads_of(seed, genome, coverage, length, errors):
    r = np.random.default_rng(seed)
    g = r.integers(0, 4, genome)
    n = genome * coverage // length
    at = r.integers(0, genome - length, n)
    codes = g[at[:, None] + np.arange(length)]
    flip = r.random(codes.shape) < errors
    codes = np.where(flip, r.integers(0, 4, codes.shape), codes)
    return np.frombuffer(b"ACGT", np.uint8)[codes].reshape(-1)


@pytest.mark.parametrize("nbins", [1, 16])
@pytest.mark.parametrize("distinct", [0, 600_000])
def test_many_buckets_that_repeat(nbins, distinct):
    import torch
    k, p, length = 40, 9, 200
    reads = reads_of(3, 200_000, 24, length, 0.003)
    if distinct:
        extra = np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(4).integers(0, 4, distinct)]
        reads = np.concatenate([reads, extra])
    offs = np.arange(0, len(reads) + 1, length, dtype=np.uint64)
    want = F.oracle_count_bins(F.oracle_partition(reads, offs, k, p, 0, nbins), k, nbins)
    d_reads, d_offs = torch.from_numpy(reads.copy()).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        for _ in range(2):
            _, cv = ctx.pipeline_device(d_reads, len(reads), d_offs, len(offs) - 1, G.params(k, p, nbins))
            bin_off, keys, counts = ctx.count_copy_out(cv)
            assert np.array_equal(bin_off, want["bin_off"])
            assert np.array_equal(keys[:, 0], want["keys_lo"])
            assert np.array_equal(keys[:, 1], want["keys_hi"])
            assert np.array_equal(counts, want["counts"])
