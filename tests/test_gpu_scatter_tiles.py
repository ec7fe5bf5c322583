"""Chunks of several tiles in the scatter of k-mers to buckets, one CTA an SM
(mean bins above 2 M bases) and two, and buckets larger than one CTA sorts at
once, as a tuned shape asks for them.  Against the oracle."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu

PAIR = 2 << 20    # bases of a mean bin up to which two CTAs share an SM
TILE = 16384      # 8-byte keys of a tile where one has it
LAST = [1, TILE - 1, TILE, TILE + 1]


def one_read(bases, seed):
    r = np.random.default_rng(seed)
    b = np.frombuffer(b"ACGT", np.uint8)[r.integers(0, 4, bases)].copy()
    b[bases // 2:bases // 2 + bases // 8] = b[:bases // 8]  # repeats
    return b, np.array([0, bases], np.uint64)


def check(bases, k, tune):
    import torch
    reads, offs = one_read(bases, bases % 89)
    want = F.oracle_count_bins(F.oracle_partition(reads, offs, k, 7, 0, 1), k, 1)
    assert int(want["counts"].astype(np.int64).sum()) == bases - k + 1
    d_reads, d_offs = torch.from_numpy(reads).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        ctx.tune_set(G.TuneParams(*tune, 0, 0))
        _, cv = ctx.pipeline_device(d_reads, len(reads), d_offs, 1, G.params(k, 7, 1))
        _, keys, counts = ctx.count_copy_out(cv)
    assert np.array_equal(keys[:, 0], want["keys_lo"])
    if k > 32:
        assert np.array_equal(keys[:, 1], want["keys_hi"])
    assert np.array_equal(counts, want["counts"])


@pytest.mark.parametrize("chunk", [32768, 131072])
@pytest.mark.parametrize("last", LAST)
@pytest.mark.parametrize("k", [21, 45])
def test_tiles_of_a_chunk(k, last, chunk):
    kmers = (PAIR // chunk + 1) * chunk + last  # whole chunks, then a tile more or less
    check(kmers + k - 1, k, (0, chunk))


@pytest.mark.parametrize("bases", [PAIR - 1, PAIR, PAIR + 1])
def test_both_sides_of_the_rule(bases):
    check(bases, 31, (0, 32768))


@pytest.mark.parametrize("k", [25, 63])
@pytest.mark.parametrize("target", [256, 4096, 16384, 65536])
def test_buckets_asked_for(target, k):
    check(PAIR + 4321, k, (target, 0))
