"""Pairs sorted by their leading bits and then run by run: runs around the
length that is ranked in shared memory and around a tile, k-mers that share
many leading bases (their runs are left to a sort of their own, or, where
they are most of the input, all pairs are sorted), one k-mer repeated, and
few keys; position lists and merged lists against the oracle."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F
from gkc_b200 import synth

pytestmark = pytest.mark.gpu

BASES = np.frombuffer(b"ACGT", np.uint8)


def shared_prefix(r, k, n, lead, distinct, group):
    """n reads of one k-mer each: `lead` bases of the group's own, then one of
    `distinct` tails."""
    tails = BASES[r.integers(0, 4, (distinct, k - lead))]
    reads = np.full((n, k), 65, np.uint8)
    reads[:, lead:] = tails[r.integers(0, distinct, n)]
    reads[:, 4:7] = BASES[[group // 16, group // 4 % 4, group % 4]]
    return reads.reshape(-1)


def build(seed, k, groups, more):
    """Groups (reads, leading bases, tails) and `more` random reads of 150 bases."""
    r = np.random.default_rng(seed)
    parts, lens = [], []
    for g, (n, lead, distinct) in enumerate(groups):
        parts.append(shared_prefix(r, k, n, lead, distinct, g))
        lens += [k] * n
    parts.append(BASES[r.integers(0, 4, more * 150)])
    lens += [150] * more
    order = r.permutation(len(lens))
    starts = np.concatenate([[0], np.cumsum(lens)])
    flat = np.concatenate(parts)
    reads = np.concatenate([flat[starts[i]:starts[i + 1]] for i in order])
    offs = np.concatenate([[0], np.cumsum(np.asarray(lens)[order])]).astype(np.uint64)
    return np.ascontiguousarray(reads), offs


CASES = [
    [],
    [(1, 18, 1)],
    [(511, 18, 400), (512, 17, 400), (513, 16, 400)],
    [(1023, 18, 900), (1024, 17, 5), (1537, 16, 1000)],
    [(6000, 17, 1)],                       # one k-mer: long, but in order
    [(6000, 17, 2), (700, 16, 700)],
    [(30000, 17, 9000), (2000, 16, 40)],   # more than half of all
]


@pytest.mark.parametrize("k", [31, 45, 63])
@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("more", [3, 200])
def test_position_lists(k, case, more):
    import torch
    reads, offs = build(100 * case + k, k, CASES[case], more)
    d_reads, d_offs = torch.from_numpy(reads).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    want = F.oracle_subsample(reads, offs, k, 7, 1)
    with G.Context(0) as ctx:
        from test_gpu_windows import subsample
        nd, kw, keys, pos_off, pos = subsample(torch, ctx, reads, offs, k, 7, 1)
    assert np.array_equal(keys[:, 0], want["keys_lo"])
    if kw == 2:
        assert np.array_equal(keys[:, 1], want["keys_hi"])
    assert np.array_equal(pos_off, want["pos_off"])
    assert np.array_equal(pos, want["pos"])


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_merged_lists(k, case):
    import torch
    reads, offs = build(100 * case + k, k, CASES[case], 40)
    d_reads, d_offs = torch.from_numpy(reads).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    want = F.oracle_count_bins(F.oracle_partition(reads, offs, k, 7, 0, 1), k, 1)
    with G.Context(0) as ctx:
        ctx.pipeline_device(d_reads, len(reads), d_offs, len(offs) - 1, G.params(k, 7, 8))
        _, keys, counts = ctx.count_output(merged=True, key_words=1 if k <= 32 else 2)
    assert np.array_equal(keys[:, 0], want["keys_lo"])
    if k > 32:
        assert np.array_equal(keys[:, 1], want["keys_hi"])
    assert np.array_equal(counts, want["counts"])
