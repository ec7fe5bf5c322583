"""Superkmers cut into pieces of a few k-mers: lengths around a piece, none,
one or thousands of k-mers, runs of superkmers without any (more than a
warp's batch of them), first and last in a group, against the oracle."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu


def lengths(kind, k, r):
    """k-mers a superkmer (0: shorter than k)."""
    if kind == "around":
        return r.integers(0, 14, 3000)
    if kind == "ones":
        return np.ones(4000, np.int64)
    if kind == "gaps":  # 33, 64 and 100 without k-mers in a row, at the ends and between
        one = [0] * 33 + [5, 0, 1, 4] + [0] * 64 + [8, 3] + [0] * 100 + [2] * 31
        return np.array(one * 9 + [0] * 40)
    if kind == "every other":
        w = r.integers(1, 30, 5000)
        w[::2] = 0
        return w
    if kind == "long":
        return np.array([4, 20000, 1, 70000, 3, 0, 2, 9] * 2)
    return np.array([int(kind)])


@pytest.mark.parametrize("k", [3, 21, 31, 32, 33, 47, 64])
@pytest.mark.parametrize("kind", ["around", "ones", "gaps", "every other", "long", "0", "1", "6", "7"])
def test_group_of_odd_superkmers(kind, k):
    r = np.random.default_rng(k)
    w = np.asarray(lengths(kind, k, r))
    lens = np.where(w > 0, w + k - 1, r.integers(0, k, len(w))).astype(np.uint32)
    nbytes = (lens.astype(np.int64) + 3) // 4
    packed = r.integers(0, 256, int(nbytes.sum()), dtype=np.uint8)
    skms = F.Skms(np.zeros(len(w), np.uint32), lens, (np.cumsum(nbytes) - nbytes).astype(np.uint64), packed)
    want = F.oracle_count_bins(skms, k, 1)
    with G.Context(0) as ctx:
        nd = ctx.count_superkmers_host(k, lens, packed)
        assert nd == len(want["keys_lo"])
        _, keys, counts = ctx.count_copy_out(ctx.count_device(G.params(k, 3, 1)))
    assert np.array_equal(keys[:, 0], want["keys_lo"])
    if k > 32:
        assert np.array_equal(keys[:, 1], want["keys_hi"])
    assert np.array_equal(counts, want["counts"])
