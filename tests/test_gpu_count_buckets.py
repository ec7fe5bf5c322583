"""The count kernel at the edges of its bucket table: buckets of a given
number of distinct keys, with and without repeats, from one key to more than
the table takes (slices, and sub-buckets that no digit splits).  The keys are
given as superkmers of exactly k bases; the expected list is their sorted
unique canonical values.  Whole numbers: equality, no tolerance."""
import numpy as np
import pytest

import gkc_b200 as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


def canonical(codes):
    """Canonical key of every row of base codes, as Python integers."""
    k = codes.shape[1]
    low = [int("".join(map(str, r)), 4) for r in codes.tolist()]
    rc = [int("".join(map(str, r)), 4) for r in (3 - codes[:, ::-1]).tolist()]
    assert k <= 64
    return [min(a, b) for a, b in zip(low, rc)]


def count(ctx, codes):
    k = codes.shape[1]
    n = len(codes)
    width = (k + 3) // 4
    padded = np.zeros((n, 4 * width), np.uint8)
    padded[:, :k] = codes
    q = padded.reshape(n, width, 4)
    packed = (q[..., 0] << 6 | q[..., 1] << 4 | q[..., 2] << 2 | q[..., 3]).astype(np.uint8)
    nd = ctx.count_superkmers_host(k, np.full(n, k, np.uint32), packed.reshape(-1))
    v = G.CountView()
    v.n_distinct, v.nbins, v.key_words = nd, 1, 1 if k <= 32 else 2
    _, keys, counts = ctx.count_copy_out(v)
    got = [int(r[0]) | (int(r[1]) << 64 if len(r) > 1 else 0) for r in keys]
    return got, counts


def check(ctx, codes):
    want = {}
    for x in canonical(codes):
        want[x] = want.get(x, 0) + 1
    got, counts = count(ctx, codes)
    assert got == sorted(want)
    assert counts.tolist() == [want[x] for x in got]


def prefixed(rng, n, k, prefix):
    codes = rng.integers(0, 4, (n, k), dtype=np.uint8)
    codes[:, :len(prefix)] = prefix
    return codes


# 8-byte keys: the table takes 4096 distinct keys; 16-byte keys: 3072
EDGES = [1, 2, 8, 9, 31, 32, 33, 255, 257, 513, 2049, 3071, 3072, 3073, 4095, 4096, 4097, 6200, 9000]


@pytest.mark.parametrize("k", [16, 25, 32, 33, 63])
@pytest.mark.parametrize("distinct", EDGES)
def test_one_bucket(ctx, k, distinct):
    """All keys start with eight A: one bucket whatever the digits."""
    rng = np.random.default_rng(1000 * k + distinct)
    codes = prefixed(rng, distinct, k, [0] * 8)
    check(ctx, codes)
    # each key one to seven times, in random order
    rep = np.repeat(codes, rng.integers(1, 8, distinct), axis=0)
    check(ctx, rep[rng.permutation(len(rep))])


@pytest.mark.parametrize("k", [31, 63])
def test_one_key_many_times(ctx, k):
    """Counts above 16 bits: the bucket is larger than the table's counters take."""
    rng = np.random.default_rng(k)
    one = prefixed(rng, 1, k, [0] * 8)
    few = prefixed(rng, 40, k, [0] * 8)
    check(ctx, np.concatenate([np.repeat(one, 70_000, axis=0), few]))
    check(ctx, np.repeat(one, 65_535, axis=0))


@pytest.mark.parametrize("k", [31, 63])
def test_clusters_no_digit_splits(ctx, k):
    """Two neighbouring clusters of keys that share all but their last bases,
    and an outlier that sets the bucket's range: sub-buckets of more distinct
    keys than the table takes, one after the other."""
    rng = np.random.default_rng(7 + k)
    deep = [0] * 8 + [1] * (k - 8 - 9)
    a = prefixed(rng, 12_000, k, deep[:-1] + [1])
    b = prefixed(rng, 9_000, k, deep[:-1] + [2])
    c = prefixed(rng, 2_000, k, [0] * 8 + [3] * 4)
    codes = np.concatenate([a, b, c, a[:500]])
    check(ctx, codes[rng.permutation(len(codes))])
