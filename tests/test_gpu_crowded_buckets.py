"""Buckets that one key fills: its copies are left out where a bucket is
opened, at any level, and added to its run.  The key the smallest, the largest
or in the middle, about a quarter of the keys or nearly all, buckets about the
size from which this is looked for, another such key on the next level.  The
keys are superkmers of exactly k bases; the expected list is their sorted
unique canonical values."""
import time

import numpy as np
import pytest

import gkc_b200 as G
from test_gpu_count_buckets import check, prefixed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


def crowd(rng, n, k, share, place, deep=8):
    """n keys with `deep` leading A, one of them `share` of all."""
    codes = prefixed(rng, n, k, [0] * deep)
    codes[:, -1] = 0  # its reverse complement begins with T: each key is its own canonical form
    one = codes[0].copy()
    one[deep:deep + 6] = {"first": 0, "middle": 1, "last": 3}[place]
    codes[rng.permutation(n)[:int(share * n)]] = one
    return codes


@pytest.mark.parametrize("k", [21, 31, 32, 33, 63])
@pytest.mark.parametrize("place", ["first", "middle", "last"])
@pytest.mark.parametrize("n,share", [(70_000, 0.26), (70_000, 0.9), (70_000, 0.9999), (100_000, 0.24), (12_289, 0.5),
                                     (16_385, 0.5), (16_384, 0.5), (30_000, 0.25)])
def test_one_key(ctx, n, share, place, k):
    check(ctx, crowd(np.random.default_rng(n + k), n, k, share, place))


@pytest.mark.parametrize("k", [31, 63])
def test_levels(ctx, k):
    """Crowds within crowds: the keys that share ever more leading bases with
    one key, half of the rest each time, and the outliers around them."""
    rng = np.random.default_rng(k)
    parts, n = [], 120_000
    for deep in (8, 14, 20, 26):
        parts.append(crowd(rng, n, k, 0.5, "middle" if deep % 4 else "first", min(deep, k - 8)))
        n = n * 2 // 3
    codes = np.concatenate(parts)
    check(ctx, codes[rng.permutation(len(codes))])


def test_time_of_few_letters():
    import torch
    r = np.random.default_rng(3)
    n, ms = 6_000_000, []
    offs = torch.arange(0, n + 1, 150, dtype=torch.int64, device="cuda")
    with G.Context(0) as ctx:
        for rare in (0.75, 0.015):
            d = torch.from_numpy(np.frombuffer(b"ACGT", np.uint8)[(r.random(n) < rare) * r.integers(1, 4, n)]).cuda()
            best = 1e9
            for _ in range(5):
                torch.cuda.synchronize()
                t = time.perf_counter()
                ctx.pipeline_device(d, n, offs, offs.numel() - 1, G.params(21, 7, 31))
                best = min(best, time.perf_counter() - t)
            ms.append(1e3 * best)
    assert ms[1] < 25 * ms[0], ms  # one bucket of most keys, opened by one CTA
