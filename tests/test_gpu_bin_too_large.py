"""A bin of 2^32 k-mers or more is refused (offsets inside a bin are 32-bit):
the call ends with an error before any kernel works on the bin, and the
context goes on counting."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu

GKC_ERR_CAPACITY = 6
LONGEST = (1 << 24) - 1  # bases of a superkmer


@pytest.mark.parametrize("k", [32, 9])
def test_bin_of_too_many_kmers(k):
    import torch
    if torch.cuda.mem_get_info()[0] < 125 << 30:
        pytest.skip("needs 125 GB of free device memory")
    n = (1 << 32) // (LONGEST - k + 1) + 1
    assert n * (LONGEST - k + 1) >= 1 << 32
    lens = np.full(n, LONGEST, np.uint32)
    packed = np.zeros(n * ((LONGEST + 3) // 4), np.uint8)
    few = np.array([100, k, 57], np.uint32)
    some = np.random.default_rng(k).integers(0, 256, int(((few + 3) // 4).sum()), dtype=np.uint8)
    with G.Context(0) as ctx:
        with pytest.raises(G.GkcError) as e:
            ctx.count_superkmers_host(k, lens, packed)
        assert e.value.status == GKC_ERR_CAPACITY and "2^32" in str(e.value)
        got = ctx.count_superkmers_host(k, few, some)
    first = np.concatenate([[0], np.cumsum((few + 3) // 4)]).astype(np.uint64)
    skm = F.Skms(np.zeros(3, np.uint32), few, first[:3], some)
    assert got == len(F.oracle_count_bins(skm, k, 1)["counts"])
