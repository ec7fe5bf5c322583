"""The superkmers of a group counted from host memory, copied out again: as
they came, and without minimizers."""
import numpy as np
import pytest

import gkc_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 30_000])
def test_group_copied_out(n):
    r = np.random.default_rng(n)
    lens = r.integers(1, 60, n).astype(np.uint32)
    nbytes = (lens.astype(np.int64) + 3) // 4
    packed = r.integers(0, 256, int(nbytes.sum()), dtype=np.uint8)
    bin_off, got_lens, got_off = np.zeros(2, np.uint64), np.zeros(n, np.uint32), np.zeros(n, np.uint64)
    got, mm = np.zeros(len(packed), np.uint8), np.zeros(n, np.uint32)
    with G.Context(0) as ctx:
        ctx.count_superkmers_host(21, lens, packed)
        ctx._check(ctx._L.gkc_partition_copy_out(ctx.h, *(a.ctypes.data for a in (bin_off, got_lens, got_off, got, mm))),
                   "partition_copy_out")
    assert bin_off.tolist() == [0, n]
    assert np.array_equal(got_lens, lens) and np.array_equal(got, packed)
    assert np.array_equal(got_off, (np.cumsum(nbytes) - nbytes).astype(np.uint64))
    assert (mm == 0xFFFFFFFF).all()
