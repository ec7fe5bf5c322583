"""Groups of k-mers sorted by their lower word where they share the upper one:
k around the rule (by the bin's size), k-mers that cross a multiple of 2^32,
repeated and distinct, against the oracle."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F
from gkc_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [14, 15, 16, 17, 18, 20, 21, 22])
@pytest.mark.parametrize("copies", [1, 3, 12])
def test_k_around_the_rule(k, copies):
    import torch
    reads, _ = synth.iid_reads(k + copies, 600, 1000 // (1 + copies // 3), 0.0)
    if copies > 1:
        reads = np.tile(reads, copies)
    # k-mers that begin like the first and the last of an upper word's range
    edge = np.frombuffer((b"ACGTACTGAGGCTTAACCGTTAGCATCG" + b"A" * 18 + b"CAGTC" + b"C" * 19 + b"GATTC") * 40, np.uint8)
    reads = np.concatenate([reads, edge])
    offs = np.arange(0, len(reads), 500, dtype=np.uint64)
    offs = np.append(offs, np.uint64(len(reads)))
    want = F.oracle_count_bins(F.oracle_partition(reads, offs, k, 7, 0, 2), k, 2)
    d_reads, d_offs = torch.from_numpy(reads.copy()).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        _, cv = ctx.pipeline_device(d_reads, len(reads), d_offs, len(offs) - 1, G.params(k, 7, 2))
        bin_off, keys, counts = ctx.count_copy_out(cv)
    assert np.array_equal(bin_off, want["bin_off"])
    assert np.array_equal(keys[:, 0], want["keys_lo"])
    assert np.array_equal(counts, want["counts"])
