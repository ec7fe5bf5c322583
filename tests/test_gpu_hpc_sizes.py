"""Homopolymer compression on both sides of the size from which the reads'
offsets have a kernel of their own (a tile of 8192 bytes for each of four CTAs
on 148 SMs), against a compaction by numpy."""
import numpy as np
import pytest

import gkc_b200 as G

pytestmark = pytest.mark.gpu

EDGE = 148 * 4 * 8192


@pytest.mark.parametrize("orig", [True, False])
@pytest.mark.parametrize("total", [EDGE - 8191, EDGE, EDGE + 1, 2 * EDGE + 77])
def test_compressed_reads_and_offsets(total, orig):
    import torch
    r = np.random.default_rng(total)
    b = np.repeat(np.frombuffer(b"ACGTN", np.uint8)[r.integers(0, 5, total)], r.integers(1, 4, total))[:total].copy()
    cuts = np.unique(np.concatenate([[0, total], r.integers(0, total, total // 300)])).astype(np.uint64)
    offs = np.concatenate([cuts[:1], cuts[:5], cuts[4:], cuts[-1:], cuts[-1:]])  # some reads are empty
    n = len(offs) - 1
    starts = np.zeros(total + 1, bool)
    starts[offs.astype(np.int64)] = True
    keep = starts[:total].copy()
    keep[1:] |= b[1:] != b[:-1]
    before = np.concatenate([[0], np.cumsum(keep)])
    first = np.maximum.accumulate(np.where(starts[:total], np.arange(total), 0))
    d, o = torch.from_numpy(b).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    out = torch.zeros(total, dtype=torch.uint8, device="cuda")
    ooffs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    pos = torch.zeros(total, dtype=torch.int32, device="cuda")
    with G.Context(0) as ctx:
        ctx.hpc_device(d, total, o, n, out, ooffs, pos if orig else None)
    m = int(before[-1])
    assert np.array_equal(ooffs.cpu().numpy(), before[offs.astype(np.int64)])
    assert np.array_equal(out[:m].cpu().numpy(), b[keep]) and int(out[m:].sum()) == 0
    if orig:
        assert np.array_equal(pos[:m].cpu().numpy(), (np.arange(total) - first)[keep])
