"""Superkmers packed for the exchange and handed over from the host, at the
edges of the kernels that move them: warps with fewer than 32 superkmers,
ranges that begin at odd addresses, superkmers longer than the staging area,
destinations without any, and group sizes around a block and the small scan."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F
from gkc_b200 import synth

pytestmark = pytest.mark.gpu


def reads_of(kind):
    if kind == "one":
        return np.frombuffer(b"ACGTTGCATGCCGATAGGCTAACTGTACCGAT", np.uint8).copy(), np.array([0, 32], np.uint64)
    if kind == "long":  # homopolymers: superkmers of 15 000 bases among short ones
        parts = [synth.iid_reads(7, 40, 100, 0.0)[0], np.full(15000, 65, np.uint8),
                 synth.iid_reads(8, 40, 100, 0.0)[0], np.full(4100, 67, np.uint8)]
        lens = [100] * 40 + [15000] + [100] * 40 + [4100]
        return np.concatenate(parts), np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    return synth.iid_reads(9, 700, 150, 0.003)


@pytest.mark.parametrize("kind", ["one", "long", "many"])
@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("bounds", [[0, 16], [0, 5, 5, 16], [0, 1, 2, 3, 16]])
def test_pack_moves_every_superkmer(kind, shift, bounds):
    import torch
    reads, offs = reads_of(kind)
    d_reads, d_offs = torch.from_numpy(reads).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        v = ctx.partition_device(d_reads, len(reads), d_offs, len(offs) - 1, G.params(15, 7, 16))
        bin_off, lens, boff, packed, _ = ctx.partition_copy_out(v)
        nbytes = (lens.astype(np.int64) + 3) // 4
        desc = torch.zeros(len(lens), dtype=torch.int64, device="cuda")
        room = torch.full((int(nbytes.sum()) + shift + 8,), 0xEE, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        skm, byt, _, _ = ctx.exchange_pack(v, bounds, desc, room[shift:])
    want = np.concatenate([packed[int(b):int(b) + int(m)] for b, m in zip(boff, nbytes)])
    got = room.cpu().numpy()
    assert np.array_equal(got[shift:shift + len(want)], want)
    assert (got[:shift] == 0xEE).all() and (got[shift + len(want):] == 0xEE).all()
    start = np.concatenate([[0], np.cumsum(nbytes)])[:-1]
    d = desc.cpu().numpy().view(np.uint64)
    assert np.array_equal((d & np.uint64(0xFFFFFF)).astype(np.uint32), lens)
    assert [int(x) for x in skm] == [int(bin_off[b] - bin_off[a]) for a, b in zip(bounds[:-1], bounds[1:])]
    for r in range(len(bounds) - 1):
        lo, hi = int(bin_off[bounds[r]]), int(bin_off[bounds[r + 1]])
        if hi > lo:
            assert np.array_equal((d[lo:hi] >> np.uint64(24)).astype(np.int64), start[lo:hi] - start[lo])
        assert int(byt[r]) == int(nbytes[lo:hi].sum())


@pytest.mark.parametrize("n", [0, 1, 31, 255, 256, 257, 24575, 24576, 24577])
@pytest.mark.parametrize("k", [3, 21, 33])
def test_group_from_the_host(n, k):
    r = np.random.default_rng(1000 * k + n)
    lens = r.integers(0, 50, n).astype(np.uint32)
    nbytes = (lens.astype(np.int64) + 3) // 4
    packed = r.integers(0, 4, int(nbytes.sum()), dtype=np.uint8)  # few distinct k-mers
    skms = F.Skms(np.zeros(n, np.uint32), lens, (np.cumsum(nbytes) - nbytes).astype(np.uint64), packed)
    want = F.oracle_count_bins(skms, k, 1)
    with G.Context(0) as ctx:
        nd = ctx.count_superkmers_host(k, lens, packed)
        assert nd == len(want["keys_lo"])
        _, keys, counts = ctx.count_copy_out(ctx.count_device(G.params(k, 3, 1)))
    assert np.array_equal(keys[:, 0], want["keys_lo"])
    if k > 32:
        assert np.array_equal(keys[:, 1], want["keys_hi"])
    assert np.array_equal(counts, want["counts"])
