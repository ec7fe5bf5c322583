"""The tile kernels (superkmer partition, per-window minimizers) at the edges
of their tiles and words: shortest and longest windows of p-mers, reads that
end on word and tile boundaries, runs of bytes that are no base, superkmers
longer than a tile's halo, reads at unaligned device addresses.  Against the
oracle; whole numbers, no tolerance."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu

TILE, CORE = 3840, 3584  # windows per tile; core windows of a partition tile


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


def reads_of(seed):
    r = np.random.default_rng(seed)
    lens = [1, 31, 32, 33, 64, 95, 3, TILE - 1, TILE, TILE + 1, CORE, CORE + 1, 2 * CORE, 500, 8000, 17, 63, 64, 65]
    lens += r.integers(1, 400, 60).tolist()
    b = np.frombuffer(b"ACGTacgtUu", np.uint8)[r.integers(0, 10, sum(lens))].copy()
    offs = np.zeros(len(lens) + 1, np.uint64)
    offs[1:] = np.cumsum(lens)
    n = len(b)
    for at in (CORE - 5, TILE - 40, 2 * CORE, 3 * TILE + 7):  # no bases across word and tile boundaries
        b[at:at + int(r.integers(1, 70))] = ord("N")
    b[n // 3:n // 3 + 900] = ord("A")                        # one long superkmer of filtered p-mers
    b[n // 2:n // 2 + 700] = np.tile(np.frombuffer(b"CAG", np.uint8), 234)[:700]
    b[r.integers(0, n, 12)] = np.frombuffer(b"\x00 \xc1-@`.*2XRY", np.uint8)  # bytes near the letters' codes
    return b, offs


def on_device(reads, offs, shift):
    import torch
    buf = torch.zeros(len(reads) + 64, dtype=torch.uint8, device="cuda")
    d_reads = buf[shift:shift + len(reads)]
    d_reads.copy_(torch.from_numpy(reads))
    d_offs = torch.from_numpy(offs.view(np.int64)).cuda()
    torch.cuda.synchronize()
    return buf, d_reads, d_offs


KP = [(3, 3), (16, 16), (17, 16), (31, 11), (32, 3), (36, 4), (37, 4), (64, 3), (64, 16), (25, 15)]


@pytest.mark.parametrize("shift", [0, 1, 8])
@pytest.mark.parametrize("k,p", KP)
def test_partition_tiles(ctx, k, p, shift):
    reads, offs = reads_of(10 * k + p)
    buf, d_reads, d_offs = on_device(reads, offs, shift)
    nb = 64
    want = F.oracle_partition(reads, offs, k, p, 0, nb)
    v = ctx.partition_device(d_reads, len(reads), d_offs, len(offs) - 1, G.params(k, p, nb))
    bin_off, lens, boff, packed, mm = ctx.partition_copy_out(v)
    bins = np.repeat(np.arange(nb, dtype=np.uint32), np.diff(bin_off).astype(np.int64))
    assert F.Skms(bins, lens, boff, packed, minimizer=mm).multisets(nb) == want.multisets(nb)


@pytest.mark.parametrize("shift", [0, 3])
@pytest.mark.parametrize("filter_id", [G.FILTER_NEW2, G.FILTER_ALL, G.FILTER_NEW, G.FILTER_SIGNATURE])
@pytest.mark.parametrize("k,p", KP)
def test_minimizer_tiles(ctx, k, p, filter_id, shift):
    import torch
    if filter_id == G.FILTER_SIGNATURE and p > 14:
        pytest.skip("covered by smaller p")
    reads, offs = reads_of(10 * k + p + 5)
    n = len(reads)
    buf, d_reads, d_offs = on_device(reads, offs, shift)
    mm = torch.zeros(n, dtype=torch.int32, device="cuda")
    pos = torch.zeros(n, dtype=torch.uint8, device="cuda")
    strand = torch.zeros(n, dtype=torch.int8, device="cuda")
    torch.cuda.synchronize()
    want = [np.full(n, 0xFFFFFFFF, np.uint32), np.full(n, 255, np.uint8), np.zeros(n, np.int8)]
    try:
        F.set_filter(filter_id)
        ctx.set_filter(filter_id)
        for i in range(len(offs) - 1):
            b, e = int(offs[i]), int(offs[i + 1])
            if e - b >= k:
                for w, x in zip(want, F.oracle_minimizers(reads[b:e], k, p, with_pos=True)):
                    w[b:b + len(x)] = x
        ctx.minimizers_device(d_reads, n, d_offs, len(offs) - 1, G.params(k, p, 1), mm, pos, strand)
    finally:
        F.set_filter(G.FILTER_NEW2)
        ctx.set_filter(G.FILTER_NEW2)
    assert np.array_equal(mm.cpu().numpy().view(np.uint32), want[0])
    assert np.array_equal(pos.cpu().numpy(), want[1])
    assert np.array_equal(strand.cpu().numpy(), want[2])


@pytest.mark.parametrize("shift", [0, 5])
@pytest.mark.parametrize("first", [0, 7])
@pytest.mark.parametrize("total", [1, 15, 16, 33, 8191, 8192, 8193, 40_000])
def test_hpc_tiles(ctx, total, first, shift):
    """Homopolymer compression over its 8192-byte tiles: runs and reads that
    end on tile, word and thread boundaries, empty reads, reads that do not
    start at the first byte, unaligned addresses."""
    import torch
    r = np.random.default_rng(100 * total + first)
    b = np.repeat(np.frombuffer(b"ACGTN", np.uint8)[r.integers(0, 5, total)], r.integers(1, 6, total))[:total].copy()
    if total > 8200:
        b[8100:8300] = ord("A")  # a run across a tile
    first = min(first, total - 1)
    cuts = np.unique(np.concatenate([r.integers(first, total + 1, 30), [first, total], np.arange(8192, total, 8192)]))
    cuts = cuts[cuts >= first]
    offs = np.concatenate([cuts[:1], cuts[:1], cuts, cuts[-1:]]).astype(np.uint64)  # empty reads at both ends
    buf, d_reads, d_offs = on_device(b, offs, shift)
    n = len(offs) - 1
    out = torch.zeros(total + 16, dtype=torch.uint8, device="cuda")[shift:]
    ooffs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    orig = torch.zeros(total + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.hpc_device(d_reads, total, d_offs, n, out, ooffs, orig)
    want, want_pos, want_offs = [], [], [0]
    for i in range(n):
        read = b[int(offs[i]):int(offs[i + 1])]
        keep = np.ones(len(read), bool)
        keep[1:] = read[1:] != read[:-1]
        want.append(read[keep])
        want_pos.append(np.flatnonzero(keep))
        want_offs.append(want_offs[-1] + int(keep.sum()))
    m = want_offs[-1]
    assert ooffs.cpu().tolist() == want_offs
    assert np.array_equal(out[:m].cpu().numpy(), np.concatenate(want))
    assert np.array_equal(orig[:m].cpu().numpy(), np.concatenate(want_pos))
    assert int(out[m:].sum()) == 0  # nothing written past the kept bytes
