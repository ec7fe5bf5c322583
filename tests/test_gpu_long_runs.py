"""Superkmers that run past a partition tile and its halo: their ends at the
steps of the block's search for them, ended by other bases, a byte that is no
base, the read's end and the data's end.  Against the oracle; and such reads
take no longer than a few times the others, whatever the runs' length."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu

SEEN = 3808  # the first tile has the windows [0, 3808), of which 3584 are its own
ENDS = [-1, 0, 1, 2, 254, 255, 256, 257, 258, 511, 512, 513, 1500]


@pytest.mark.parametrize("k,p", [(31, 11), (25, 15), (64, 3)])
@pytest.mark.parametrize("stop", ["bases", "N", "read", "data"])
def test_ends(k, p, stop):
    r = np.random.default_rng(k)
    letters = np.frombuffer(b"ACGT", np.uint8)
    first = 3500 if k < 64 else 3400
    with G.Context(0) as ctx:
        for end in ENDS:
            n = SEEN + end + k - 1 - first  # the last window of the run's own bases begins at SEEN + end - 1
            run = np.resize(np.frombuffer(b"CAGGT", np.uint8), n)
            head, tail = letters[r.integers(0, 4, first)], letters[r.integers(0, 4, 400)]
            cuts = [0, first + n + 400]
            if stop == "N":
                tail[0] = ord("N")
            elif stop == "read":
                cuts = [0, first + n, first + n + 400]
            elif stop == "data":
                tail, cuts = tail[:0], [0, first + n]
            reads, offs = np.concatenate([head, run, tail]), np.array(cuts, np.uint64)
            want = F.oracle_partition(reads, offs, k, p, 0, 32)
            v = ctx.partition_host(reads, offs, G.params(k, p, 32))
            bin_off, lens, boff, packed, mm = ctx.partition_copy_out(v)
            bins = np.repeat(np.arange(32, dtype=np.uint32), np.diff(bin_off).astype(np.int64))
            assert F.Skms(bins, lens, boff, packed).multisets(32) == want.multisets(32), end
            assert int(want.len.max()) >= n - k  # the run is one superkmer


@pytest.mark.parametrize("run,every", [(300, 2000), (1000, 4000), (8000, 16000)])
def test_time_of_runs(run, every):
    import torch
    letters = np.frombuffer(b"ACGT", np.uint8)
    plain = letters[np.random.default_rng(7).integers(0, 4, 16_000_000)]
    runs = plain.copy()
    for at in range(0, len(runs) - run, every):
        runs[at:at + run] = np.resize(np.frombuffer(b"CAGGT", np.uint8), run)
    offs = torch.arange(0, len(plain) + 1, 8000, dtype=torch.int64, device="cuda")
    ms = []
    with G.Context(0) as ctx:
        for b in (plain, runs):
            d = torch.from_numpy(b).cuda()
            for _ in range(4):
                ctx.partition_device(d, len(b), offs, offs.numel() - 1, G.params(31, 11, 256))
            ms.append(min(ctx.timings().partition_ms for _ in range(5)
                          if ctx.partition_device(d, len(b), offs, offs.numel() - 1, G.params(31, 11, 256))))
    assert ms[1] < 12 * ms[0], ms
