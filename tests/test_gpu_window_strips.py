"""Per-window minimizers and position lists at each number of windows a warp
takes (fewer for small inputs), with reads full of bytes that are no base, and
the superkmers of such reads.  Against the oracle; a small call with many such
bytes takes no longer than a few times one without."""
import time

import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu

# bytes: one side and the other of 148 SMs' tiles of 8 * 448, 480, 224, 96 and 32 windows
SIZES = [700, 148 * 8 * 96 - 1, 148 * 8 * 96, 148 * 8 * 224 - 1, 148 * 8 * 224, 148 * 8 * 448, 148 * 8 * 480 - 1, 148 * 8 * 480 + 5000]


def reads_of(n, bad, seed):
    r = np.random.default_rng(seed)
    b = np.frombuffer(b"ACGT", np.uint8)[r.integers(0, 4, n)].copy()
    b[r.random(n) < bad] = ord("N")
    if bad:
        b[n // 3:n // 3 + 300] = np.frombuffer(b"ACGTN", np.uint8)[r.integers(0, 5, len(b[n // 3:n // 3 + 300]))]
    cuts = np.unique(np.concatenate([[0, n], r.integers(0, n, n // 500 + 1)])).astype(np.uint64)
    return b, cuts


@pytest.mark.parametrize("k,p", [(31, 11), (64, 3), (16, 16), (25, 15)])
@pytest.mark.parametrize("bad", [0.0, 0.002, 0.3])
@pytest.mark.parametrize("n", SIZES)
def test_strips(n, bad, k, p):
    import torch
    reads, offs = reads_of(n, bad, n + k)
    d, o = torch.from_numpy(reads).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    mm = torch.zeros(n, dtype=torch.int32, device="cuda")
    pos, strand = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.int8, device="cuda")
    want = [np.full(n, 0xFFFFFFFF, np.uint32), np.full(n, 255, np.uint8), np.zeros(n, np.int8)]
    for b, e in zip(offs[:-1].astype(int), offs[1:].astype(int)):
        if e - b >= k:
            for w, x in zip(want, F.oracle_minimizers(reads[b:e], k, p, with_pos=True)):
                w[b:b + len(x)] = x
    with G.Context(0) as ctx:
        ctx.minimizers_device(d, n, o, len(offs) - 1, G.params(k, p, 1), mm, pos, strand)
        assert np.array_equal(mm.cpu().numpy().view(np.uint32), want[0])
        assert np.array_equal(pos.cpu().numpy(), want[1]) and np.array_equal(strand.cpu().numpy(), want[2])
        from test_gpu_windows import subsample
        lists = F.oracle_subsample(reads, offs, k, p, 3)
        nd, kw, keys, pos_off, positions = subsample(torch, ctx, reads, offs, k, p, 3)
        assert np.array_equal(keys[:, 0], lists["keys_lo"])
        if kw == 2:
            assert np.array_equal(keys[:, 1], lists["keys_hi"])
        assert np.array_equal(pos_off, lists["pos_off"]) and np.array_equal(positions, lists["pos"])
        if n < 300_000:
            part = F.oracle_partition(reads, offs, k, p, 0, 64)
            v = ctx.partition_device(d, n, o, len(offs) - 1, G.params(k, p, 64))
            bin_off, lens, boff, packed, _ = ctx.partition_copy_out(v)
            bins = np.repeat(np.arange(64, dtype=np.uint32), np.diff(bin_off).astype(np.int64))
            assert F.Skms(bins, lens, boff, packed).multisets(64) == part.multisets(64)


def test_time_of_a_small_call():
    import torch
    n = 15_000
    o = torch.arange(0, n + 1, 150, dtype=torch.int64, device="cuda")
    mm = torch.zeros(n, dtype=torch.int32, device="cuda")
    us = []
    with G.Context(0) as ctx:
        for bad in (0.0, 0.3):
            r = np.random.default_rng(1)
            b = np.frombuffer(b"ACGT", np.uint8)[r.integers(0, 4, n)].copy()
            b[r.random(n) < bad] = ord("N")
            d, best = torch.from_numpy(b).cuda(), 1e9
            for _ in range(30):
                torch.cuda.synchronize()
                t = time.perf_counter()
                ctx.minimizers_device(d, n, o, 100, G.params(31, 11, 1), mm, None, None)
                best = min(best, time.perf_counter() - t)
            us.append(1e6 * best)
    assert us[1] < 3 * us[0], us
