"""Runs of keys with equal leading bits over several tiles of the kernel that
orders them: each tile has a part of the run, and one key alone, at any place,
may make it a run that has to be sorted.  Position lists against the oracle;
and reads of few letters, whose keys are mostly one run, take no longer than
some times what reads of even letters do."""
import numpy as np
import pytest

import gkc_b200 as G
import oracle_ffi as F

pytestmark = pytest.mark.gpu

BASES = np.frombuffer(b"ACGT", np.uint8)


def kmers(r, n, prefix, k):
    """n k-mers that begin with `prefix` (A.. or C..) and end with A: each is
    its own canonical form."""
    b = BASES[r.integers(0, 4, (n, k))]
    b[:, :len(prefix)] = np.frombuffer(prefix, np.uint8)
    b[:, -1] = 65
    return b


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("shift", [0, 1, 511, 1023])
@pytest.mark.parametrize("length", [512, 513, 1024, 1025, 1536, 2049, 5000])
def test_one_key_of_a_run_differs(length, shift, k):
    import torch
    from test_gpu_windows import subsample
    r = np.random.default_rng(length + shift)
    first, last = kmers(r, shift, b"AC", k), kmers(r, 700, b"CC", k)
    one = kmers(r, 1, b"CAGTCAGTCAGTCAGTCAGT", k)
    with G.Context(0) as ctx:
        for at in sorted({-1, 0, 1, 511, 512, 513, 1023 - shift, 1024 - shift, 2048 - shift, length - 2, length - 1}):
            if at >= length or at < -1:
                continue
            run = np.repeat(one, length, axis=0)
            if at >= 0:
                run[at, k - 3] = 65 if one[0, k - 3] != 65 else 67
            reads = np.concatenate([last, run, first]).reshape(-1)
            offs = (np.arange(len(reads) // k + 1) * k).astype(np.uint64)
            want = F.oracle_subsample(reads, offs, k, 7, 1)
            nd, kw, keys, pos_off, pos = subsample(torch, ctx, reads, offs, k, 7, 1)
            assert np.array_equal(keys[:, 0], want["keys_lo"]), at
            if kw == 2:
                assert np.array_equal(keys[:, 1], want["keys_hi"]), at
            assert np.array_equal(pos_off, want["pos_off"]) and np.array_equal(pos, want["pos"]), at


@pytest.mark.parametrize("k", [31, 63])
def test_time_of_few_letters(k):
    import time
    import torch
    r = np.random.default_rng(k)
    n = 15_000_000
    offs = torch.arange(0, n + 1, 150, dtype=torch.int64, device="cuda")
    ms = []
    with G.Context(0) as ctx:
        for rare in (0.75, 0.015):  # share of bases that are no A
            reads = BASES[(r.random(n) < rare) * r.integers(1, 4, n)]
            d = torch.from_numpy(reads).cuda()
            best = 1e9
            for _ in range(6):
                torch.cuda.synchronize()
                t = time.perf_counter()
                ctx.subsample_positions_device(d, n, offs, offs.numel() - 1, G.params(k, 11, 1), 1)
                best = min(best, time.perf_counter() - t)
            ms.append(1e3 * best)
    assert ms[1] < 5 * ms[0], ms  # passes over all bits for the few, over a half or a quarter of them for the others
