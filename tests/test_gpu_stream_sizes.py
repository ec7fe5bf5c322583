"""Streaming calls whose sizes change from call to call run launch by launch;
two calls of one size in a row on a slot are captured, the third replays.
Reads with more superkmers than their bases suggest outgrow the first
workspaces and are run again, whichever call finds that out."""
import numpy as np
import pytest

import gkc_b200 as G
from gkc_b200 import synth
from test_gpu_stream import check, expect, outputs, pinned

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as T
    return T


K, P, NB = 15, 5, 16


def dense(n_reads, length):
    """0.59 superkmers a base at k 15, p 5: the first workspaces hold 0.25 and a few more."""
    unit = np.frombuffer(b"ACTGCTGGGGGCGCGGGGCCCCCAA", np.uint8)
    reads = np.resize(unit, n_reads * length).astype(np.uint8)
    return reads, (np.arange(n_reads + 1) * length).astype(np.uint64)


@pytest.mark.parametrize("ahead", [1, 2, 3])
def test_sizes_and_densities_that_change(torch, ahead):
    batches = [synth.iid_reads(1, 300, 150, 0.002), dense(150, 700), synth.iid_reads(2, 301, 150, 0.002),
               dense(150, 700), dense(151, 700), dense(150, 700), synth.iid_reads(3, 700, 150, 0.0),
               dense(150, 700), dense(200, 800), synth.iid_reads(4, 1, 150, 0.0)]
    want = [expect(*b, K, P, NB) for b in batches]
    with G.Context(0) as ctx:
        prm = G.params(K, P, NB)
        ins = [(pinned(torch, r), pinned(torch, o)) for r, o in batches]
        cap = max(int(o[-1]) for _, o in batches)
        outs = [outputs(torch, NB, cap) for _ in range(4)]
        tickets = []

        def wait(i):
            nd, _ = ctx.stream_wait(tickets[i])
            check(outs[i % 4], want[i], nd)

        for i, (r, o) in enumerate(ins):
            if i >= ahead:
                wait(i - ahead)
            tickets.append(ctx.stream_submit(r, o, len(batches[i][1]) - 1, prm, *outs[i % 4], cap))
        for i in range(len(ins) - ahead, len(ins)):
            wait(i)


def test_device_calls_first_second_third(torch):
    """Direct, captured, replayed; another input in between starts over."""
    a, b = synth.iid_reads(5, 400, 150, 0.002), dense(150, 700)
    with G.Context(0) as ctx:
        prm = G.params(K, P, NB)
        dev = [(torch.from_numpy(r.copy()).cuda(), torch.from_numpy(o.view(np.int64).copy()).cuda()) for r, o in (a, b)]
        want = [expect(*x, K, P, NB) for x in (a, b)]
        for i, replayed in ((0, 0), (0, 1), (0, 1), (1, 0), (1, 1), (1, 1), (0, 0)):
            r, o = dev[i]
            _, cv = ctx.pipeline_device(r, r.numel(), o, o.numel() - 1, prm)
            assert ctx.timings().graph_replayed == replayed
            bo, keys, counts = ctx.count_copy_out(cv)
            assert np.array_equal(np.asarray(bo), want[i]["bin_off"])
            assert np.array_equal(np.asarray(keys).reshape(-1), want[i]["keys_lo"])
            assert np.array_equal(np.asarray(counts), want[i]["counts"])
