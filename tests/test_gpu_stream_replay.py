"""Streamed calls of one size whose reads differ in superkmers: a replay that
outgrows the workspaces of the call it was captured from is run again, like a
first call of its size."""
import pytest

import gkc_b200 as G
from gkc_b200 import synth
from test_gpu_stream import check, expect, outputs, pinned
from test_gpu_stream_sizes import K, NB, P, dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ahead", [1, 2, 3])
def test_denser_reads_of_one_size(ahead):
    import torch
    kinds = "sssssdsddssdddds"  # sparse, dense: captured sparse on both slots, then both kinds replayed
    batches = [synth.iid_reads(i, 300, 150, 0.002) if c == "s" else dense(300, 150) for i, c in enumerate(kinds)]
    want = [expect(*b, K, P, NB) for b in batches]
    with G.Context(0) as ctx:
        prm = G.params(K, P, NB)
        ins = [(pinned(torch, r), pinned(torch, o)) for r, o in batches]
        outs = [outputs(torch, NB, 300 * 150) for _ in range(4)]
        tickets = []

        def wait(i):
            nd, _ = ctx.stream_wait(tickets[i])
            check(outs[i % 4], want[i], nd)

        for i, (r, o) in enumerate(ins):
            if i >= ahead:
                wait(i - ahead)
            tickets.append(ctx.stream_submit(r, o, 300, prm, *outs[i % 4], 300 * 150))
        for i in range(len(ins) - ahead, len(ins)):
            wait(i)
