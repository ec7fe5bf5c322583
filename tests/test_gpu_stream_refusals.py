"""What the synchronous pipeline refuses, the streamed form refuses with the
same status, at the call's wait: a superkmer of 2^24 bases or more."""
import numpy as np
import pytest

import gkc_b200 as G
from gkc_b200 import synth
from test_gpu_stream import check, expect, outputs, pinned

pytestmark = pytest.mark.gpu

GKC_ERR_INVALID_ARG = 1
K, P, NB = 31, 11, 16


def test_read_too_long():
    import torch
    run = np.resize(np.frombuffer(b"CAGGT", np.uint8), (1 << 24) + 200)
    offs = np.array([0, len(run)], np.uint64)
    other = synth.iid_reads(1, 300, 150, 0.002)
    prm = G.params(K, P, NB)
    with G.Context(0) as ctx:
        with pytest.raises(G.GkcError) as e:
            ctx.pipeline_host(run, offs, prm)
        assert e.value.status == GKC_ERR_INVALID_ARG
        out = outputs(torch, NB, len(run))
        (r, o), (r2, o2) = ((pinned(torch, x), pinned(torch, y)) for x, y in ((run, offs), other))
        for _ in range(3):  # launch by launch, captured, replayed
            ticket = ctx.stream_submit(r, o, 1, prm, *out, len(run))
            between = ctx.stream_submit(r2, o2, 300, prm, *out, len(run))
            with pytest.raises(G.GkcError) as e:
                ctx.stream_wait(ticket)
            assert e.value.status == GKC_ERR_INVALID_ARG
            nd, _ = ctx.stream_wait(between)
            check(out, expect(*other, K, P, NB), nd)
