"""Histogram chunks that are asked for are taken, 65536 among them; zero leaves
them to the input's size, and the tuner compares each size once."""
import numpy as np
import pytest

import gkc_b200 as G
from gkc_b200 import synth

pytestmark = pytest.mark.gpu


def table_bytes(chunk):
    """Device bytes of a run, which hold one row of digits a chunk."""
    import torch
    reads, offs = synth.iid_reads(3, 20_000, 150, 0.0)
    d, o = torch.from_numpy(reads).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        if chunk is not None:
            ctx.tune_set(G.TuneParams(0, chunk, 0, 0))
            assert ctx.tune_get().chunk_kmers == chunk
        ctx.pipeline_device(d, len(reads), o, len(offs) - 1, G.params(31, 11, 1))
        return ctx.device_bytes()


def test_chunks_asked_for():
    rows = {c: table_bytes(c) for c in (None, 0, 16384, 32768, 65536, 131072)}
    assert rows[None] == rows[0] == rows[16384]  # 3 M bases: the smallest
    assert rows[16384] > rows[32768] > rows[65536] > rows[131072]


def test_tuner_times_each_chunk_once():
    import torch
    reads, offs = synth.iid_reads(5, 20_000, 150, 0.0)
    d, o = torch.from_numpy(reads).cuda(), torch.from_numpy(offs.view(np.int64)).cuda()
    with G.Context(0) as ctx:
        rep = ctx.autotune_device(d, len(reads), o, len(offs) - 1, G.params(31, 11, 16), force=True)
        assert rep.defaults.chunk_kmers == 0
        assert rep.candidates == 1 + 1 + 2 + 3  # the default is 16384 here, no candidate of its own
        assert ctx.tune_get().chunk_kmers == rep.chosen.chunk_kmers
    G.lib().gkc_tune_cache_clear()
