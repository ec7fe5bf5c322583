"""A call that fails for want of memory no longer reads its page-locked inputs
once it has returned: the caller frees them then."""
import ctypes as C

import numpy as np
import pytest

import gkc_b200 as G
from test_gpu_stream import outputs, pinned

pytestmark = pytest.mark.gpu

GKC_ERR_BUDGET = 5
BYTES = 256 << 20  # some milliseconds of copying


@pytest.mark.parametrize("call", ["superkmers", "pipeline", "partition", "stream"])
def test_inputs_are_read_no_more(call):
    import torch
    letters = np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(1).integers(0, 4, 1 << 20)]
    reads = torch.from_numpy(np.tile(letters, BYTES >> 20)).pin_memory()
    stream = torch.cuda.Stream()
    with G.Context(0, BYTES + (64 << 20)) as ctx:  # the inputs fit, the results do not
        ctx.count_superkmers_host(31, np.full(9, 40, np.uint32), np.zeros(90, np.uint8))  # loads the kernels
        ctx.set_stream(stream.cuda_stream)
        offs = pinned(torch, np.array([0, BYTES], np.uint64))
        prm = G.params(31, 11, 16)
        with pytest.raises(G.GkcError) as e:
            if call == "superkmers":
                lens = torch.full((64,), BYTES // 64 * 4 - 1, dtype=torch.int32).pin_memory()
                ctx._check(ctx._L.gkc_count_superkmers_host(ctx.h, 31, lens.data_ptr(), reads.data_ptr(), 64,
                                                            G.MODE_BATCHED, None), "count")
            elif call == "stream":
                ctx.stream_submit(reads, offs, 1, prm, *outputs(torch, 16, 1), 1)
            else:
                run = ctx._L.gkc_pipeline_host if call == "pipeline" else ctx._L.gkc_partition_host
                mode = (G.MODE_BATCHED,) if call == "pipeline" else ()
                ctx._check(run(ctx.h, C.byref(prm), *mode, reads.data_ptr(), offs.data_ptr(), 1, None), call)
        idle = stream.query()
        assert e.value.status == GKC_ERR_BUDGET
        assert idle, "the inputs are still being copied"
        stream.synchronize()
