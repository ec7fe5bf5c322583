"""The HBM estimate of a job covers what its run takes, from one bin to the
most there can be, and a job whose budget is its estimate runs."""
import numpy as np
import pytest

import gkc_b200 as G
from gkc_b200 import synth

pytestmark = pytest.mark.gpu

BINS = [1, 31, 256, 2048, 2049, 1 << 18, 1 << 20]


@pytest.mark.parametrize("hpc", [False, True])
@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("reads_n", [7, 20_000])
def test_estimate_covers_a_run(reads_n, k, hpc):
    reads, offs = synth.iid_reads(reads_n, reads_n, 151, 0.001)
    for nbins in BINS:
        prm = G.params(k, 11, nbins, hpc)
        with G.Context(0) as ctx:
            ctx.pipeline_host(reads, offs, prm)
            used = ctx.device_bytes()
        assert used <= G.job_hbm_estimate(prm, len(reads), reads_n), nbins


@pytest.mark.parametrize("nbins", BINS)
def test_job_runs_in_its_estimate(nbins):
    reads, offs = synth.iid_reads(2, 3000, 150, 0.001)
    prm = G.params(31, 11, nbins)
    with G.Server(0, hbm_budget=G.job_hbm_estimate(prm, len(reads), 3000), max_running=2) as srv:
        for _ in range(2):
            job = srv.submit(reads, offs, prm)
            assert srv.wait(job).state == G.JOB_DONE
            assert int(np.asarray(srv.result(job)[2]).sum()) > 0
            srv.release(job)
