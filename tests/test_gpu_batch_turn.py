"""FP16 jobs of more than 64 signals in a batch: their F stages share a launch and so do their corner turns, and every
job's result is as alone, bit for bit."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

pytestmark = pytest.mark.gpu


def make(sizes):
    """sizes: antennas, polarisations, channels, subbands, FFTs, FFTs per chunk, X form"""
    jobs = [synth.random_job(nant=a, npol=p, nchan=c, numffts=n, bw=32e6, seed=17 * k + a, nsubband=s)
            for k, (a, p, c, s, n, _, _) in enumerate(sizes)]
    cfgs = [fx.make_config(a, c, n, j.bw, j.lo, npol=p, nsubband=s, sb_spacing=j.bw, chunk_ffts=t, xmode=x)
            for (a, p, c, s, n, t, x), j in zip(sizes, jobs)]
    batch = fx.Batch(cfgs)
    for k, j in enumerate(jobs):
        batch.upload(k, j.data)
        batch.set_model(k, j.delays, j.fileoffsets)
    return jobs, cfgs, batch


def test_launches():
    _, _, batch = make([(72, 1, 128, 1, 64, 0, fx.FXC_X_TC_FP16)] * 8)
    with batch:
        assert batch.launch_count() == 2 * 8 + 1 + 1 + 8   # delay table and counts per job, F, turn, X per job


FP16, PLAIN = fx.FXC_X_TC_FP16, fx.FXC_X_PLAIN_FP32


@pytest.mark.parametrize("budget,sizes", [
    (None, [(65, 1, 128, 1, 64, 0, FP16), (100, 1, 128, 2, 100, 64, FP16), (40, 2, 256, 1, 70, 0, FP16),
            (8, 1, 128, 1, 130, 64, FP16), (70, 1, 128, 1, 128, 0, FP16), (12, 1, 128, 1, 90, 0, PLAIN)]),
    # 8 MiB of spectra: chunks of several parts beside chunks of one
    ("8", [(72, 1, 128, 1, 300, 0, FP16), (66, 1, 128, 1, 64, 0, FP16), (33, 2, 128, 2, 200, 64, FP16)]),
])
def test_as_alone(budget, sizes, monkeypatch):
    if budget:
        monkeypatch.setenv("FXC_SPECTRA_BUDGET_MB", budget)
    jobs, cfgs, batch = make(sizes)
    with batch:
        got = []
        for _ in range(3):   # eager, captured, replayed
            batch.reset()
            batch.process()
            got.append([batch.visibilities(k) for k in range(len(jobs))])
    for k, j in enumerate(jobs):
        with fx.Correlator(cfgs[k]) as c:
            c.upload(j.data)
            c.process_device(*c.device_input(), j.delays, j.fileoffsets)
            want, wc = c.visibilities()
        for g in got:
            np.testing.assert_array_equal(g[k][1], wc)
            np.testing.assert_array_equal(g[k][0], want)
