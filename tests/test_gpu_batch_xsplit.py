"""Plain jobs on the tensor cores in a batch: one X launch per group of jobs, and every job's result as alone, bit for
bit, whatever else is in its launch."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

pytestmark = pytest.mark.gpu


def make(sizes):
    """sizes: antennas, polarisations, channels, subbands, FFTs, FFTs per chunk"""
    jobs = [synth.random_job(nant=a, npol=p, nchan=c, numffts=n, bw=32e6, seed=31 * k + a, nsubband=s)
            for k, (a, p, c, s, n, _) in enumerate(sizes)]
    cfgs = [fx.make_config(a, c, n, j.bw, j.lo, npol=p, nsubband=s, sb_spacing=j.bw, chunk_ffts=t)
            for (a, p, c, s, n, t), j in zip(sizes, jobs)]
    for a, p, c, s, n, _ in sizes:
        assert fx.lib().fxc_debug_xsplit_pays(a * p, c, s, n, 148)
    batch = fx.Batch(cfgs)
    for k, j in enumerate(jobs):
        batch.upload(k, j.data)
        batch.set_model(k, j.delays, j.fileoffsets)
    return jobs, cfgs, batch


def test_one_launch():
    sizes = [(4, 1, 128, 1, 100, 0)] * 16
    _, _, batch = make(sizes)
    with batch:
        assert batch.launch_count() == 2 * 16 + 2   # delay table and counts per job, F, X


@pytest.mark.parametrize("sizes", [
    # one group of each kind: signal counts at the edges of its block, long and short items, one or several chunks
    [(2, 1, 128, 1, 64, 0), (7, 1, 256, 1, 100, 0), (8, 1, 128, 1, 128, 64), (1 + 4, 1, 512, 2, 33, 0)],
    [(4, 2, 128, 1, 100, 0), (3, 2, 256, 1, 128, 0), (2, 2, 512, 1, 70, 64)],
    [(9, 1, 1024, 1, 2200, 0), (16, 1, 256, 1, 64, 0), (10, 1, 2048, 1, 300, 128), (12, 1, 128, 3, 90, 0)],
    [(33, 1, 128, 1, 65, 0), (40, 1, 512, 1, 200, 64), (34, 1, 1024, 1, 128, 0)],
    [(32, 2, 256, 1, 64, 0), (29, 2, 1024, 1, 300, 0), (32, 2, 128, 1, 40, 0)],
    # several groups, among other jobs
    [(24, 1, 1024, 1, 150, 0), (31, 1, 1024, 1, 64, 0), (24, 1, 256, 1, 32, 0), (56, 1, 512, 1, 90, 0), (5, 1, 128, 1, 128, 0),
     (64, 1, 256, 2, 129, 64), (6, 1, 128, 1, 50, 0)],
])
def test_as_alone(sizes):
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
