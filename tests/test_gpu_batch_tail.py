"""A batch job on the FP32 units whose last chunk is so short that it fills one time segment: its partial sums are
added like any other chunk's.  Bit-identical to the job alone."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nant,nchan,numffts", [(4, 128, 530), (6, 256, 1025), (12, 128, 576)])
def test_short_last_chunk(nant, nchan, numffts):
    job = synth.random_job(nant=nant, npol=1, nchan=nchan, numffts=numffts, bw=32e6, seed=nant, nsubband=1)
    cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=1, chunk_ffts=512)
    with fx.Batch([cfg, cfg]) as b:
        for j in range(2):
            b.upload(j, job.data)
            b.set_model(j, job.delays, job.fileoffsets)
        b.process()
        got = b.visibilities(0)
    with fx.Correlator(cfg) as c:
        c.process(job.data, job.delays, job.fileoffsets)
        want = c.visibilities()
    np.testing.assert_array_equal(got[1], want[1])
    np.testing.assert_array_equal(got[0], want[0])
