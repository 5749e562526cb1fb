"""FP8 form: the F stage of a short call takes smaller blocks of FFTs than that of a call that fills the SMs.  Antennas
are scaled each by itself, so the baselines of a few antennas are the same, bit for bit, alone and among many."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cpx", [False, True])
@pytest.mark.parametrize("npol", [1, 2])
@pytest.mark.parametrize("nchan", [512, 1024, 2048, 4096])
@pytest.mark.parametrize("numffts", [37, 128])
def test_block_size(nchan, npol, cpx, numffts):
    few, many = 3, 70
    job = synth.random_job(nant=many, npol=npol, nchan=nchan, numffts=numffts, bw=32e6, seed=nchan + npol, cpx=cpx)
    out = []
    for n in (few, many):
        cfg = fx.make_config(n, nchan, numffts, job.bw, job.lo, npol=npol, xmode=fx.FXC_X_TC_FP8, cpx=cpx)
        with fx.Correlator(cfg) as c:
            c.process(job.data[:, :n], job.delays[:n], job.fileoffsets[:n])
            out.append(c.visibilities())
    bls = lambda n: [(i, j) for i in range(n) for j in range(i + 1, n)] + [(i, i) for i in range(n)]
    at = [bls(many).index(b) for b in bls(few)]
    np.testing.assert_array_equal(out[0][1], out[1][1][at])
    np.testing.assert_array_equal(out[0][0], out[1][0][:, at])
