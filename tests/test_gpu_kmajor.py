"""The corner turn of the FFT F stage's FP16 spectra (k_kmajor): a chunk turned in several parts, with a
ragged last part, against the whole chunk at once.  Same FP16 values, same MMAs: bit-identical visibilities."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nant,npol,nchan,nsb,numffts,xmode", [
    (70, 1, 256, 1, 300, fx.FXC_X_TC_FP16), (35, 2, 128, 3, 200, fx.FXC_X_TC_FP16),
    (5, 2, 256, 2, 300, fx.FXC_X_TC_FP8), (66, 1, 4096, 1, 130, fx.FXC_X_TC_FP16)])
def test_turn_in_parts(nant, npol, nchan, nsb, numffts, xmode, monkeypatch):
    job = synth.random_job(nant=nant, npol=npol, nchan=nchan, numffts=numffts, bw=32e6, seed=nant + nchan, nsubband=nsb)
    out = {}
    for parts in (False, True):
        if parts:   # an eighth of the budget holds 64 FFT slots before the turn; the chunk is given
            monkeypatch.setenv("FXC_SPECTRA_BUDGET_MB", str(max(1, 8 * 64 * nant * npol * nchan * nsb * 4 >> 20)))
        else:
            monkeypatch.delenv("FXC_SPECTRA_BUDGET_MB", raising=False)
        cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=npol, nsubband=nsb, xmode=xmode, chunk_ffts=256)
        with fx.Correlator(cfg) as c:
            c.process(job.data, job.delays, job.fileoffsets)
            out[parts] = c.visibilities()
    np.testing.assert_array_equal(out[False][1], out[True][1])
    np.testing.assert_array_equal(out[False][0], out[True][0])
