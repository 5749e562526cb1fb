"""Calls of few FFTs in the plain form: the error of the X stage alone, against 64-bit sums of the library's own FP32
spectra, whatever the length of the subintegration the context was made for."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

U = 2.0 ** -24   # unit roundoff of FP32


def test_rule():
    pays = fx.lib().fxc_debug_xsplit_pays
    assert [pays(32, 2048, 2, n, 148) for n in (1, 31, 32, 5000)] == [0, 0, 1, 1]
    assert [pays(8, 128, 1, n, 148) for n in (1, 31, 32, 128, 129)] == [0, 0, 1, 1, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("nant,npol,nchan,numffts", [(4, 2, 128, 100), (12, 1, 1024, 300), (20, 2, 512, 64)])
@pytest.mark.parametrize("nfft", [1, 2, 4, 8, 31, 32, 64])
def test_short_call(nant, npol, nchan, numffts, nfft):
    assert fx.lib().fxc_debug_xsplit_pays(nant * npol, nchan, 1, numffts, 148)
    job = synth.random_job(nant=nant, npol=npol, nchan=nchan, numffts=numffts, bw=32e6, seed=nfft)
    job.fileoffsets[:] = job.delays[:, 2]        # every FFT of every antenna inside its samples
    cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=npol)
    with fx.Correlator(cfg) as c:
        c.process(job.data, job.delays, job.fileoffsets, 0, nfft)
        vis, counts = c.visibilities()
        s = c.spectra(job.data, job.delays, job.fileoffsets, 0, nfft)[0].astype(np.complex128)
    g = np.einsum("itc,jtc->ijc", s, s.conj())
    bls = [(i, j) for i in range(nant) for j in range(i + 1, nant)] + [(i, i) for i in range(nant)]
    want = np.array([[g[i * npol + l, j * npol + m] for l in range(npol) for m in range(npol)] for i, j in bls])
    # FP32 sums of nfft products: a unit roundoff of the products and half of one for each addition, at random
    assert np.linalg.norm(vis[0] - want) < U * (1 + 0.5 * nfft ** 0.5) * np.linalg.norm(want)


@pytest.mark.gpu
def test_short_last_window():
    """Host rows go through the device in windows: a short last one takes the path of the whole call, as a short last
    chunk of device rows does."""
    job = synth.random_job(nant=12, npol=1, nchan=1024, numffts=70, bw=32e6, seed=3)
    cfg = fx.make_config(12, 1024, 70, job.bw, job.lo, npol=1, chunk_ffts=64)
    with fx.Correlator(cfg) as c:
        c.process(job.data, job.delays, job.fileoffsets)
        host = c.visibilities()
        c.reset()
        c.upload(job.data)
        ptr, pitch = c.device_input()
        c.process_device(ptr, pitch, job.delays, job.fileoffsets)
        device = c.visibilities()
    np.testing.assert_array_equal(host[1], device[1])
    np.testing.assert_array_equal(host[0], device[0])
