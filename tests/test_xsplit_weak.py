"""Weak and sparse 8-bit complex samples through the plain X stage on the tensor cores: spectra of a few units next to
FP16's subnormals.  Against the 64-bit oracle."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth
from oracle import fxoracle as fo

pytestmark = pytest.mark.gpu

# Norm of a product spectrum's error over the spectrum's: the FFTs' rounding (1.6e-7 of each factor, at random:
# 2.3e-7), the split (2^-23 of each factor at most: 1.2e-7 at random), and what the truncating additions leave around
# their mean (2^-23).
TOL = 5e-7


def samples(kind, shape, nchan, rng):
    """int8 [antenna][sample][re, im]"""
    unit = rng.integers(-1, 2, shape, dtype=np.int8)
    if kind == "units":
        return unit
    sparse = unit * (rng.random(shape[:-1]) < 1 / 64)[..., None].astype(np.int8)
    if kind == "sparse":
        return sparse
    if kind == "one":                       # one unit sample per FFT
        out = np.zeros(shape, np.int8)
        at = np.arange(0, shape[1], nchan)
        for a in range(shape[0]):
            out[a, at + rng.integers(0, nchan, len(at)), 0] = 1
        return out
    sparse[0] = rng.integers(-128, 128, shape[1:], dtype=np.int8)   # "mixed": one antenna at full scale
    return sparse


@pytest.mark.parametrize("kind", ["units", "sparse", "one", "mixed"])
@pytest.mark.parametrize("npol,nchan", [(1, 256), (2, 1024), (1, 4096)])
def test_weak_complex(npol, nchan, kind):
    nant, numffts = 10, 64
    assert fx.lib().fxc_debug_xsplit_pays(nant * npol, nchan, 1, numffts, 148)
    job = synth.random_job(nant=nant, npol=npol, nchan=nchan, numffts=numffts, bw=32e6, seed=nchan, cpx=True)
    rng = np.random.default_rng(nchan + npol)
    n = job.data.shape[-1] // (2 * npol)
    x = np.stack([samples(kind, (nant, n, 2), nchan, rng) for _ in range(npol)], axis=2)   # [ant][sample][pol][2]
    job.data[0] = x.reshape(nant, -1).view(np.uint8)
    cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=npol, cpx=True)
    with fx.Correlator(cfg) as c:
        c.process(job.data, job.delays, job.fileoffsets)
        vis, counts = c.visibilities()
    ref, rc = fo.correlate(job.data[0], job.delays, job.fileoffsets, job.bw, job.lo, nchan, npol, numffts=numffts,
                           maxoffset_ffts=numffts, cpx=True)
    np.testing.assert_array_equal(counts, rc)
    assert fo.vis_error(vis[0], ref)[1].max() < TOL
