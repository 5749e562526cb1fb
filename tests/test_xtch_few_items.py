"""FP16 tensor-core X stage, up to 32 signals and few channels: work items of 4 channels with 64-row tiles
(difx_tests_b200/csrc/fx_xtch.cu).  On the CPU the tiles' place in shared memory; on the GPU the same visibilities, bit
for bit, as from K-major spectra."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

TILES = 64 * 1024


@pytest.mark.parametrize("nsig", [1, 2, 31, 32])
def test_tiles(nsig):
    tile = 64 * 128
    words = set()
    for ch in range(4):
        for s in range(nsig):
            for part in range(2):
                r = 2 * s + part
                for k in range(8):
                    for w in range(4):
                        words.add(ch * tile + r * 128 + ((k ^ (r & 7)) << 4) + 4 * w)
    assert len(words) == 4 * nsig * 2 * 32 and max(words) + 4 <= 4 * tile
    assert 3 * tile + 128 * 128 <= TILES   # the last tile's operand is 128 rows long


@pytest.mark.gpu
@pytest.mark.parametrize("nant,npol,nchan,numffts,chunk", [
    (2, 1, 128, 64, 0), (3, 1, 512, 200, 64), (16, 2, 512, 130, 0), (31, 1, 256, 100, 0), (32, 1, 128, 1030, 0),
    (32, 1, 1024, 70, 0)])   # (the last has items for two rounds: 8 channels each)
def test_as_kmajor(nant, npol, nchan, numffts, chunk, monkeypatch):
    job = synth.random_job(nant=nant, npol=npol, nchan=nchan, numffts=numffts, bw=32e6, seed=nant + nchan)
    cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=npol, xmode=fx.FXC_X_TC_FP16, chunk_ffts=chunk)
    out = []
    for spectra in (None, "f16"):
        if spectra:
            monkeypatch.setenv("FXC_TC_SPECTRA", spectra)
        with fx.Correlator(cfg) as c:
            c.upload(job.data)
            c.process_device(*c.device_input(), job.delays, job.fileoffsets)
            out.append(c.visibilities())
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][0], out[1][0])
