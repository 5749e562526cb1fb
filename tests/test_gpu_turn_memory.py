"""The corner turn's buffer of the FP16 form takes what the context's other buffers leave: a context that fits with a
smaller one is made, and its results are the same."""
import numpy as np
import pytest
import torch

import difx_tests_b200 as fx
from difx_tests_b200 import synth

pytestmark = pytest.mark.gpu


def test_little_memory(monkeypatch):
    monkeypatch.setenv("FXC_SPECTRA_BUDGET_MB", "4096")
    nant, nchan, numffts = 128, 4096, 900
    # with room enough the 960 slots are turned 256 at a time; 64 at a time need a quarter of that
    turn = 256 * nant * nchan * 4
    job = synth.random_job(nant=nant, npol=1, nchan=nchan, numffts=numffts, bw=32e6, seed=1)
    cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=1, xmode=fx.FXC_X_TC_FP16)

    def run():
        with fx.Correlator(cfg) as c:
            used = torch.cuda.mem_get_info()[0]
            c.upload(job.data)
            c.process_device(*c.device_input(), job.delays, job.fileoffsets)
            return used, c.visibilities()[0]

    run()                                        # kernels are loaded
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    left, want = run()
    need = free - left
    filler = torch.empty(free - (need - turn // 2), dtype=torch.uint8, device="cuda")
    try:
        got = run()[1]
    finally:
        del filler
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(got, want)
