"""The plan cache under the plain form on the tensor cores: a batch reads the entry a context of the same form reads,
and an autotuner writes no plan it did not time over one of the file."""
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth

pytestmark = pytest.mark.gpu


def config(job, xmode=fx.FXC_X_PLAIN_FP32):
    return fx.make_config(job.nant, job.nchan, job.numffts, job.bw, job.lo, npol=job.npol, xmode=xmode)


@pytest.fixture
def cache(tmp_path, monkeypatch):
    path = tmp_path / "plans.txt"
    path.write_text("F 1024 1 8\nH 1024 1 32\nX 2 1\n")
    monkeypatch.setenv("FXC_PLAN_CACHE", str(path))
    return path


@pytest.mark.parametrize("nant,xmode,want", [
    (12, fx.FXC_X_PLAIN_FP32, 8), (3, fx.FXC_X_PLAIN_FP32, 8), (12, fx.FXC_X_TC_FP16, 32), (70, fx.FXC_X_TC_FP16, 32)])
def test_batch_reads_the_forms_entry(cache, nant, xmode, want):
    job = synth.random_job(nant=nant, npol=1, nchan=512, numffts=100, bw=32e6, seed=1)
    with fx.Correlator(config(job, xmode)) as c, fx.Batch([config(job, xmode)] * 2) as b:
        assert c.plan()[0] == b.plan(0)[0] == want


@pytest.mark.parametrize("xmode", [fx.FXC_X_PLAIN_FP32, fx.FXC_X_TC_FP16])
def test_untimed_plans_stay(cache, xmode):
    job = synth.random_job(nant=12, npol=1, nchan=512, numffts=100, bw=32e6, seed=1)
    before = cache.read_text()
    with fx.Correlator(config(job, xmode)) as c:
        c.set_plan(16, 0)
        c.upload(job.data)
        c.process_device(*c.device_input(), job.delays, job.fileoffsets)
        c.autotune(reps=1)
    with fx.Batch([config(job, xmode)] * 2) as b:
        for k in range(2):
            b.upload(k, job.data)
            b.set_model(k, job.delays, job.fileoffsets)
        b.process()
        b.autotune(reps=1)
    assert cache.read_text() == before
