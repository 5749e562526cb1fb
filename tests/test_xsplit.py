"""The plain X stage on the tensor cores (difx_tests_b200/csrc/fx_xsplit.cu).  On the CPU: the cast's index
arithmetic restated from the kernel (reads inside a stage, every 16-byte chunk of the tiles' rows stored once and
with the FFTs both operands share, bank passes), the sums' way out (every pair and channel once), the rule that
selects the stage.  On the GPU: sizes at its edges against the 64-bit oracle, and a batch against single jobs."""
import itertools

import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth
from oracle import fxoracle as fo

BT, NQ, NV, NCW, NSM = 16, 2, 4, 8, 148

SIZES = [(n, p) for n in (1, 2, 5, 8, 9, 31, 32, 33, 48, 63, 64) for p in (1, 2) if n % p == 0]


@pytest.mark.parametrize("nsig,npol", SIZES)
@pytest.mark.parametrize("h", range(NQ))
def test_cast(nsig, npol, h):
    cb = 8 if nsig <= 32 else 4
    cpt, swp, ng, upw = cb // NV, 8 // cb, 4, 32 // (4 * cb)
    stage = nsig * BT * cb * 8
    reads, stores = {}, {}
    for warp, lane in itertools.product(range(NCW), range(32)):
        c, tg = lane % cb, lane // cb % ng
        for n, u in enumerate(range(warp * upw + lane // (ng * cb), nsig // npol, NCW * upw)):
            if npol == 2:
                at = [(u * BT + ng * i) * cb + tg * cb + c for i in range(4)]
                sets = [(2 * u + p, [(tg + ng * i, p) for i in range(4)]) for p in range(2)]
                ffts = [[t for t, _ in s[1]] for s in sets]
            else:
                at = [(u * (BT // 2) + ng * i) * cb + tg * cb + c for i in range(2)]
                sets = [(u, None)]
                ffts = [[2 * tg, 2 * tg + 1, 2 * (tg + ng), 2 * (tg + ng) + 1]]
            for i, a in enumerate(at):
                reads.setdefault((warp, n, i), []).append((lane, 16 * a))
            for (s, _), ts in zip(sets, ffts):
                r = s ^ (swp * c)
                row = c % cpt * 32 + r
                stores.setdefault((warp, n, s if npol == 1 else s % 2), []).append(
                    (lane, c // cpt, row, (ng * h + tg) ^ (r & 7), tuple(ts), s, c))
    seen = {}
    for group in stores.values():
        for q in range(4):   # a quarter warp's 16-byte stores: all banks once
            slots = [(t * 128 * 128 + row * 128 + (k << 4)) // 16 % 8 for lane, t, row, k, *_ in group if lane // 8 == q]
            assert len(set(slots)) == len(slots)
        for lane, t, row, k, ts, s, c in group:
            assert row < 64 and (t, row, k) not in seen
            seen[t, row, k] = (ts, s, c)
    for group in reads.values():
        assert all(0 <= a and a + 16 <= stage for _, a in group)
    assert len(seen) == nsig * cb * ng
    for (t, row, k), (ts, s, c) in seen.items():
        # the FFTs of a logical chunk are those of every row: the contraction pairs equal FFTs
        assert c // cpt == t and ts == seen[t, (s ^ (swp * c)) + c % cpt * 32, k][0]
        logical = k ^ (row & 7)
        assert h * ng <= logical < (h + 1) * ng
        tg = logical - h * ng
        want = tuple(tg + ng * i for i in range(4)) if npol == 2 else (2 * tg, 2 * tg + 1, 2 * tg + 8, 2 * tg + 9)
        assert ts == want
    for s in range(nsig):   # all FFTs of the stage
        for c in range(cb):
            assert sorted(t for ts, s1, c1 in seen.values() if (s1, c1) == (s, c) for t in ts) == list(range(BT))


@pytest.mark.parametrize("nsig", sorted({n for n, _ in SIZES}))
def test_sums_out(nsig):
    cb = 8 if nsig <= 32 else 4
    swp, out = 8 // cb, {}
    rng = np.random.default_rng(nsig)
    x = rng.standard_normal((cb, nsig)) + 1j * rng.standard_normal((cb, nsig))
    for t in range(2):
        for ee in range(1 if cb == 8 else 2):
            v = np.full((128, 65), np.nan)
            for e in range(2):
                if cb == 4 and e != ee:
                    continue
                tile = e + 2 * t
                rows = np.zeros((64 * (cb // 4), 1), complex)[:64]
                for c in range(cb // 4 * tile, cb // 4 * (tile + 1)):
                    for s in range(nsig):
                        rows[(c % (cb // 4)) * 32 + (s ^ (swp * c))] = x[c, s]
                hh = np.concatenate([rows, rows.imag - 1j * rows.real])   # (Re, Im) and (Im, -Re)
                d = (hh.real @ rows.real.T) + (hh.imag @ rows.imag.T)
                for q in range(4):
                    if cb == 8:
                        v[32 * q:32 * q + 32, 32 * e:32 * e + 32] = d[32 * q:32 * q + 32, 32 * (q & 1):32 * (q & 1) + 32]
                    else:
                        v[32 * q:32 * q + 32, :64] = d[32 * q:32 * q + 32]
            for w, lane in itertools.product(range(8), range(32)):
                if cb == 8:
                    cells = [(i, lane, 2 * (w & 1) + y, 32 * y, 32 * (w & 1)) for i in range(w >> 1, nsig, 4) for y in range(2)]
                else:
                    cells = [(i, j, ee + 2 * t, 0, 0) for i in range(w, nsig, 8) for j in range((i & ~31) + lane, nsig, 32)]
                for i, j, c, r0, c0 in cells:
                    if i <= j < nsig:
                        c = 4 * t + c if cb == 8 else c
                        k = swp * c
                        re, im = v[r0:, c0:], v[r0 + 64:, c0:]
                        assert (i, j, c) not in out
                        out[i, j, c] = 0.5 * (re[i ^ k, j ^ k] + re[j ^ k, i ^ k]) + 0.5j * (im[i ^ k, j ^ k] - im[j ^ k, i ^ k])
    assert len(out) == cb * nsig * (nsig + 1) // 2
    for (i, j, c), got in out.items():
        assert abs(got - x[c, i] * np.conj(x[c, j])) < 1e-12


@pytest.mark.parametrize("nsig,nchan,nsb,numffts,want", [
    (8, 128, 1, 128, 1), (8, 128, 1, 129, 0), (8, 2048, 1, 128, 0), (9, 2048, 1, 128, 1),   # short calls
    (9, 1024, 1, 5000, 1), (9, 512, 1, 5000, 0), (8, 4096, 8, 5000, 0), (32, 1024, 1, 129, 1), (32, 256, 3, 129, 0),
    (33, 512, 1, 5000, 1), (33, 256, 1, 5000, 0), (64, 4096, 8, 31250, 1), (65, 4096, 8, 64, 0)])
def test_rule(nsig, nchan, nsb, numffts, want):
    assert fx.lib().fxc_debug_xsplit_pays(nsig, nchan, nsb, numffts, NSM) == want


# ------------------------------------------------------------------------------ GPU
# Largest error of a product's spectrum over its largest value: the FFTs' rounding (up to 1e-6 of a spectrum), 2^-22
# of the split, 8 truncations of at most 2^-23 in 32 FFTs (their mean is put back), and the roundings of up to 64
# additions to a running sum (2^-24 each, at random: 8).
VIS_TOL = 2e-6

GPU_CASES = [  # nant, npol, nchan, subbands, FFTs, complex, FFTs per chunk
    (2, 1, 128, 1, 64, False, 0), (3, 1, 256, 2, 100, False, 0), (4, 2, 128, 1, 127, False, 64),
    (32, 1, 128, 1, 65, False, 0), (33, 1, 128, 1, 70, False, 0), (31, 2, 128, 1, 64, False, 0),
    (9, 1, 1024, 1, 2113, False, 0),     # two segments
    (9, 1, 4096, 1, 130, False, 64),     # items drawn from the counter; three chunks, the last of 2 FFTs
    (16, 2, 1024, 1, 200, False, 128), (17, 2, 256, 2, 200, False, 0), (64, 1, 512, 2, 160, False, 0),
    (24, 2, 512, 1, 200, True, 0), (10, 1, 1024, 1, 150, True, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("nant,npol,nchan,nsb,numffts,cpx,chunk", GPU_CASES)
def test_against_oracle(nant, npol, nchan, nsb, numffts, cpx, chunk):
    assert fx.lib().fxc_debug_xsplit_pays(nant * npol, nchan, nsb, numffts, NSM)
    job = synth.random_job(nant=nant, npol=npol, nchan=nchan, numffts=numffts, bw=32e6, seed=nant + nchan, nsubband=nsb,
                           cpx=cpx)
    cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=npol, nsubband=nsb, sb_spacing=job.bw, cpx=cpx,
                         chunk_ffts=chunk)
    with fx.Correlator(cfg) as c:
        c.process(job.data, job.delays, job.fileoffsets)
        vis, counts = c.visibilities()
        c.reset()
        c.process(job.data, job.delays, job.fileoffsets)
        np.testing.assert_array_equal(c.visibilities()[0], vis)
    for sb in range(nsb):
        ref, rc = fo.correlate(job.data[sb], job.delays, job.fileoffsets, job.bw, float(job.sb_lo[sb]), nchan, npol,
                               numffts=numffts, maxoffset_ffts=numffts, cpx=cpx)
        np.testing.assert_array_equal(counts, rc)
        assert fo.vis_error(vis[sb], ref)[0].max() < VIS_TOL


@pytest.mark.gpu
def test_batch_is_single():
    sizes = [(12, 1, 1024, 1, 300), (5, 1, 512, 2, 300), (40, 1, 512, 1, 100), (8, 2, 1024, 1, 64)]
    jobs = [synth.random_job(nant=a, npol=p, nchan=c, numffts=n, bw=32e6, seed=a, nsubband=s) for a, p, c, s, n in sizes]
    cfgs = [fx.make_config(a, c, n, j.bw, j.lo, npol=p, nsubband=s, sb_spacing=j.bw) for (a, p, c, s, n), j in zip(sizes, jobs)]
    batch = fx.Batch(cfgs)
    for k, j in enumerate(jobs):
        batch.upload(k, j.data)
        batch.set_model(k, j.delays, j.fileoffsets)
    batch.process()
    for k, j in enumerate(jobs):
        got, counts = batch.visibilities(k)
        with fx.Correlator(cfgs[k]) as c:
            c.process(j.data, j.delays, j.fileoffsets)
            want, wc = c.visibilities()
        np.testing.assert_array_equal(counts, wc)
        np.testing.assert_array_equal(got, want)
