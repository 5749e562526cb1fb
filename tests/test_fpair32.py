"""The F stage's plan with one exchange (difx_tests_b200/csrc/fx_fpair.cuh, 1024 and 2048 real points).  On the CPU:
its factorisation and index maps restated in float64, against the rotated DFT, and the words that the sample
expansion reads.  On the GPU: both lengths, odd FFT counts and single pairs, against the 64-bit oracle."""
import numpy as np
import pytest

import difx_tests_b200 as fx
from difx_tests_b200 import synth
from oracle import fxoracle as fo


def bitrev(v, bits):
    return int(format(v, f"0{bits}b")[::-1], 2)


def butterfly32(v, w, q0, lo):
    for q in range(q0, 5):
        half = 32 >> (q + 1)
        for kp in range(1 << q):
            base = bitrev(kp, q) * 2 * half if q else 0
            ref = kp if q == 0 or kp < 1 << (q - 1) else kp - (1 << (q - 1))
            wd = w(q, ref) * (1 if ref == kp else -1j)
            for h in range(half):
                a, b = v[base + h], v[base + half + h]
                s = a + wd * b
                v[base + h], v[base + half + h] = s, (np.nan if lo and q == 4 else s - 2 * a)


@pytest.mark.parametrize("F", [1024, 2048])
def test_one_exchange_is_the_dft(F):
    H0, NT, logf = F // 1024, F // 32, int(np.log2(F))
    G = NT // H0
    rng = np.random.default_rng(F)
    x = rng.standard_normal(F)
    phase = rng.uniform(-0.4, 0.4, logf)                       # of the bits of n, most significant first
    rho = np.exp(-2j * np.pi * phase)
    n = np.arange(F)
    rot = np.exp(-2j * np.pi * sum(phase[s] * (n >> (logf - 1 - s) & 1) for s in range(logf)))
    buf = np.full(F + F // 32, np.nan, complex)
    for t in range(NT):
        h, tp = t // G, t % G
        if H0 == 2:
            r0 = -rho[0] if h else rho[0]
            v = [x[r * G + tp] + r0 * x[r * G + tp + F // 2] for r in range(32)]
        else:
            v = [0j] * 32
            for r in range(16):
                a, b = x[r * G + tp], x[(r + 16) * G + tp]
                v[r], v[r + 16] = a + rho[0] * b, rho[0] * b - a
        butterfly32(v, lambda q, k: rho[H0 - 1 + q] * np.exp(-2j * np.pi * (h + H0 * k) / (H0 << (q + 1))), 2 - H0, False)
        for r in range(32):
            at = (h + H0 * r) * (G + 1) + tp
            assert np.isnan(buf[at])
            buf[at] = v[bitrev(r, 5)]
    out = np.full(F // 2, np.nan, complex)
    for t in range(NT):
        v = list(buf[t * (G + 1) + np.arange(32)])
        NS = 32 * H0
        butterfly32(v, lambda q, k: rho[4 + H0 + q] * np.exp(-2j * np.pi * (t + NS * k) / (NS << (q + 1))), 0, True)
        for e in range(16):
            c = t + NT * e
            out[c] = v[bitrev(e, 5)] * (-1) ** bin(c & ~(H0 - 1)).count("1")
    ref = np.fft.fft(x * rot)[:F // 2]
    assert np.abs(out - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("F,npol", [(1024, 1), (1024, 2), (2048, 1), (2048, 2)])
@pytest.mark.parametrize("offset", [0, 1, 7, 15, 16, 17, 31, 1023])
def test_words_hold_the_samples(F, npol, offset):
    """Every lane's words: the FFT's bits alone are touched, and the shifted words are the samples in order."""
    rng = np.random.default_rng(offset)
    nword = (2 * npol * (F + offset) + 31) // 32
    row = rng.integers(0, 2 ** 32, nword, dtype=np.uint64)
    bits = np.unpackbits(row.astype("<u4").view(np.uint8), bitorder="little")
    bit = offset * 2 * npol
    sh = bit & 31
    got = np.zeros(2 * npol * F, np.uint8)
    for t in range(32):
        for g in range(F // 512):
            at = (bit >> 5) + npol * t + 32 * npol * g
            w = [row[at + k] if k < npol or sh else 0 for k in range(npol + 1)]   # IndexError: past the row
            for k in range(npol):
                v = (int(w[k]) | int(w[k + 1]) << 32) >> sh & 0xFFFFFFFF
                i = 32 * npol * (t + 32 * g) + 32 * k
                got[i:i + 32] = [v >> b & 1 for b in range(32)]
    np.testing.assert_array_equal(got, bits[bit:bit + 2 * npol * F])


# as the other tests of FP32 visibilities against 64 bits: relative to the largest value of a product's spectrum
VIS_TOL = 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("nchan", [512, 1024])
@pytest.mark.parametrize("nant,npol,numffts", [(2, 1, 1), (2, 2, 1), (3, 1, 65), (3, 2, 64), (70, 1, 131), (2, 1, 9001)])
def test_against_oracle(nchan, nant, npol, numffts):
    job = synth.random_job(nant=nant, npol=npol, nchan=nchan, numffts=numffts, bw=32e6, seed=nant + nchan, nsubband=1)
    cfg = fx.make_config(nant, nchan, numffts, job.bw, job.lo, npol=npol)
    with fx.Correlator(cfg) as c:
        c.process(job.data, job.delays, job.fileoffsets)
        vis, counts = c.visibilities()
    ref, rc = fo.correlate(job.data[0], job.delays, job.fileoffsets, job.bw, job.lo, nchan, npol, numffts=numffts,
                           maxoffset_ffts=numffts)
    np.testing.assert_array_equal(counts, rc)
    assert fo.vis_error(vis[0], ref)[0].max() < VIS_TOL
