"""CPU restatement of the paired FFT F stage (difx_tests_b200/csrc/fx_fpair.cuh): its FMA-form butterflies with
the fringe rotation folded in, its index maps and its sample expansion, in numpy.  In float64 the
factorisation is the rotated DFT itself (2e-13 of max|X|: thirteen stages of float64 roundings), every
shared-memory index stays inside its buffer and is written before it is read."""
import numpy as np
import pytest

from oracle import fxoracle as fo

LASTR = {256: 16, 512: 2, 1024: 4, 2048: 8, 4096: 16, 8192: 2}


def plan(F, cpx):
    C = F if cpx else F // 2
    npass = 2 if F == 256 else 3 if F <= 4096 else 4
    stride = 1 << (int(np.log2(C)) // 2)
    return dict(C=C, NT=F // 16, npass=npass, stride=stride, S=F // stride, logf=int(np.log2(F)), BUF=F + F // 16)


def padi(i):
    return i + (i >> 4)


def bitrev(v, bits):
    return int(format(v, f"0{bits}b")[::-1], 2) if bits else 0


def butterfly(v, R, w, lo):
    """v: list of R arrays; w(q, k'): twiddle of stage q, sub-transform k' (its rho included)."""
    M = int(np.log2(R))
    for q in range(M):
        half = R >> (q + 1)
        for kp in range(1 << q):
            base = bitrev(kp, q) * (R >> q)
            ref = kp if q == 0 or kp < 1 << (q - 1) else kp - (1 << (q - 1))   # the others: -i times one
            wd = w(q, ref) * (1 if ref == kp else -1j)
            for h in range(half):
                a, b = v[base + h], v[base + half + h]
                s = a + wd * b
                v[base + h], v[base + half + h] = s, (None if lo and q == M - 1 else s - 2 * a)


def fpair_fft(x, rho, F, cpx):
    """One lane: F samples, rho[stage] -> channels with the sign (-1)^popcount(c) still on them."""
    p = plan(F, cpx)
    NT, t = p["NT"], np.arange(p["NT"])
    buf = np.full(p["BUF"], np.nan, complex)

    def load(idx):
        assert idx.min() >= 0 and idx.max() < p["BUF"]
        assert not np.isnan(buf[idx]).any()
        return buf[idx].copy()

    out = np.full(p["C"], np.nan, complex)
    NS = 1
    for ps in range(p["npass"]):
        last = ps == p["npass"] - 1
        R = LASTR[F] if last else 16
        NB, M = 16 // R, int(np.log2(R))
        lo = last and not cpx
        v = {}
        for b in range(NB):
            j = t + b * NT
            v[b] = [x[j + r * (F // R)].astype(complex) if ps == 0 else load(padi(t) + b * (NT + NT // 16)
                    + r * (F // R + F // R // 16)) for r in range(R)]
            for r in range(R):   # the padded offsets fold
                assert np.array_equal(padi(t) + b * (NT + NT // 16) + r * (F // R + F // R // 16),
                                      padi(j + r * (F // R)))
        buf[:] = np.nan
        for b in range(NB):
            j = t + b * NT
            jm = j & (NS - 1)
            butterfly(v[b], R, lambda q, kp: rho[4 * ps + q] * np.exp(-2j * np.pi * (jm + NS * kp) / (NS << (q + 1))), lo)
            for r in range(R // 2 if lo else R):
                y = v[b][bitrev(r, M)]
                if last:
                    out[t + NT * (b + NB * r)] = y
                else:
                    idx = padi((j // NS) * NS * R + (j & (NS - 1))) + r * (1 if NS == 1 else NS + NS // 16)
                    assert idx.max() < p["BUF"] and np.isnan(buf[idx]).all()
                    for k in range(0, NT, 8):   # 16-byte elements: a quarter warp on eight bank groups
                        assert NT < 8 or len(set(idx[k:k + 8] % 8)) == 8
                    buf[idx] = y
        NS *= R
    return out


@pytest.mark.parametrize("cpx", [False, True])
@pytest.mark.parametrize("F", [256, 512, 1024, 2048, 4096, 8192])
def test_rotated_fft(F, cpx):
    if cpx and F == 8192:
        pytest.skip("complex samples: at most 4096 channels")
    p = plan(F, cpx)
    rng = np.random.default_rng(F + cpx)
    x = rng.standard_normal(F) + (1j * rng.standard_normal(F) if cpx else 0)
    a, b, lo, frac, bw = 3.1e-9, 2.0000001e-4, 1.4e9 + 0.25, 3.3e-9, 64e6
    # factors as pair_entry builds them
    rho = []
    for s in range(p["logf"]):
        bit = p["logf"] - 1 - s
        w = 2.0 ** bit / F if 2 ** bit < p["S"] else (2 ** bit // p["S"]) * p["stride"] / F
        rho.append(np.exp(-2j * np.pi * (w * a * lo)))
    c = np.arange(p["C"])
    sign = np.array([(-1.0) ** bin(k).count("1") for k in c])
    ph = (b - np.trunc(b)) * lo + (lo - np.trunc(lo)) * np.trunc(b)
    fac = np.exp(1j * np.pi * c * (2 * bw / p["C"]) * frac) * np.exp(-2j * np.pi * ph) * sign
    got = fpair_fft(x, rho, F, cpx) * fac
    rot = fo.fringe_rotator(np.array(a), np.array(b), lo, p["C"], ref_args=False, cpx=cpx)
    ref = np.fft.fft(x * rot)[: p["C"]] * np.exp(2j * np.pi * c * bw * frac / p["C"])
    assert np.abs(got - ref).max() < 1e-8 * np.abs(ref).max()      # phases of 1e5 turns in float64
    plain = fpair_fft(x, np.ones(p["logf"]), F, cpx) * sign
    ref = np.fft.fft(x)[: p["C"]]
    assert np.abs(plain - ref).max() < 2e-13 * np.abs(ref).max()


@pytest.mark.parametrize("F", [256, 512, 1024, 2048, 4096, 8192])
def test_first_exchange_and_sample_permutation(F):
    """Real input: thread t = 16 d0 + u takes samples n = r NT + u NT / 16 + d0, its exchange row holds what the
    16 threads of d0 hand to butterfly t of pass 1, and its byte reads hit distinct banks."""
    NT = F // 16
    t = np.arange(NT)
    u, d0 = t & 15, t >> 4
    n0 = u * (NT // 16) + d0
    assert np.array_equal(np.sort(n0), t)                   # every sample column once
    # pass 0 of column n0 gives outputs k0 = 0 .. 15 at Stockham index 16 n0 + k0; pass 1 thread j reads j + r NT
    row = {}
    for k0 in range(16):
        for a, i in zip(272 * d0 + 17 * u + k0, 16 * n0 + k0):
            assert a not in row and a < F + F // 16
            row[a] = i
    for r in range(16):
        got = [row[a] for a in 272 * d0 + 17 * r + u]
        assert np.array_equal(got, t + r * NT)
        # pass 1's stores fall into the thread's own row, at padi of their Stockham index
        assert np.array_equal(272 * d0 + 17 * r + u, padi((t >> 4) * 256 + (t & 15) + 16 * r))
    swz = {512: 3, 256: 1}.get(NT, 0)
    for r in range(16):
        n = n0 + r * NT
        addr = (n0 ^ (((n0 >> 7) & swz) << 2)) + r * NT     # as pass 0 reads
        word = (n >> 2) ^ ((n >> 7) & swz)                  # as the expansion writes (words of 16 samples permuted)
        assert np.array_equal(addr, 4 * word + (n & 3))
        for w in range(0, NT, 32):
            words = set(addr[w:w + 32] >> 2)
            assert len(set(x % 32 for x in words)) == len(words)


@pytest.mark.parametrize("npol", [1, 2])
@pytest.mark.parametrize("F", [256, 1024, 8192])
def test_sample_expansion(F, npol):
    """Packed bytes at every sample offset mod 64 -> the table offset 8 (code A + 4 code B) of each sample."""
    rng = np.random.default_rng(F + npol)
    M32 = 0xFFFFFFFF
    inb = ((F * npol // 4 + 1 + 15 + 15) // 16 * 16) + 16       # staging buffer of one window
    for off in range(64 // npol):
        bit = off * 2 * npol
        first = bit >> 3
        base = first & ~15
        nvec = (F * npol // 4 + 1 + (first - base) + 15) >> 4
        assert 16 * nvec <= inb - 16
        rel = bit - 8 * base
        win = [rng.integers(0, 256, inb, dtype=np.uint8) for _ in range(2)]
        codes = []
        for l in range(2):
            s = np.arange(F)
            w = win[0] if npol == 2 else win[l]
            at = rel + s * 2 * npol + (2 * l if npol == 2 else 0)
            codes.append((w[at >> 3] >> (at & 7)) & 3)
        want = 8 * (codes[0] + 4 * codes[1])
        words = [w.view("<u4").astype(object) for w in win]
        got = np.zeros(F, int)
        for t in range(F // 16):
            nib = []
            if npol == 2:
                i = 2 * t + (rel >> 5)
                assert 4 * (i + 2) + 4 <= inb
                for h in range(2):
                    nib.append((((words[0][i + h + 1] << 32) | words[0][i + h]) >> (rel & 31)) & M32)
            else:
                sp = []
                for l in range(2):
                    i = t + (rel >> 5)
                    assert 4 * (i + 1) + 4 <= inb
                    a = (((words[l][i + 1] << 32) | words[l][i]) >> (rel & 31)) & M32
                    row = []
                    for h in range(2):
                        x = (a >> 16) if h else a & 0xFFFF
                        x = (x | (x << 8)) & 0x00FF00FF
                        x = (x | (x << 4)) & 0x0F0F0F0F
                        row.append((x | (x << 2)) & 0x33333333)
                    sp.append(row)
                nib = [sp[0][h] | (sp[1][h] << 2) for h in range(2)]
            for h in range(2):
                ev, od = (nib[h] << 3) & 0x78787878, (nib[h] >> 1) & 0x78787878
                by = [(ev >> 8 * k) & 255 for k in range(4)] + [(od >> 8 * k) & 255 for k in range(4)]
                for w, sel in enumerate((0x5140, 0x7362)):
                    for k in range(4):
                        got[16 * t + 8 * h + 4 * w + k] = by[(sel >> 4 * k) & 15]
        assert np.array_equal(got, want)
