"""CPU check of the index arithmetic of the tensor-core X stage on channel-contiguous FP16 spectra
(difx_tests_b200/csrc/fx_xtch.cu), restated from the kernel: the turn's reads stay inside a stage and take
no bank conflicts, its stores fill every 4-byte word of K half h of rows < 2 nsig of each channel's tile
exactly once, with the FFT pair and the part (Re / Im) the K-major SWIZZLE_128B layout puts there, at most
one bank pass per store, and the tiles' 128-row operand reads stay inside the shared block."""
import pytest

BT, RING, TILES, NTW = 32, 128 * 1024, 64 * 1024, 8


def turn(nsig, cb, h):
    tile = 512 // cb * 128
    reads, writes = {}, {}
    for warp in range(NTW):
        for s0 in range(4 * warp, nsig, 4 * NTW):
            for u in range(2 if cb == 4 else 4):
                for lane in range(32):
                    w, g = (lane & 15, lane >> 4) if cb == 4 else (lane >> 1, lane & 1)
                    j = (w >> 2) & 1 if cb == 4 else (w >> 1) & 1
                    s = s0 + (u + 2 * g if cb == 4 else (u >> 1) + 2 * (g ^ (u & 1)))
                    if s >= nsig:
                        continue
                    base = (s * BT + 2 * w) * 4 * cb + (0 if cb == 4 else 16 * g)
                    for n, t in ((0, j), (1, 1 - j)):
                        reads.setdefault((warp, s0, u, n), []).append((lane, base + t * 4 * cb))
                    k = 4 * h + (w >> 2)
                    for part in range(2):
                        r = 2 * s + part
                        for c in range(4):
                            ch = c if cb == 4 else 4 * g + c
                            writes.setdefault((warp, s0, u, part, c), []).append(
                                (lane, ch * tile + (w & 3) * 4 + r * 128 + ((k ^ (r & 7)) << 4), ch, r, 32 * h + 2 * w))
    return tile, reads, writes


@pytest.mark.parametrize("h", [0, 1])
@pytest.mark.parametrize("nsig", [1, 2, 3, 5, 8, 31, 32, 33, 50, 63, 64])
def test_turn(nsig, h):
    cb = 8 if nsig <= 32 else 4
    stage = nsig * BT * cb * 4
    assert RING // stage >= 4
    tile, reads, writes = turn(nsig, cb, h)
    assert cb * tile == TILES and (cb - 1) * tile + 128 * 128 <= TILES + RING
    for ops in reads.values():
        assert all(0 <= a and a + 16 <= stage and a % 16 == 0 for _, a in ops)
        for q in range(4):   # 16-byte reads: a quarter warp per pass, 8 slots of 16 bytes
            slots = [a // 16 % 8 for lane, a in ops if lane // 8 == q]
            assert len(set(slots)) == len(slots)
    seen = {}
    for ops in writes.values():
        banks = [a // 4 % 32 for _, a, *_ in ops]
        assert len(set(banks)) == len(banks)
        for _, a, ch, r, fft in ops:
            assert a not in seen
            seen[a] = (ch, r, fft)
    want = {}
    for ch in range(cb):
        for r in range(2 * nsig):
            for fft in range(32 * h, 32 * h + 32, 2):
                chunk = fft // 8
                want[ch * tile + r * 128 + ((chunk ^ (r & 7)) << 4) + fft % 8 * 2] = (ch, r, fft)
    assert seen == want
