"""The correlations this library is measured on.

A case is one subintegration (or the part of one that a call covers) from packed samples to
visibilities, through the entry points a user's program calls: reset, process, read the
visibilities.  `listed()` holds the sizes that stand for a kind of use each; `draw()` gives other
sizes of the same kinds.  `exact()` restates the correlation in 64 bits with torch alone.

Fields of a case:
  api       "device"  input rows already on the device, visibilities left there
            "window"  device rows streamed in windows of `window` FFTs, device-resident accumulators
            "host"    pinned host rows in, pinned host visibilities out (the reference's own call)
            "batch"   twelve uneven jobs in one batch, visibilities read to pinned host memory
  nant npol nchan nsb numffts   antennas, polarisations, channels, subbands, FFTs
  form      X stage: "plain" (FP32), "fp16", "fp8" (tensor cores)
  fstage    F stage: "auto" (FP32 FFT), "tc32", "tc16" (tensor-core DFTs)
  cpx       False: 2-bit real samples; True: 8-bit complex samples
  mhz       bandwidth of a subband
"""
import ctypes
import math

import numpy as np
import torch

import difx_tests_b200 as fx

LO = 1.4e9
RHO = 0.1                                # share of the samples all antennas have in common
HIMAG = float(np.float32(3.3359))        # quantiser levels -HIMAG, -1, 1, HIMAG
CODE_P = (0.1635, 0.3365, 0.3365, 0.1635)   # a unit Gaussian cut at -0.98, 0, 0.98

FORMS = {"plain": fx.FXC_X_PLAIN_FP32, "fp16": fx.FXC_X_TC_FP16, "fp8": fx.FXC_X_TC_FP8}
FSTAGES = {"auto": fx.FXC_F_AUTO, "tc32": fx.FXC_F_TC32, "tc16": fx.FXC_F_TC16}


def _case(name, nant, npol, nchan, nsb, numffts, form="plain", fstage="auto", api="device", cpx=False, mhz=64,
          window=0):
    return {"name": name, "api": api, "nant": nant, "npol": npol, "nchan": nchan, "nsb": nsb, "numffts": numffts,
            "form": form, "fstage": fstage, "cpx": cpx, "mhz": mhz, "window": window}


def listed():
    return [
        # a quick look at a few milliseconds of data: launches and host latency count
        _case("quick_look", 4, 2, 128, 1, 100, mhz=32),
        # the reference's own test4 scale: 25 ms of 4 antennas
        _case("small_array", 4, 1, 256, 1, 3125, mhz=32),
        # an odd number of antennas, subbands and FFTs: no tile, chunk or segment comes out even
        _case("ragged_array", 23, 1, 512, 3, 2777, mhz=32),
        # the reference's test16 scale: 16 dual-polarisation antennas, 1 s, in FP32 throughout
        _case("dual_pol_plain", 16, 2, 2048, 4, 31250),
        # the same with the tensor-core X stage
        _case("dual_pol_fp16", 16, 2, 2048, 4, 31250, form="fp16"),
        # a 64-antenna array, half a second of 8 subbands, in FP32 throughout
        _case("array64_plain", 64, 1, 1024, 8, 31250),
        # the same in the fastest form at FP32 F-stage accuracy: tensor-core DFT and X stage
        _case("array64_tc32", 64, 1, 1024, 8, 31250, form="fp16", fstage="tc32"),
        # many antennas where the X stage is the larger part: FP8 operands
        _case("array200_fp8", 200, 1, 1024, 1, 4096, form="fp8"),
        # a large full-polarisation array, one subband of it, streamed in windows
        _case("large_stream", 256, 2, 4096, 1, 2048, form="fp16", api="window", window=1024),
        # twelve uneven jobs submitted at once
        {"name": "uneven_batch", "api": "batch", "jobs": 12, "draw": 3},
        # 8-bit complex samples: every FFT bin a channel
        _case("complex8", 24, 2, 1024, 2, 3000, cpx=True),
        # the drop-in call: host rows in, host visibilities out
        _case("host_rows", 16, 2, 2048, 2, 6250, api="host"),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: 2 to 256 antennas, 128 to 4096 channels, 64 to 31250 FFTs."""
    while True:
        kind = rng.choice(["plain", "plain", "plain", "fp16", "fp16", "tc32", "tc16", "fp8", "complex", "host",
                           "window", "batch"])
        if kind == "batch":
            return {"api": "batch", "jobs": rng.randint(3, 12), "draw": rng.randint(4, 10 ** 6)}
        form, fstage, api, cpx, window = "plain", "auto", "device", False, 0
        nant, npol, nchan = _loguniform(rng, 2, 256), rng.choice([1, 2]), 1 << rng.randint(7, 12)
        nsb, numffts = rng.randint(1, 8), _loguniform(rng, 64, 31250)
        if kind in ("fp16", "fp8"):
            form = kind
        elif kind in ("tc32", "tc16"):
            form, fstage, npol, nchan = "fp16", kind, 1, 1024
        elif kind == "complex":
            cpx, nchan = True, max(nchan, 256)
            form = rng.choice(["plain", "fp16"])
        elif kind == "host":
            api = "host"
        elif kind == "window":
            api, form = "window", rng.choice(["plain", "fp16"])
            window = 64 * rng.randint(2, 16)
        c = _case("", nant, npol, nchan, nsb, numffts, form, fstage, api, cpx, rng.choice([16, 32, 64]), window)
        del c["name"]
        nsig = nant * npol
        samples = nsig * nsb * numffts * nchan * (1 if cpx else 2)
        mac = samples * (nsig + 1)
        in_bytes = samples * (2 if cpx else 0.25)
        # costs: at most the listed cases'; the host's copies at most a tenth of a second
        if (samples <= 16e9 and mac <= (1e12 if form == "plain" else 4e12) and in_bytes <= (5e9 if api != "host" else 1e9)
                and _vis_count(c) * 8 <= (4e9 if api != "host" else 4e8)):
            return c


# ------------------------------------------------------------------------------ sizes
def _fft_len(c):
    return c["nchan"] if c["cpx"] else 2 * c["nchan"]


def _row_bytes(c):
    """Packed bytes of one antenna and subband: numffts + 1 FFTs."""
    bits = 16 if c["cpx"] else 2
    return _fft_len(c) * (c["numffts"] + 1) * bits * c["npol"] // 8


def _vis_count(c):
    nant = c["nant"]
    return c["nsb"] * nant * (nant + 1) // 2 * c["npol"] ** 2 * c["nchan"]


def _jobs(case):
    """The jobs of a batch: antennas from 4 to 56, 256 to 8192 points, 1 to 8 subbands, 5 to 200 ms."""
    rng = np.random.default_rng(case["draw"])
    ants = [4, 6, 8, 10, 12, 16, 20, 24, 32, 40, 48, 56]
    jobs = []
    for a in ants[12 - case["jobs"]:]:
        F = int(rng.choice([256, 512, 1024, 4096, 8192]))
        nsb = int(rng.integers(1, 9))
        n = int(round(float(rng.uniform(5e-3, 200e-3)) * 64e6 / F))
        jobs.append(_case("", a, 1, F // 2, nsb, n, mhz=32))
    return jobs


def _work1(c):
    F, nsig = _fft_len(c), c["nant"] * c["npol"]
    ffts = nsig * c["nsb"] * c["numffts"]
    return {"bytes": float(c["nsb"] * c["nant"] * _row_bytes(c) + _vis_count(c) * 8),
            "flops": float(ffts * (5 * F * math.log2(F) + 6 * F)
                           + 8 * nsig * (nsig + 1) // 2 * c["nchan"] * c["nsb"] * c["numffts"])}


def work(case):
    """Samples in once, visibilities out once; the FFTs, the two rotations and the multiply-adds."""
    jobs = [_work1(j) for j in (_jobs(case) if case["api"] == "batch" else [case])]
    return {k: sum(j[k] for j in jobs) for k in ("bytes", "flops")}


# ------------------------------------------------------------------------------ inputs
def _delays(c, seed):
    """Quadratic delay model per antenna (seconds; the polynomial's t counts FFTs) and file offsets."""
    rng = np.random.default_rng(seed)
    T = _fft_len(c) / ((1.0 if c["cpx"] else 2.0) * c["mhz"] * 1e6)
    n = c["nant"]
    a0, a1, a2 = rng.uniform(-1e-3, 1e-3, n), rng.uniform(-3e-6, 3e-6, n), rng.uniform(-1e-10, 1e-10, n)
    return np.stack([a2 * T * T, a1 * T, a0], axis=1), a0.copy()


def _byte_table(dev):
    """65536 bytes of four 2-bit codes with a quantised Gaussian's frequencies."""
    p = np.asarray(CODE_P)
    prob = np.array([p[b & 3] * p[(b >> 2) & 3] * p[(b >> 4) & 3] * p[b >> 6] for b in range(256)])
    edge = np.concatenate([[0.0], np.cumsum(prob / prob.sum())])
    return torch.from_numpy(np.repeat(np.arange(256), np.diff(np.round(edge * 65536).astype(int))).astype(np.uint8)).to(dev)


def _fill(rows, c, seed):
    """Samples of every (subband, antenna) row: a share RHO common to the subband's antennas."""
    dev = rows.device
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    nb = _row_bytes(c)

    def fresh():
        if c["cpx"]:
            out = torch.empty(nb, dtype=torch.int8, device=dev)
            for at in range(0, nb, 1 << 26):
                n = min(1 << 26, nb - at)
                out[at:at + n] = (20.0 * torch.randn(n, generator=g, device=dev)).clamp_(-127, 127).round_().to(torch.int8)
            return out.view(torch.uint8)
        r = torch.randint(-2 ** 31, 2 ** 31, (nb,), generator=g, device=dev, dtype=torch.int32)
        return table[(r & 0xFFFF)], r

    table = None if c["cpx"] else _byte_table(dev)
    for sb in range(c["nsb"]):
        common = fresh()
        for ant in range(c["nant"]):
            own = fresh()
            row = rows[sb * c["nant"] + ant]
            if c["cpx"]:
                m = torch.rand(nb // 2, generator=g, device=dev).lt_(RHO).bool().repeat_interleave(2)
                row[:nb] = torch.where(m, common, own)
            else:
                row[:nb] = torch.where((own[1] >> 16) + 32768 < int(RHO * 65536), common[0], own[0])


class _Wrap:
    """A device buffer of the library as a torch tensor."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "|u1", "version": 2}


def _config(c):
    return fx.make_config(c["nant"], c["nchan"], c["numffts"], c["mhz"] * 1e6, LO, npol=c["npol"], nsubband=c["nsb"],
                          xmode=FORMS[c["form"]], cpx=c["cpx"], fstage=FSTAGES[c["fstage"]], window_ffts=c["window"])


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _vis_shape(c):
    nant = c["nant"]
    return (c["nsb"], nant * (nant + 1) // 2, c["npol"] ** 2, c["nchan"])


def prepare(case, seed):
    if case["api"] == "batch":
        return _prepare_batch(case, seed)
    c = case
    delays, offs = _delays(c, seed)
    corr = fx.Correlator(_config(c))
    s = {"case": c, "corr": corr, "delays": delays, "offs": offs}
    nrow, nb = c["nsb"] * c["nant"], _row_bytes(c)
    if c["api"] == "device":
        ptr, pitch = corr.device_input()
        rows = torch.as_tensor(_Wrap(ptr, (nrow, pitch)), device="cuda")
        _fill(rows, c, seed)
        s.update(ptr=ptr, pitch=pitch)
    elif c["api"] == "window":
        pitch = (nb + 32 + 255) // 256 * 256
        rows = torch.zeros((nrow, pitch), dtype=torch.uint8, device="cuda")
        _fill(rows, c, seed)
        s.update(rows=rows, pitch=pitch)
    else:
        rows = torch.empty((nrow, nb), dtype=torch.uint8, device="cuda")
        _fill(rows, c, seed)
        host = _pinned((c["nsb"], c["nant"], nb), torch.uint8)
        torch.from_numpy(host).view(nrow, nb).copy_(rows)
        s.update(host=host, out=_pinned(_vis_shape(c), torch.complex64))
    if c["api"] != "host":
        s["vis"] = torch.empty(_vis_shape(c), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()   # the samples are there before the library's own stream reads them
    return s


def _prepare_batch(case, seed):
    jobs = _jobs(case)
    batch = fx.Batch([_config(c) for c in jobs])
    out = []
    for j, c in enumerate(jobs):
        rows = torch.empty((c["nsb"] * c["nant"], _row_bytes(c)), dtype=torch.uint8, device="cuda")
        _fill(rows, c, seed * 64 + j)
        host = _pinned((c["nsb"], c["nant"], _row_bytes(c)), torch.uint8)
        torch.from_numpy(host).view(rows.shape).copy_(rows)
        batch.upload(j, host)
        batch.set_model(j, *_delays(c, seed * 64 + j))
        out.append((_pinned(_vis_shape(c), torch.complex64), _pinned(c["nant"] * (c["nant"] + 1) // 2, torch.int32)))
        batch.synchronize()
    return {"case": case, "batch": batch, "out": out}


def run(s):
    c = s["case"]
    if c["api"] == "batch":
        batch = s["batch"]
        batch.reset()
        batch.process()
        for j, (vis, counts) in enumerate(s["out"]):
            st = fx.lib().fxc_batch_get_visibilities(batch._b, j, vis.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                                                     counts.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), 0)
            if st != fx.FXC_OK:
                raise fx.FxcError(st, "fxc_batch_get_visibilities")
        return {"vis": [v for v, _ in s["out"]], "counts": [n for _, n in s["out"]]}
    corr = s["corr"]
    corr.reset()
    if c["api"] == "host":
        corr.process(s["host"], s["delays"], s["offs"])
        vis, counts = corr.visibilities(out=s["out"])
        return {"vis": vis, "counts": counts}
    if c["api"] == "device":
        corr.process_device(s["ptr"], s["pitch"], s["delays"], s["offs"])
    else:
        # each window's rows begin two FFTs before its first FFT: the delays move the samples
        F, W = _fft_len(c), c["window"]
        per_fft = _row_bytes(c) // (c["numffts"] + 1)
        for first in range(0, c["numffts"], W):
            lead = max(0, first - 2)
            end = min(first + W + 2, c["numffts"] + 1)
            corr.process_device_window(s["rows"].data_ptr() + lead * per_fft, s["pitch"],
                                       np.full(c["nant"], lead * F, np.int64), (end - lead) * per_fft, s["delays"],
                                       s["offs"], first, min(W, c["numffts"] - first))
    counts = corr.visibilities_device(s["vis"].data_ptr())
    return {"vis": s["vis"], "counts": counts}


# ------------------------------------------------------------------------------ 64 bits
def _table(c, delays, offs):
    """Delay model, integer sample offset, fractional delay and validity of every (antenna, FFT)."""
    F = _fft_len(c)
    Ts = 1.0 / ((1.0 if c["cpx"] else 2.0) * c["mhz"] * 1e6)
    k = np.arange(c["numffts"], dtype=np.float64)[None, :]
    q, l, c0 = (delays[:, i:i + 1] for i in range(3))
    d0, d1, d2 = (q * t * t + l * t + c0 for t in (k, k + 0.5, k + 1.0))
    a = d2 - d0
    b = d0 + (d1 - (a * 0.5 + d0)) / 3.0
    nf = (a * 0.5 + b - offs[:, None]) / Ts
    n = np.trunc(nf + 0.5)
    frac = -(nf - n) * Ts
    off = k * F - n
    last = (c["numffts"] - 1) * F
    frac = np.where(off == -1, frac + Ts, np.where(off == last + 1, frac - Ts, frac))
    off = np.where(off == -1, 0, np.where(off == last + 1, last, off))
    return a, b, frac, off.astype(np.int64), (off >= 0) & (off <= last)


def _exact1(c, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    F, C, nant, npol, nsig = _fft_len(c), c["nchan"], c["nant"], c["npol"], c["nant"] * c["npol"]
    rows = torch.zeros((c["nsb"] * nant, _row_bytes(c) + 8), dtype=torch.uint8, device=dev)
    _fill(rows, c, seed)
    a, b, frac, off, valid = _table(c, *_delays(c, seed))
    at = [torch.from_numpy(np.ascontiguousarray(x)).to(dev) for x in (a, b, frac, off, valid)]
    bw = c["mhz"] * 1e6
    stride = 1 << (int(math.log2(C)) // 2)   # rotators: sub (fine) and step (coarse) factors
    S = F // stride
    sub_x = torch.arange(S, device=dev, dtype=torch.float64) / F
    step_x = torch.arange(stride, device=dev, dtype=torch.float64) * stride / F
    chan_w = 2 * math.pi * bw / C * torch.arange(C, device=dev, dtype=torch.float64)
    levels = torch.tensor([-HIMAG, -1.0, 1.0, HIMAG], dtype=torch.float64, device=dev)
    n = torch.arange(F, device=dev)
    iu, ju = [], []
    bls = [(i, j) for i in range(nant - 1) for j in range(i + 1, nant)] + [(i, i) for i in range(nant)]
    for i, j in bls:
        for l in range(npol):
            for m in range(npol):
                iu.append(i * npol + l)
                ju.append(j * npol + m)
    iu, ju = torch.tensor(iu, device=dev), torch.tensor(ju, device=dev)
    out = torch.empty(_vis_shape(c), dtype=torch.complex128, device=dev)
    nt = max(1, (1 << 26) // (nsig * F))

    def turns(ph):   # exp(-2 pi i ph), the whole turns taken out first
        x = -2.0 * math.pi * (ph - torch.trunc(ph))
        return torch.polar(torch.ones_like(x), x)

    for sb in range(c["nsb"]):
        lo = LO + sb * bw
        data = rows[sb * nant:(sb + 1) * nant]
        V = torch.zeros((C, nsig, nsig), dtype=torch.complex128, device=dev)
        for t0 in range(0, c["numffts"], nt):
            ta, tb, tf, to, tv = (x[:, t0:t0 + nt] for x in at)
            m = ta.shape[1]
            s = to.clamp(0, (c["numffts"] - 1) * F)[:, :, None] + n
            if c["cpx"]:
                x = torch.empty((nant, npol, m, F), dtype=torch.complex128, device=dev)
                signed = data.view(torch.int8)
                for p in range(npol):
                    at2 = (2 * (s * npol + p)).view(nant, -1)
                    x[:, p] = torch.complex(signed.gather(1, at2).double(),
                                            signed.gather(1, at2 + 1).double()).view(nant, m, F)
            else:
                x = torch.empty((nant, npol, m, F), dtype=torch.float64, device=dev)
                per = 4 // npol
                byte = data.gather(1, (s // per).view(nant, -1)).view(nant, m, F).to(torch.int32)
                for p in range(npol):
                    sh = ((s % per) * (2 * npol) + 2 * p).to(torch.int32)
                    x[:, p] = levels[((byte >> sh) & 3).long()]
            whole = torch.trunc(tb)
            ph = (sub_x * ta[..., None] + (tb - whole)[..., None]) * lo
            if lo - math.trunc(lo) > 1e-11:
                ph = ph + (lo - math.trunc(lo)) * whole[..., None]
            rot = (turns(step_x * ta[..., None] * lo)[..., :, None] * turns(ph)[..., None, :]).reshape(nant, 1, m, F)
            X = torch.fft.fft(x * rot)[..., :C]
            w = chan_w * tf[..., None]
            X = X * (torch.polar(torch.ones_like(w), w) * tv[..., None])[:, None]
            X = X.reshape(nsig, m, C).permute(2, 0, 1).contiguous()
            V.baddbmm_(X, X.conj().transpose(1, 2))
        for p in range(npol * npol):   # [bl][prod][chan]
            i, j = iu[p::npol * npol], ju[p::npol * npol]
            for at0 in range(0, len(i), 4096):
                out[sb, at0:at0 + 4096, p] = V[:, i[at0:at0 + 4096], j[at0:at0 + 4096]].T
    counts = np.array([int((valid[i] & valid[j]).sum()) for i, j in bls], np.int32)
    return out, counts


def exact(case, seed):
    if case["api"] == "batch":
        got = [_exact1(c, seed * 64 + j) for j, c in enumerate(_jobs(case))]
        return {"vis": [v for v, _ in got], "counts": [n for _, n in got]}
    vis, counts = _exact1(case, seed)
    return {"vis": vis, "counts": counts}
