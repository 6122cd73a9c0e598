"""The calls whose speed this repository is judged by.

``listed()`` names twelve of them, from a small streaming block to the
256-channel batch; ``draw(rng)`` gives more of the same ranges.  Every case
goes through the package's public classes, on the signals of
``libfalcon_dsp_gb300/workloads.py`` or generic ones, with a fresh handle
whose streaming state runs on from pass to pass, as in a receiver's loop.

``exact`` is the first pass of a fresh handle in 64 bits, from the formulas of
the path: the NCO e^{j 2 pi f/fs (n mod R)}, the polyphase sum
y[m] = sum_j h[j U + (m D mod U)] x[floor(m D / U) - j], the FIR and the
discriminator arg(x[n] conj(x[n-1])).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import libfalcon_dsp_gb300 as F
from libfalcon_dsp_gb300 import workloads as W

DEV = "cuda"
C3_FS = 61440000  # input rate of the batched channelizer
C2_FS = 10000000  # input rate of the 8-channel streaming channelizer
RATIOS = [(147, 160), (160, 147), (1, 2), (1, 10), (2, 5), (3, 125), (3, 2), (7, 8), (24, 25), (1, 64)]


def listed():
    return [
        # a receiver's streaming loop: 8 carriers of one 10 MS/s input, short blocks, CUDA graph replay
        dict(name="chan8_stream_64k", kind="channelizer", signal="qpsk", nch=8, n=1 << 16, mode="fp32", dtype="c64",
             plan=0, graph=True),
        # the reference's call on std::vector data: the same channelizer on host arrays
        dict(name="chan8_host_1m", kind="channelizer_host", n=1000003, nch=8),
        # a server's larger job in the default precision: 64 channels of one block
        dict(name="chan64_fp32_1m", kind="channelizer", signal="tones", nch=64, n=1 << 20, mode="fp32", dtype="c64",
             plan=11, graph=False),
        # the batched workload: 256 uneven channels of one 2^26-sample input on the tensor cores
        dict(name="chan256_fp16x3_64m", kind="channelizer", signal="tones", nch=256, n=1 << 26, mode="fp16x3",
             dtype="c64", plan=3, graph=True),
        # the same path from a digitiser's int16 samples, in the other 16-bit format, odd block
        dict(name="chan64_bf16x3_ci16_4m", kind="channelizer", signal="tones", nch=64, n=4000001, mode="bf16x3",
             dtype="ci16", plan=12, graph=False),
        # sample-rate conversion 48 kHz -> 44.1 kHz, 3528 taps
        dict(name="resample_147_160_1m", kind="resample", up=147, down=160, tpp=24, n=1 << 20, mode="fp32"),
        # the long channel filter of the FM receiver chain: 4095 taps, every 10th output
        dict(name="resample_4095_by10_16m", kind="resample", up=1, down=10, tpp=4095, n=1 << 24, mode="fp16x3"),
        # full-rate FIR with complex taps, default precision, odd block
        dict(name="fir64_fp32_1m", kind="fir", taps=64, n=1048573, mode="fp32"),
        # the same filter over a recording on the tensor cores
        dict(name="fir64_fp16x3_16m", kind="fir", taps=64, n=1 << 24, mode="fp16x3"),
        # tuning to four stations of one recording
        dict(name="shift4_4m", kind="shift", nch=4, n=1 << 22, dtype="c64"),
        # FM discriminator of a recording
        dict(name="polar_4m", kind="polar", n=1 << 22),
        # broadcast receiver: 1.14 MS/s in, int16 audio out, about a quarter of a second a call
        dict(name="fm_demod_256k", kind="fm", n=1 << 18, offset=150000),
    ]


def _log(rng, lo, hi):
    """A size between lo and hi, even over its logarithm; two in three odd."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, v | 1 if rng.random() < 0.67 else v)


def draw(rng):
    kind = rng.choice(["channelizer", "channelizer", "channelizer_tc", "channelizer_tc", "channelizer_host", "stream8",
                       "resample", "resample_long", "fir", "fir_tc", "shift", "polar", "fm"])
    if kind == "channelizer":
        return dict(kind="channelizer", signal="tones", nch=_log(rng, 1, 64), n=_log(rng, 1 << 12, 1 << 21),
                    mode="fp32", dtype=rng.choice(["c64", "c64", "ci16"]), plan=rng.randrange(1000), graph=False)
    if kind == "channelizer_tc":
        return dict(kind="channelizer", signal="tones", nch=_log(rng, 16, 256), n=_log(rng, 1 << 16, 1 << 24),
                    mode=rng.choice(["fp16x3", "bf16x3"]), dtype=rng.choice(["c64", "c64", "ci16"]),
                    plan=rng.randrange(1000), graph=rng.random() < 0.5)
    if kind == "stream8":
        return dict(kind="channelizer", signal="qpsk", nch=8, n=_log(rng, 1 << 12, 1 << 18), mode="fp32", dtype="c64",
                    plan=0, graph=rng.random() < 0.5)
    if kind == "channelizer_host":
        return dict(kind=kind, n=_log(rng, 1 << 12, 1 << 20), nch=8)
    if kind == "resample":
        up, down = rng.choice(RATIOS)
        return dict(kind=kind, up=up, down=down, tpp=rng.randint(12, 64), n=_log(rng, 1 << 12, 1 << 22),
                    mode=rng.choice(["fp32", "fp32", "fp16x3"]))
    if kind == "resample_long":
        return dict(kind="resample", up=1, down=10, tpp=_log(rng, 511, 4095), n=_log(rng, 1 << 16, 1 << 24),
                    mode=rng.choice(["fp32", "fp16x3", "bf16x3"]))
    if kind == "fir":
        return dict(kind=kind, taps=_log(rng, 8, 512), n=_log(rng, 1 << 12, 1 << 22), mode="fp32")
    if kind == "fir_tc":
        return dict(kind="fir", taps=_log(rng, 16, 512), n=_log(rng, 1 << 16, 1 << 24),
                    mode=rng.choice(["fp16x3", "bf16x3"]))
    if kind == "shift":
        return dict(kind=kind, nch=rng.randint(1, 8), n=_log(rng, 1 << 12, 1 << 24),
                    dtype=rng.choice(["c64", "c64", "ci16"]))
    if kind == "polar":
        return dict(kind=kind, n=_log(rng, 1 << 12, 1 << 24))
    return dict(kind="fm", n=_log(rng, 1 << 15, 1 << 20), offset=rng.choice([150000, -200000, 0]))


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _noise(n, seed, sigma=0.5):
    return torch.randn(n, dtype=torch.complex64, device=DEV, generator=_gen(seed)) * sigma


def _tones(n, fs, count, seed):
    """Sum of `count` tones + noise.  Synthesised on a power-of-two grid, as one inverse FFT."""
    return W.tone_signal(1 << max(n - 1, 1).bit_length(), fs, count, seed, device=DEV)[0][:n].contiguous()


def _wideband_fm(n, fs, seed, offset=0.0, snr_db=15.0):
    """A carrier at `offset` Hz, frequency modulated by 5 audio tones (75 kHz peak deviation), plus noise."""
    rng = np.random.default_rng(seed)
    tones, amps, ph = rng.uniform(50.0, 15000.0, 5), rng.uniform(0.3, 1.0, 5), rng.uniform(0, 2 * np.pi, 5)
    amps /= amps.sum()
    t = torch.arange(n, dtype=torch.float64, device=DEV) / fs
    phase = 2 * np.pi * offset * t
    for f, a, p in zip(tones, amps, ph):
        phase += 2 * np.pi * 75e3 * a / (2 * np.pi * f) * torch.sin(2 * np.pi * f * t + p)
    return (torch.polar(torch.ones_like(phase), phase).to(torch.complex64)
            + _noise(n, seed, 10 ** (-snr_db / 20))).contiguous()


def _to_ci16(x, scale):
    return torch.view_as_real(x * scale).round().clamp(-32768, 32767).to(torch.int16).contiguous()


def _lowpass(up, down, tpp):
    if tpp >= 511:  # the long channel filter: unit gain, 100 kHz cutoff at 2.4 MS/s
        m = np.arange(tpp) - (tpp - 1) / 2
        h = 2 * 100e3 / W.FM_FS * np.sinc(2 * 100e3 / W.FM_FS * m) * np.kaiser(tpp, 10.0)
        return h.astype(np.complex64)
    return W.kaiser_lowpass(up, down, tpp)


def _fir_taps(taps):
    g = np.random.default_rng(2030)
    return (0.1 / math.sqrt(2) * (g.standard_normal(taps) + 1j * g.standard_normal(taps))).astype(np.complex64)


def _shifts(nch):
    return [int(v) for v in np.random.default_rng(5).integers(-4500000, 4500000, nch)]


def _signal(case, seed):
    """(input on the GPU, sample rate, channels) of a channelizer case."""
    n = case["n"]
    if case.get("signal", "qpsk") == "qpsk":
        x, fs, chans = W.channelizer_8ch(n, seed)
        x = torch.from_numpy(x).to(DEV)
    else:
        fs, x = C3_FS, _tones(n, C3_FS, 512, seed)
        chans = W.channelizer_256_plan(float(fs), None, case["nch"], case["plan"])
    return (_to_ci16(x, 256.0) if case.get("dtype") == "ci16" else x), fs, chans


def _regions(chans, n):
    """Output regions of the channels in one buffer: [(first sample, samples)], and its size."""
    at, got = 0, []
    for ch in chans:
        cap = -(-n * ch["up_rate"] // ch["down_rate"]) + 1
        got.append((at, cap))
        at += (cap + 31) // 32 * 32
    return got, at


# ---- the calls -------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    k, n = case["kind"], case["n"]
    if k == "channelizer":
        x, fs, chans = _signal(case, seed)
        h = F.MultiRateChannelizerCuda(fs, chans)
        h.set_precision(case["mode"])
        h.set_graph(case["graph"])
        at, total = _regions(chans, n)
        buf = torch.zeros(total, dtype=torch.complex64, device=DEV)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        return dict(k=k, h=h, x=x, buf=buf, out=[buf[a:a + c] for a, c in at], s=s)
    if k == "channelizer_host":
        x, fs, chans = W.channelizer_8ch(n, seed)
        return dict(k=k, h=F.MultiRateChannelizerCuda(fs, chans), x=x)
    if k == "resample":
        x = _wideband_fm(n, W.FM_FS, seed) if case["tpp"] >= 511 else _tones(n, 48000.0, 3, seed)
        h = F.PolyphaseResamplerCuda(case["up"], case["down"], _lowpass(case["up"], case["down"], case["tpp"]))
        h.set_precision(case["mode"])
        return dict(k=k, h=h, x=x)
    if k == "fir":
        h = F.FirFilterCuda(_fir_taps(case["taps"]))
        h.set_precision(case["mode"])
        return dict(k=k, h=h, x=_noise(n, seed))
    if k == "shift":
        x = _tones(n, C2_FS, 16, seed)
        x = _to_ci16(x, 2048.0) if case["dtype"] == "ci16" else x
        return dict(k=k, h=F.FreqShiftCuda(C2_FS, _shifts(case["nch"])), x=x)
    if k == "polar":
        return dict(k=k, h=F.PolarDiscriminatorCuda(), x=_wideband_fm(n, W.FM_FS, seed))
    x = _wideband_fm(n, W.FM_RADIO_FS, seed, -case["offset"], 25.0)
    return dict(k=k, h=F.FmDemodulatorCuda(W.FM_RADIO_FS, case["offset"]), x=x)


def run(state):
    h, x = state["h"], state["x"]
    if state["k"] == "channelizer":
        h.apply(x, out=state["out"], stream=state["s"].cuda_stream)
        return state["buf"]
    if state["k"] == "fm":
        return h.demod_mono(x)
    return h.apply(x)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    k, n = case["kind"], case["n"]
    if k in ("channelizer", "channelizer_host"):
        if case.get("signal", "qpsk") == "qpsk":
            plan = [(u, d, 32) for u, d in W.C2_RATIOS]  # 16-48 taps a phase
        else:
            plan = [(c["up_rate"], c["down_rate"], len(c["coeffs"]) // c["up_rate"])
                    for c in W.channelizer_256_plan(float(C3_FS), None, case["nch"], case["plan"])]
        outs = [-(-n * u // d) for u, d, _ in plan]
        return dict(bytes=(4 if case.get("dtype") == "ci16" else 8) * n + 8 * sum(outs),
                    flops=sum(4 * t * m for (_, _, t), m in zip(plan, outs)) + 6 * sum(outs))
    if k == "resample":
        m = -(-n * case["up"] // case["down"])
        return dict(bytes=8 * n + 8 * m, flops=4 * case["tpp"] * m)
    if k == "fir":
        return dict(bytes=16 * n, flops=8 * case["taps"] * n)
    if k == "shift":
        return dict(bytes=(4 if case["dtype"] == "ci16" else 8) * n * (1 + case["nch"]), flops=6 * n * case["nch"])
    if k == "polar":
        return dict(bytes=12 * n, flops=6 * n)
    taps = 64  # two 64-tap filters, down by 5 and by 5 again
    return dict(bytes=8 * n + 2 * n // 25, flops=4 * taps * (n // 5 + n // 25) + 6 * n)


# ---- 64-bit results --------------------------------------------------------------------------------------------------
def _nco(fs, f, n):
    """e^{j 2 pi f/fs (i mod R)} for i in [0, n): R is fs/|f| times the least power of ten that makes it 1e5 or more."""
    r = fs / abs(f)
    while r < 1e5:
        r *= 10.0
    turns = (torch.arange(n, device=DEV) % int(round(r))) * (f % fs) % fs
    ang = turns.to(torch.float64) * (2 * math.pi / fs)
    return torch.polar(torch.ones_like(ang), ang)


def _polyphase(x, up, down, h, out):
    """The resampler's outputs of complex128 x into `out`; the taps' real parts, h[j up + phase]."""
    n, t = x.numel(), -(-len(h) // up)
    m = -(-n * up // down)
    xp = torch.cat([torch.zeros(t - 1, dtype=x.dtype, device=x.device), x])
    hr = np.zeros(t * up)
    hr[:len(h)] = np.real(h).astype(np.float64)
    for r in range(min(up, m)):
        rows = -(-(m - r) // up)
        first, ph = divmod(r * down, up)
        y = torch.zeros(rows, dtype=x.dtype, device=x.device)
        for j in range(t):
            a = t - 1 + first - j
            y.add_(xp[a:a + (rows - 1) * down + 1:down], alpha=float(hr[j * up + ph]))
        out[r:m:up] = y
    return m


def _c128(x):
    return (torch.view_as_complex(x.to(torch.float64)) if x.dtype == torch.int16 else x.to(torch.complex128))


def exact(case, seed):
    k, n = case["kind"], case["n"]
    if k == "channelizer":
        x, fs, chans = _signal(case, seed)
        x = _c128(x)
        at, total = _regions(chans, n)
        buf = torch.zeros(total, dtype=torch.complex128, device=DEV)
        for ch, (a, c) in zip(chans, at):
            f = ch["freq_shift_in_hz"]
            _polyphase(x * _nco(fs, f, n) if f else x, ch["up_rate"], ch["down_rate"], ch["coeffs"], buf[a:a + c])
        return buf
    if k == "channelizer_host":
        x, fs, chans = W.channelizer_8ch(n, seed)
        x = _c128(torch.from_numpy(x).to(DEV))
        got = []
        for ch in chans:
            y = torch.empty(-(-n * ch["up_rate"] // ch["down_rate"]), dtype=torch.complex128, device=DEV)
            f = ch["freq_shift_in_hz"]
            _polyphase(x * _nco(fs, f, n) if f else x, ch["up_rate"], ch["down_rate"], ch["coeffs"], y)
            got.append(y)
        return got
    if k == "resample":
        x = _c128(prepare(case, seed)["x"])
        y = torch.empty(-(-n * case["up"] // case["down"]), dtype=torch.complex128, device=DEV)
        _polyphase(x, case["up"], case["down"], _lowpass(case["up"], case["down"], case["tpp"]), y)
        return y
    if k == "fir":
        x = _c128(prepare(case, seed)["x"])
        y = torch.zeros(n, dtype=torch.complex128, device=DEV)
        for j, h in enumerate(_fir_taps(case["taps"])):
            if j < n:
                y[j:].add_(x[:n - j], alpha=complex(h))
        return y
    if k == "shift" and case["dtype"] == "c64":
        x = _c128(prepare(case, seed)["x"])
        return [x * _nco(C2_FS, f, n) if f else x for f in _shifts(case["nch"])]
    if k == "polar":
        x = _c128(prepare(case, seed)["x"])
        return torch.angle(x[1:] * torch.conj(x[:-1]))
    return None  # int16 samples: compared as whole numbers
