"""The FP32 kernel's row form over filters of every length: taps packed or
compact in shared memory or read through L1, windows walked tap by tap or run
by run, one to four rows a thread, batches of up to eight channels, and the
exact path of windows across the NCO rollover.  Two blocks each, float and
int16 input, outputs all over the stream and at its rollovers against 64-bit
sums: 1e-5 relative RMS (FP32 sums of T products are off by about sqrt(T)
2^-24, 6e-6 for the longest)."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F

pytestmark = pytest.mark.gpu

FS = 10_005_500

CASES = [  # channels, up, down, taps a phase, samples
    (2, 1, 1, 9700, 1 << 18), (1, 1, 1, 9700, 200_003), (3, 1, 10, 9000, 1 << 18), (3, 1, 100, 9000, 1 << 19),
    (4, 1, 10, 2500, 1 << 19), (8, 1, 10, 800, 1 << 19), (2, 1, 4, 4000, 1 << 18), (4, 1, 1, 700, 1 << 18),
    (2, 5, 8, 900, 1 << 18), (5, 1, 3, 64, 1 << 18), (2, 1, 2, 40, 300_001), (6, 2, 5, 33, 1 << 18),
    (7, 1, 5, 20, 1 << 18), (2, 3, 1, 50, 250_001), (4, 1, 25, 200, 1 << 20), (1, 1, 6, 300, 1 << 19),
    (16, 70, 33, 16, 250_001), (16, 70, 33, 40, 250_001),
]


def _shifts(rng, nch, taps, n):
    """Shifts whose counters roll over in n samples (every fourth channel: none)."""
    got = []
    for c in range(nch):
        f = 0
        while c % 4 != 3 and not (f and taps < F.freq_shift_params(FS, f)[0] < n):  # (rollovers: 1e5 to 1e6 samples)
            f = int(rng.integers(-FS // 2, FS // 2))
        got.append(f)
    return got


def _shifted(x, f):
    if f == 0:
        return x.astype(np.complex128)
    r, w = F.freq_shift_params(FS, f)
    return x * np.exp(1j * w * (np.arange(x.size) % r))


def _check_outputs(rng, x, f, u, d, t, h, y):
    xs = np.concatenate([np.zeros(t, np.complex128), _shifted(x, f)])
    m = set(rng.integers(0, y.size, 150).tolist()) | {0, y.size - 1}
    if f:
        r = F.freq_shift_params(FS, f)[0]
        for k in range(r, x.size, r):
            m |= {(k + int(j)) * u // d for j in rng.integers(-2, t + 2, 12)}
    m = np.array(sorted(v for v in m if 0 <= v < y.size))
    ref = np.array([np.dot(h[(v * d) % u::u][:t][::-1], xs[(v * d) // u + 1:(v * d) // u + 1 + t]) for v in m])
    err = np.sqrt(np.sum(np.abs(y[m] - ref) ** 2) / np.sum(np.abs(ref) ** 2))
    assert err <= 1e-5, (f, err)


@pytest.mark.parametrize("nch,u,d,t,n", CASES)
def test_outputs_match_64_bit_sums(nch, u, d, t, n):
    import torch
    rng = np.random.default_rng(nch * 1000 + u * 100 + d * 10 + t)
    h = [(rng.standard_normal(u * t) / np.sqrt(t)).astype(np.float32) for _ in range(nch)]
    f = _shifts(rng, nch, t, n)
    chans = [dict(freq_shift_in_hz=f[c], up_rate=u, down_rate=d, coeffs=h[c].astype(np.complex64)) for c in range(nch)]
    x16 = rng.integers(-2000, 2000, size=(n, 2)).astype(np.int16)
    x = (x16[:, 0] + 1j * x16[:, 1]).astype(np.complex64)
    a, b = F.MultiRateChannelizerCuda(FS, chans), F.MultiRateChannelizerCuda(FS, chans)
    cut = n * 5 // 8 | 1
    ya = [a.apply(torch.from_numpy(v).cuda()) for v in (x[:cut], x[cut:])]
    yb = [b.apply(torch.from_numpy(v).cuda()) for v in (x16[:cut], x16[cut:])]
    for c in range(nch):
        y = torch.cat([ya[0][c], ya[1][c]]).cpu().numpy()
        assert np.array_equal(y, torch.cat([yb[0][c], yb[1][c]]).cpu().numpy())  # the conversion is exact
        assert y.size == -(-n * u // d)
        _check_outputs(rng, x, f[c], u, d, t, h[c].astype(np.float64), y)


def _time(nch, d, t, n):
    import torch
    rng = np.random.default_rng(t)
    chans = [dict(freq_shift_in_hz=s, up_rate=1, down_rate=d, coeffs=(rng.standard_normal(t) / t).astype(np.complex64))
             for s in [1_000_001 + 100_001 * c for c in range(nch)]]
    h = F.MultiRateChannelizerCuda(FS, chans)
    x = torch.randn(n, dtype=torch.complex64, device="cuda")
    out = [torch.empty(n // d + 8, dtype=torch.complex64, device="cuda") for _ in range(nch)]
    best = 1e30
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        h.apply(x, out=out)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("nch,d,short,long,n,slack", [
    (2, 1, 4600, 9700, 1 << 19, 3.5),    # tiles of 32 rows under a halo of 9699 samples took 18 times as long
    (2, 1, 3000, 5500, 1 << 19, 3.5),
    (4, 10, 1250, 2500, 1 << 21, 1.5),   # taps of twice the size no longer fitted shared memory: 4 times as long
    (8, 10, 600, 1200, 1 << 21, 1.5),
])
def test_time_grows_with_the_taps(nch, d, short, long, n, slack):
    # taps that leave room for one CTA fewer on an SM may cost some more, not several times the work
    assert _time(nch, d, long, n) <= slack * long / short * _time(nch, d, short, n)
