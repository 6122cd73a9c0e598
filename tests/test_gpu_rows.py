"""The FP32 kernel's tiles: staged phases (all of them, the windows' runs
alone, more runs than a tile can hold), rows a thread, channels a batch, and
tile heights of short and long blocks, each streamed over three blocks against
the FP32 oracle within 1e-5 relative RMS with exact counts.  Float and int16
input."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F
from oracle import oracle as O
from tests.golden_io import rel_rms

pytestmark = pytest.mark.gpu

# (up, down, taps a phase) of the channels; one decimation group each unless named
PLANS = {
    "one_run": [(1, 320, 40)],
    "three_runs": [(3, 320, 33), (3, 320, 20), (1, 320, 64)],
    "two_runs_odd": [(2, 625, 48)],
    "touching_runs": [(3, 160, 50), (3, 160, 54)],
    "too_many_runs": [(7, 600, 8), (1, 600, 30)],
    "dense": [(3, 8, 37)] * 9 + [(1, 8, 12)] * 5,
    "dense_long_taps": [(1, 20, 130), (1, 20, 3)],
    "uneven_groups": [(1, 4, 64), (3, 25, 17), (1, 320, 12), (2, 125, 64), (1, 64, 33), (1, 1, 5)],
    "one_tap": [(1, 50, 1), (7, 50, 1)],
}


# more work sets than a launch holds in batches of four channels: batches of eight
PLANS["wide_batches"] = [(9, 20, 5)] * 199 + [(9, 20, 12)]


@pytest.mark.parametrize("sizes", [(1, 31, 4099), (70001, 5, 65536), (1 << 20, 999983, 77)])
@pytest.mark.parametrize("plan", sorted(PLANS))
def test_tiles_match_the_oracle(plan, sizes):
    import torch
    if plan == "wide_batches":
        sizes = [min(n, 20011) for n in sizes]  # 200 channels
    rng = np.random.default_rng(len(plan) * 1000 + sizes[0])
    fs = 10_000_000
    chans = []
    for i, (u, d, t) in enumerate(PLANS[plan]):
        h = (rng.standard_normal(u * t) / np.sqrt(t)).astype(np.complex64)
        f = 0 if i % 4 == 3 else int(rng.integers(-fs // 2, fs // 2)) or 1
        chans.append(dict(freq_shift_in_hz=f, up_rate=u, down_rate=d, coeffs=h))
    a, b = F.MultiRateChannelizerCuda(fs, chans), F.MultiRateChannelizerCuda(fs, chans)
    ref = O.Channelizer(fs, chans)
    for n in sizes:
        x16 = rng.integers(-2000, 2000, size=(n, 2)).astype(np.int16)
        x = (x16[:, 0] + 1j * x16[:, 1]).astype(np.complex64)
        ya = [y.cpu().numpy() for y in a.apply(torch.from_numpy(x).cuda())]
        yb = [y.cpu().numpy() for y in b.apply(torch.from_numpy(x16).cuda())]
        for p, q, r in zip(ya, yb, ref.apply(x)):
            assert p.size == q.size == r.size
            assert np.array_equal(p, q)  # the conversion is exact
            if r.size >= 32:
                assert rel_rms(p, r) <= 1e-5
            elif r.size:
                assert np.max(np.abs(p - r)) <= 1e-5 * 2000 * 8
