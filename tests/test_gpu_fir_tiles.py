"""Long-block FIR and integer decimation of one channel (the sliding-window
form whose outputs leave through shared memory): block lengths around whole
tiles of 1792 rows, real and complex taps, streamed, against the FP32 oracle
within 1e-5 relative RMS with exact counts.  An infinite sample marks the
outputs of its window and no others."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F
from oracle import oracle as O
from tests.golden_io import rel_rms

pytestmark = pytest.mark.gpu

TILE = 1792


def _x(rng, n):
    return ((rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 0.5).astype(np.complex64)


@pytest.mark.parametrize("taps", [16, 64, 257])
@pytest.mark.parametrize("tail", [-1, 0, 1])
def test_fir(taps, tail):
    import torch
    rng = np.random.default_rng(taps + tail)
    h = ((rng.standard_normal(taps) + 1j * rng.standard_normal(taps)) / np.sqrt(2 * taps)).astype(np.complex64)
    f, o = F.FirFilterCuda(h), O.FIR(h)
    for n in (TILE * 160 + tail, TILE * 153 + 7):
        x = _x(rng, n)
        assert rel_rms(f.apply(torch.from_numpy(x).cuda()).cpu().numpy(), o.apply(x)) <= 1e-5


@pytest.mark.parametrize("down,taps", [(2, 33), (5, 64), (7, 16)])
def test_decimator(down, taps):
    import torch
    rng = np.random.default_rng(down)
    h = (rng.standard_normal(taps) / np.sqrt(taps)).astype(np.complex64)
    f, o = F.PolyphaseResamplerCuda(1, down, h), O.Resampler(1, down, h)
    for n in (TILE * 155 * down + 1, TILE * 200 * down - 3):
        x = _x(rng, n)
        y, r = f.apply(torch.from_numpy(x).cuda()).cpu().numpy(), o.apply(x)
        assert y.size == r.size and rel_rms(y, r) <= 1e-5


@pytest.mark.parametrize("up,down,tpp", [(3, 2, 60), (2, 5, 17), (7, 8, 33), (5, 3, 16)])
def test_rational(up, down, tpp):
    """The few-phase rates: every phase of a tile's rows leaves together."""
    import torch
    rng = np.random.default_rng(up * 10 + down)
    h = (rng.standard_normal(up * tpp) / np.sqrt(tpp)).astype(np.complex64)
    f, o = F.PolyphaseResamplerCuda(up, down, h), O.Resampler(up, down, h)
    for n in (TILE * 160 * down + 1, TILE * 155 * down - 1, TILE * 170 * down + 2):
        x = _x(rng, n)
        y, r = f.apply(torch.from_numpy(x).cuda()).cpu().numpy(), o.apply(x)
        assert y.size == r.size and rel_rms(y, r) <= 1e-5


def test_infinite_sample_marks_its_window():
    import torch
    n, taps = TILE * 160, 64
    h = (np.random.default_rng(4).standard_normal(taps) + 0.5).astype(np.complex64) * (1 + 1j)
    x = np.ones(n, np.complex64)
    x[5000] = complex(np.inf, 1.0)
    y = F.FirFilterCuda(h).apply(torch.from_numpy(x).cuda()).cpu().numpy()
    hit = np.zeros(n, bool)
    hit[5000:5000 + taps] = True
    assert not np.any(np.isfinite(y.real[hit])) and np.all(np.isfinite(y[~hit]))
