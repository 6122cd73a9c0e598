"""Rational resampling by many phases (the many-phase kernel, and the rates
beside its rule that keep the row form), streamed over blocks with every
starting phase, one output a thread and full tiles, float and int16, against
the FP32 oracle: exact counts and state, 1e-5 relative RMS.  An infinite
sample marks the outputs of its window in both parts and no others."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F
from oracle import oracle as O
from tests.golden_io import rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("up,down,tpp", [(147, 160, 24), (160, 147, 13), (16, 63, 512), (16, 1, 3), (17, 70, 9),
                                         (15, 16, 30), (24, 26, 20), (255, 256, 32), (255, 256, 33), (31, 124, 1)])
@pytest.mark.parametrize("sizes", [(1, 2, 161, 4097), (400_003, 3, 65536)])
def test_streamed_blocks(up, down, tpp, sizes):
    import torch
    rng = np.random.default_rng(up * 1000 + down)
    h = (rng.standard_normal(up * tpp - (tpp > 1)) / np.sqrt(tpp)).astype(np.complex64)  # a ragged last tap row
    a, b, o = F.PolyphaseResamplerCuda(up, down, h), F.PolyphaseResamplerCuda(up, down, h), O.Resampler(up, down, h)
    for n in sizes:
        x16 = rng.integers(-2000, 2000, size=(n, 2)).astype(np.int16)
        x = (x16[:, 0] + 1j * x16[:, 1]).astype(np.complex64)
        p = a.apply(torch.from_numpy(x).cuda()).cpu().numpy()
        q = b.apply(torch.from_numpy(x16).cuda()).cpu().numpy()
        r = o.apply(x)
        assert p.size == q.size == r.size and a.state() == b.state()
        assert np.array_equal(p, q)
        if r.size >= 32:
            assert rel_rms(p, r) <= 1e-5
        elif r.size:
            assert np.max(np.abs(p - r)) <= 1e-5 * 2000 * 8


def test_infinite_sample_marks_its_windows():
    import torch
    up, down, tpp = 147, 160, 24
    h = np.random.default_rng(3).standard_normal(up * tpp).astype(np.complex64)
    x = np.ones(5000, np.complex64)
    x[1000] = complex(np.inf, 0.0)
    y = F.PolyphaseResamplerCuda(up, down, h).apply(torch.from_numpy(x).cuda()).cpu().numpy()
    i = np.arange(y.size) * down // up
    hit = (i >= 1000) & (i < 1000 + tpp)
    assert np.all(~np.isfinite(y.real[hit])) and np.all(np.isnan(y.imag[hit]))
    assert np.all(np.isfinite(y.real[~hit])) and np.all(np.isfinite(y.imag[~hit]))
