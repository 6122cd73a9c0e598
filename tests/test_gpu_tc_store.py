"""Every way the tensor-core epilogue stores a row (whole rows of 3, 5, 6 and
7 outputs through shared memory, 32-byte and 16-byte pieces, single outputs),
with row counts around a block of 32 rows and a tile, outputs at addresses
that are and are not 16 or 32 bytes aligned, streamed over blocks, against the
FP32 form at 100 dB (the split form's floor on such plans is 113 dB)."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ups,down", [((3, 1), 8), ((3, 3, 3, 1), 16), ((5, 1, 2), 12), ((7, 1), 40), ((6, 2, 6), 25),
                                      ((4, 4, 2), 9), ((8, 3), 35), ((9, 2), 20)])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_store_forms(ups, down, offset):
    import torch
    rng = np.random.default_rng(down * 10 + offset)
    fs = 10_000_000
    chans = [dict(freq_shift_in_hz=int(rng.integers(-fs // 2, fs // 2)) if i else 0, up_rate=u, down_rate=down,
                  coeffs=(rng.standard_normal(u * 20) / np.sqrt(20)).astype(np.complex64)) for i, u in enumerate(ups)]
    a, b = F.MultiRateChannelizerCuda(fs, chans), F.MultiRateChannelizerCuda(fs, chans)
    b.set_precision("fp16x3")
    for n in (31 * down, 128 * down + 1, 70_001, 300_007):
        x = torch.from_numpy(((rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 0.5).astype(np.complex64)).cuda()
        want = a.apply(x)
        bufs = [torch.full((w.numel() + offset + 8,), 7.0, dtype=torch.complex64, device="cuda") for w in want]
        got = b.apply(x, out=[q[offset:offset + w.numel()] for q, w in zip(bufs, want)])
        b.status()
        assert b.tc_groups() == 1
        for g, w, q in zip(got, want, bufs):
            assert g.numel() == w.numel()
            err = (g - w).abs().double().square().sum().item()
            assert err <= 1e-10 * w.abs().double().square().sum().item()
            assert bool((q[:offset] == 7).all()) and bool((q[offset + w.numel():] == 7).all())
