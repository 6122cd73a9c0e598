"""Resamplers around the most output phases a launch's work sets hold (256):
256 phases stream any block; above, a block of at most 256 outputs is computed
(against the oracle, 1e-5 relative RMS) and a longer one is refused."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F
from libfalcon_dsp_gb300 import _capi
from oracle import oracle as O
from tests.golden_io import rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("up,down", [(255, 256), (256, 255), (257, 256), (401, 400), (512, 511)])
def test_phases_at_the_limit(up, down):
    import torch
    rng = np.random.default_rng(up)
    h = (rng.standard_normal(12 * up) / 3).astype(np.complex64)
    r, o = F.PolyphaseResamplerCuda(up, down, h), O.Resampler(up, down, h)
    for n in (200, 250, 50, 4000):
        x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
        if up > 256 and r.out_count(n) > 256:
            with pytest.raises(F.FdspError) as e:
                r.apply(torch.from_numpy(x).cuda())
            assert _capi.STATUS[e.value.status] == "FDSP_ERR_UNSUPPORTED"
            continue
        y, want = r.apply(torch.from_numpy(x).cuda()).cpu().numpy(), o.apply(x)
        assert y.size == want.size and rel_rms(y, want) <= 1e-5
