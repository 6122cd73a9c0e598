"""The sliding-window form of one unshifted real-tap channel: three CTAs an SM
(tiles that leave room, few phases) and two with the taps read ahead, one phase
and several, two blocks each, outputs all over the stream against 64-bit sums
within 1e-5 relative RMS, and a shifted channel's beside them."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F
from tests.test_gpu_long_rows import FS, _check_outputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f", [0, 1234567])
@pytest.mark.parametrize("u,d,t,n", [(1, 1, 17, 1 << 20), (1, 1, 1000, 1 << 20), (1, 1, 8000, 1 << 19),
                                     (1, 4, 3000, 1 << 21), (1, 10, 500, 1 << 22), (1, 10, 4500, 1 << 22),
                                     (3, 2, 60, 1 << 20), (2, 5, 2000, 1 << 21), (1, 25, 700, 1 << 23)])
def test_outputs_match_64_bit_sums(u, d, t, n, f):
    import torch
    rng = np.random.default_rng(t)
    h = (rng.standard_normal(u * t) / np.sqrt(t)).astype(np.float32)
    c = F.MultiRateChannelizerCuda(FS, [dict(freq_shift_in_hz=f, up_rate=u, down_rate=d, coeffs=h.astype(np.complex64))])
    x = (rng.integers(-2000, 2000, n) + 1j * rng.integers(-2000, 2000, n)).astype(np.complex64)
    cut = n * 11 // 16 | 1
    y = torch.cat([c.apply(torch.from_numpy(v).cuda())[0].clone() for v in (x[:cut], x[cut:])]).cpu().numpy()
    assert y.size == -(-n * u // d)
    _check_outputs(rng, x, f, u, d, t, h.astype(np.float64), y)
