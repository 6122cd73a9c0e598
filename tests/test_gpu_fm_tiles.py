"""The FM demodulator's tiles: streamed blocks whose discriminator outputs end
at, before and after a tile of the de-emphasis kernel, blocks of one output,
and calls on either side of the one-cluster normalisation's limit, against the
oracle: exact counts, int16 audio within one count and 99.5 % equal (FP32 sums
in another order move a truncated value across an integer now and then)."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F
from libfalcon_dsp_gb300 import filter_design as FD
from libfalcon_dsp_gb300.workloads import FM_RADIO_FS, fm_station
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TILE = 1024  # discriminator outputs a block


@pytest.mark.parametrize("outs", [(1, 1, TILE - 1, TILE, TILE + 1), (TILE, 512, 2 * TILE, 31, 33), (700_000, 10_000)])
def test_audio_matches_the_oracle(outs):
    import torch
    t = FD.design_table()
    dem = F.FmDemodulatorCuda(FM_RADIO_FS, 150000)
    o = O.FmDemod(FM_RADIO_FS, 150000, t[(FM_RADIO_FS, 228000, 64, FD.REMEZ)], t[(228000, 45600, 64, FD.REMEZ)])
    x, _ = fm_station(5 * sum(outs), seed=17)
    at = 0
    for n in outs:
        b = x[at:at + 5 * n]
        at += 5 * n
        got, want = dem.demod_mono(torch.from_numpy(b).cuda()).cpu().numpy(), o.demod_mono(b)
        assert got.size == want.size
        if want.size:
            d = np.abs(got.astype(np.int32) - want.astype(np.int32))
            assert d.max() <= 1
            if want.size >= 200:
                assert np.mean(d == 0) >= 0.995
