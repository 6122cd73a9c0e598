"""A tensor-core call whose work does not fit 32 bits of item cost (24000 taps
over 2^30 samples): every output is written, and outputs all over the block,
its ends included, agree with 64-bit sums.

Bound: 60 dB, as for shorter filters (tests/test_gpu_tc_fir.py); FP32 sums of
24000 products are off by about sqrt(24000) 2^-24, 100 dB."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TAPS, N = 24000, 1 << 30


def test_every_item_runs():
    import torch

    import libfalcon_dsp_gb300 as F
    if torch.cuda.mem_get_info()[0] < 48 << 30:
        pytest.skip("needs 48 GB of device memory")
    rng = np.random.default_rng(11)
    h = ((rng.standard_normal(TAPS) + 1j * rng.standard_normal(TAPS)) * 0.01).astype(np.complex64)
    x = torch.randn(N, dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    y = torch.full((N,), float("nan"), dtype=torch.complex64, device="cuda")
    f = F.FirFilterCuda(h)
    f.set_precision("fp16x3")
    got = f.apply(x, out=y)
    torch.cuda.synchronize()
    assert f.tc_groups() == 1 and got.numel() == N
    f.status()
    for part in y.split(1 << 27):
        assert not torch.isnan(torch.view_as_real(part)).any()
    g = torch.from_numpy(h[::-1].astype(np.complex128)).cuda()
    at = sorted({0, TAPS - 1, N - 1} | {int(v) for v in rng.integers(0, N, 200)} |
                {k * (N // 152) + j for k in range(1, 152, 10) for j in (-1, 0)})
    err = ref2 = 0.0
    for i in at:
        w = x[max(0, i - TAPS + 1):i + 1].to(torch.complex128)
        ref = complex((w * g[TAPS - w.numel():]).sum())
        err += abs(complex(y[i]) - ref) ** 2
        ref2 += abs(ref) ** 2
    assert 10 * np.log10(ref2 / err) >= 60.0
