"""The discriminator streamed over blocks that end at, before and after a
block of its kernel (1024 outputs), down to one sample, against the oracle:
exact counts, angles within 2e-6 modulo 2 pi (a product whose imaginary part
rounds to the other side of zero turns +pi into -pi)."""
import numpy as np
import pytest

import libfalcon_dsp_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 1, 2, 1023, 1024, 1025), (1025, 1, 4096, 5), (70_001, 1024, 3)])
def test_streamed_blocks(sizes):
    import torch
    rng = np.random.default_rng(sum(sizes))
    g, o = F.PolarDiscriminatorCuda(), O.Polar()
    for n in sizes:
        x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
        a, b = g.apply(torch.from_numpy(x).cuda()).cpu().numpy(), o.apply(x)
        assert a.size == b.size
        np.testing.assert_allclose(np.angle(np.exp(1j * (a.astype(np.float64) - b))), 0, atol=2e-6)
