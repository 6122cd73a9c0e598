"""The discriminator's state under capture: one apply captured in the caller's
CUDA graph and replayed block after block carries x[-1] from replay to replay,
as direct applies do (angles equal bit for bit), and hands it back to them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 1024, 5000])
def test_replays_carry_the_last_sample(n):
    import torch

    import libfalcon_dsp_gb300 as F
    rng = np.random.default_rng(n)
    blocks = [torch.from_numpy((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)).cuda()
              for _ in range(6)]
    direct = F.PolarDiscriminatorCuda()
    want = [direct.apply(b).clone() for b in blocks]

    p = F.PolarDiscriminatorCuda()
    p.apply(blocks[0])
    x, y = torch.empty_like(blocks[0]), torch.empty(n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        p.apply(x, out=y)
    for k in range(1, 5):
        x.copy_(blocks[k])
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want[k]), k
    assert torch.equal(p.apply(blocks[5]), want[5])
