"""Output buffers in the Python call path: what a handle keeps, what it
accepts and what it returns."""
import gc

import pytest

pytestmark = pytest.mark.gpu


def _channelizer():
    import libfalcon_dsp_gb300 as F
    from libfalcon_dsp_gb300.workloads import kaiser_lowpass
    return F.MultiRateChannelizerCuda(1_000_000, [
        {"freq_shift_in_hz": s, "up_rate": 1, "down_rate": 4, "coeffs": kaiser_lowpass(1, 4, 16)} for s in (0, 1000, -77)])


def _ci16(n):
    import torch
    return torch.randint(-1000, 1000, (n, 2), dtype=torch.int16, device="cuda")


@pytest.mark.parametrize("own", [False, True])
def test_int16_apply_keeps_no_output_memory(own):
    import torch
    h, x = _channelizer(), _ci16(1 << 20)
    h.apply(x)
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    out = [torch.empty((1 << 18) + 1, dtype=torch.complex64, device="cuda") for _ in range(3)] if own else None
    res = h.apply(x, out=out)
    assert [r.numel() for r in res] == [1 << 18] * 3 and torch.cuda.memory_allocated() > before
    del res, out
    gc.collect()
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() <= before


class _Buffer:
    """A device buffer that is no tensor: an address and a size."""

    def __init__(self, n):
        import torch
        self.t = torch.zeros(n, dtype=torch.complex64, device="cuda")

    def data_ptr(self):
        return self.t.data_ptr()

    def numel(self):
        return self.t.numel()

    def __getitem__(self, i):
        return self.t[i]


@pytest.mark.parametrize("dtype", ["c64", "ci16"])
def test_outputs_may_be_any_object_with_an_address_and_a_size(dtype):
    import torch
    x = _ci16(4096) if dtype == "ci16" else torch.randn(4096, dtype=torch.complex64, device="cuda")
    want = _channelizer().apply(x)
    got = _channelizer().apply(x, out=[_Buffer(1030) for _ in range(3)])
    for a, b in zip(got, want):
        assert torch.equal(a, b)
