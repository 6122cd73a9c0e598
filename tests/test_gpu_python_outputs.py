"""Output buffers in the Python call path: what a handle keeps, what it
accepts and what it returns."""
import gc

import numpy as np
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
    for _ in range(3):
        res = h.apply(x, out=out)
    assert [r.numel() for r in res] == [1 << 18] * 3 and torch.cuda.memory_allocated() > before
    del res, out
    gc.collect()
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() <= before


def test_int16_results_follow_the_callers_buffers():
    import torch
    x, want = _ci16(4001), []
    h, f = _channelizer(), _channelizer()
    for _ in range(9):  # counts of 1000 and 1001, new buffers after three calls, other ones over the same memory
        want.append([y.clone() for y in f.apply(x)])
    mem = [torch.zeros(2 * 1040, dtype=torch.complex64, device="cuda") for _ in range(3)]
    sets = [[m[:1024] for m in mem], [m[5:1030] for m in mem], [m[:1024] for m in mem]]
    for k in range(9):
        out = sets[k // 3]
        for m in mem:
            m.zero_()
        got = h.apply(x, out=out)
        for a, b, o in zip(got, want[k], out):
            assert torch.equal(a, b) and a.data_ptr() == o.data_ptr() and torch.equal(o[:a.numel()], b)
    kept = h.apply(x, out=sets[2])
    again = [t.clone() for t in kept]
    del sets, out, mem, got
    gc.collect()
    torch.randn(1 << 16, device="cuda")  # (the results keep their memory when the buffers go)
    assert all(torch.equal(a, b) for a, b in zip(kept, again))


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


def _calls():
    import torch

    import libfalcon_dsp_gb300 as F
    from libfalcon_dsp_gb300.workloads import FM_RADIO_FS, kaiser_lowpass
    n = 1000
    c = torch.randn(n, dtype=torch.complex64, device="cuda")
    c64 = lambda k: torch.empty(k, dtype=torch.complex64, device="cuda")  # noqa: E731
    i16 = lambda k: torch.empty((k, 2), dtype=torch.int16, device="cuda")  # noqa: E731
    r = F.PolyphaseResamplerCuda(1, 4, kaiser_lowpass(1, 4, 16))
    p = F.PolarDiscriminatorCuda()
    p.apply(c)
    taps = np.ones(8, np.complex64)
    d = F.FmDemodulatorCuda(FM_RADIO_FS, 150000)
    fm = torch.randn(100_000, dtype=torch.complex64, device="cuda")
    k = F.FmDemodulatorCuda(FM_RADIO_FS, 150000).demod_mono(fm).numel()
    audio = torch.empty(k, dtype=torch.int16, device="cuda")
    yield (lambda o: r.apply(c, out=o)), c64(250)
    yield (lambda o: F.FirFilterCuda(taps).apply(c, out=o)), c64(n)
    yield (lambda o: F.FirFilterCuda(taps).apply(_ci16(n), out=o)), i16(n)
    yield (lambda o: F.FreqShiftCuda(1_000_000, 1000).apply(c, out=[o])), c64(n)
    yield (lambda o: F.FreqShiftCuda(1_000_000, 1000).apply(_ci16(n), out=[o])), i16(n)
    yield (lambda o: p.apply(c, out=o)), torch.empty(n, dtype=torch.float32, device="cuda")
    yield (lambda o: d.demod_mono(fm, out=o)), audio


def test_a_full_output_is_a_view_of_the_callers_buffer():
    for call, out in _calls():
        shape = tuple(out.shape)
        y = call(out)
        assert tuple(y.shape) == shape and y.data_ptr() == out.data_ptr() and y is not out
        y.resize_(1)  # (of the result alone)
        assert tuple(out.shape) == shape
