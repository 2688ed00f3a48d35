"""The one-launch quantiser against the torch expression it stands for: the same bits for every weight."""
import pytest
import torch

from glowq_b200.cuda_w4a16 import linear as L

pytestmark = pytest.mark.gpu


def _both(w, monkeypatch):
    assert L._kernel_quantises(w, 128)
    got = L._quantize_per_group_w4(w, 128)
    with monkeypatch.context() as m:
        m.setattr(L, "_kernel_quantises", lambda *_: False)
        want = L._quantize_per_group_w4(w, 128)
    assert got[3] == want[3]
    for name, a, b in zip(("qweight", "qzeros", "scales"), got, want):
        assert a.shape == b.shape and a.dtype == b.dtype and a.is_contiguous(), name
        view = (lambda t: t.view(torch.int16)) if a.dtype == torch.float16 else (lambda t: t)
        assert torch.equal(view(a), view(b)), name


# one group, ragged and odd column counts (scalar loads), 7 / 8 / 9 groups around a zero-point word, a partial last block
@pytest.mark.parametrize("oc,ic", [(1, 128), (1, 1), (3, 200), (5, 1032), (7, 130), (9, 896), (8, 1024), (33, 1152), (17, 2047)])
def test_bits_match_the_torch_expression(oc, ic, monkeypatch):
    gen = torch.Generator(device="cuda").manual_seed(oc * 10007 + ic)
    _both(torch.randn(oc, ic, generator=gen, device="cuda", dtype=torch.float16) * 0.02, monkeypatch)


def test_strided_and_misaligned_rows(monkeypatch):
    base = torch.randn(8, 1100, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda", dtype=torch.float16)
    for w in (base[:, :1024], base[:, 8:1032], base[:, 3:1027], base[::2, 1:]):
        _both(w, monkeypatch)


def test_every_exponent_and_the_special_groups(monkeypatch):
    """Groups of any spread (scales from the smallest subnormal to the largest, and beyond: max - min overflows), constant
    and all-zero groups of both signs (scale 0), infinities and NaN."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    bits = torch.randint(-32768, 32768, (2048, 1024), generator=gen, device="cuda", dtype=torch.int32).to(torch.int16)
    exp = torch.randint(0, 31, (2048, 8), generator=gen, device="cuda", dtype=torch.int32).repeat_interleave(128, 1)
    spread = torch.minimum((bits.to(torch.int32) >> 10) & 31, exp)        # a group's exponents up to a bound of its own
    w = ((bits.to(torch.int32) & 0x83FF) | (spread << 10)).to(torch.int16).view(torch.float16).clone()
    w[0, :128], w[0, 128:256], w[0, 256:384], w[0, 384:512] = 0.0, -0.0, 3.0, -3.0
    w[1, 5], w[1, 130], w[1, 260], w[1, 384:512] = float("inf"), float("-inf"), float("nan"), float("inf")
    w[2, :128] = 65504.0
    w[2, 0] = -65504.0
    w[3, :128] = 5.960464477539063e-08
    w[3, 7] = 0.0
    _both(w, monkeypatch)


def test_from_float_keeps_everything_on_the_weights_device():
    lin = torch.nn.Linear(200, 24, bias=True, device="cuda", dtype=torch.float16)
    mod = L.CudaW4A16Linear.from_float(lin, 128)
    assert {t.device.type for t in list(mod.buffers()) + list(mod.parameters())} == {"cuda"}
    assert mod.qweight_i32.shape == (24, 32) and mod.gid.shape == (200,) and torch.equal(mod.bias.data, lin.bias.data)
    assert set(mod.state_dict()) == {"qweight_i32", "qzeros_i32", "scales_f16", "bias"}


def test_from_float_without_a_library(monkeypatch):
    lin = torch.nn.Linear(300, 40, bias=False, device="cuda", dtype=torch.float16)
    want = L.CudaW4A16Linear.from_float(lin, 128)

    def missing():
        raise RuntimeError("failed to load libglowq_w4a16.so")

    monkeypatch.setattr(L, "load_w4a16_extension", missing)
    got = L.CudaW4A16Linear.from_float(lin, 128)
    for name, t in want.state_dict().items():
        assert torch.equal(got.state_dict()[name], t), name


class _Sub(L.CudaW4A16Linear):
    """A subclass goes through its constructor: buffers of its own, replaced and moved."""


@pytest.mark.parametrize("oc,ic,bias", [(1, 1, True), (3, 128, False), (24, 200, True), (7, 1032, True), (40, 2047, False), (9, 5000, False)])
def test_a_conversion_makes_the_module_that_the_constructor_makes(oc, ic, bias):
    lin = torch.nn.Linear(ic, oc, bias=bias, device="cuda", dtype=torch.float16)
    got, want = L.CudaW4A16Linear.from_float(lin, 128), _Sub.from_float(lin, 128)
    assert [n for n, _ in got.named_buffers()] == [n for n, _ in want.named_buffers()]
    for (n, a), (_, b) in zip(got.named_buffers(), want.named_buffers()):
        assert a.dtype == b.dtype and a.device == b.device and a.stride() == b.stride() and torch.equal(a, b), n
    assert set(got.state_dict()) == set(want.state_dict()) and (got.bias is None) == (want.bias is None) == (not bias)
    assert not bias or torch.equal(got.bias, want.bias) and got.bias.requires_grad == want.bias.requires_grad
    x = torch.randn(3, ic, device="cuda", dtype=torch.float16)
    assert ic % 8 or torch.equal(got(x), want(x))
