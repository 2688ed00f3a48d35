"""The group launchers: what they look up on every call and what they hold."""
import pytest
import torch
import torch.nn as nn

from glowq_b200.correction import patch_svd_correction_wrappers_cumulative
from glowq_b200.cuda_w4a16.linear import CudaW4A16Linear
from toy_model import ToyDecoder, make_artifacts


def patched(device="cpu", rank=16, seed=0, **sizes):
    model = ToyDecoder(seed=seed, **sizes)
    for layer in model.model.layers:
        for part in (layer.self_attn, layer.mlp):
            for name, lin in list(part.named_children()):
                setattr(part, name, CudaW4A16Linear.from_float(lin.to(device), 128))
    shared, bmap = make_artifacts(model, rank=rank)
    groups = {k.rsplit(".", 1)[0] for k in bmap.values()}
    return patch_svd_correction_wrappers_cumulative(model, shared, bmap, groups)


def forward(model, x, xi):
    return [model.proj(li, p)(xi if p.endswith("down_proj") else x) for li in range(2) for p in ToyDecoder.PROJ]


def inputs(m, hidden=256, inter=384, seed=3):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(m, c, generator=gen, device="cuda", dtype=torch.float16) for c in (hidden, inter)]


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 5, 20])
def test_left_factors_that_are_parameters(m):
    model, x = patched("cuda"), inputs(m)
    with torch.no_grad():
        want = [y.clone() for y in forward(model, *x)]
        for li in range(2):
            for p in ToyDecoder.PROJ:
                w = model.proj(li, p)
                t = w.A_q
                del w.A_q
                w.A_q = nn.Parameter(t, requires_grad=False)
        for y, z in zip(want, forward(model, *x)):
            assert torch.equal(y, z)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 5, 20, 70])
def test_factors_and_weights_that_move(m):
    """A right factor replaced (by a parameter, by other values) and a model that leaves the device and comes back: every call reads
    what is there now, and no launch names the places of before to the one in front of it."""
    model, x = patched("cuda"), inputs(m)
    other = patched("cuda", seed=5)
    dev = x[0].device
    with torch.no_grad():
        want = [y.clone() for y in forward(model, *x)]
        forward(model, *x)                                 # (with the hints of the pass before)
        launchers = [model.proj(li, p).group_launcher for li in range(2) for p in ("self_attn.q_proj", "mlp.down_proj")]
        assert all(g.descriptor_address(m, dev, torch.float32) for g in launchers)
        for g in launchers:
            t = g.members[0].B_q
            del g.members[0].B_q
            g.members[0].B_q = nn.Parameter(t.clone(), requires_grad=False)
            del t
        junk = [torch.full((64, 1024), 9.0, dtype=torch.float16, device="cuda") for _ in range(64)]     # over the old ones
        assert not any(g.descriptor_address(m, dev, torch.float32) for g in launchers)
        assert all(torch.equal(y, z) for y, z in zip(forward(model, *x), want))
        assert all(g.descriptor_address(m, dev, torch.float32) for g in launchers)
        model.cpu()
        assert not any(g.descriptor_address(m, dev, torch.float32) for g in launchers)
        del junk
        torch.cuda.empty_cache()
        keep = torch.empty(1 << 20, device="cuda")
        model.cuda()
        assert all(torch.equal(y, z) for y, z in zip(forward(model, *x), want))
        for li in range(2):
            for p in ToyDecoder.PROJ:
                new = other.proj(li, p).B_q * 2
                w = model.proj(li, p)
                w.B_q = nn.Parameter(new, requires_grad=False) if "B_q" in w._parameters else new
        assert not any(torch.equal(y, z) for y, z in zip(forward(model, *x), want))
        model.proj(0, "self_attn.o_proj").B_q = torch.zeros(8, 256, dtype=torch.float16, device="cuda")
        with pytest.raises(RuntimeError):
            forward(model, *x)
        del keep
