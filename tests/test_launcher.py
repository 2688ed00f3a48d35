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
