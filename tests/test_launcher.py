"""The group launchers: what they look up on every call and what they hold."""
import copy
import gc
import pickle
import weakref
from types import SimpleNamespace

import pytest
import torch
import torch.nn as nn

from glowq_b200.correction import MiniGroupCache, patch_svd_correction_wrappers_cumulative
from glowq_b200.cuda_w4a16 import kernels as K
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


def pieces(launcher):
    scratch = getattr(launcher, "_scratch", None)
    return [] if scratch is None else list(scratch._pieces.values()) + scratch._kept


@pytest.mark.gpu
def test_token_counts_share_a_piece():
    """Prompts of many lengths, decode in between: one piece a launcher, of the largest call's size, and results without a history."""
    model = patched("cuda")
    x = {m: inputs(m, seed=m) for m in (1, 3, 8, 20, 64, 70, 257, 300, 411, 700)}
    with torch.no_grad():
        want = {m: forward(patched("cuda"), *x[m]) for m in x}
        for m in (700, 1, 8, 300, 3, 64, 20, 411, 1, 257, 70, 8, 700, 1):
            assert all(torch.equal(y, z) for y, z in zip(forward(model, *x[m]), want[m])), m
    for li in range(2):
        for p in ("self_attn.q_proj", "self_attn.o_proj", "mlp.gate_proj", "mlp.down_proj"):
            (piece,) = pieces(model.proj(li, p).group_launcher)
            assert piece.numel() < 18 << 20


def test_a_dropped_model_is_gone_at_once():
    gc.collect()
    gc.disable()
    try:
        model = patched()
        refs = [weakref.ref(o) for li in range(2) for p in ToyDecoder.PROJ for w in [model.proj(li, p)]
                for o in (w, w.inner, w.group_launcher, w.inner.qweight_i32)]
        part = model.proj(0, "self_attn.k_proj")
        launcher = part.group_launcher
        del model
        alive = [r() for r in refs if r() is not None]
        assert {id(o) for o in alive} == {id(o) for o in (part, part.inner, launcher, part.inner.qweight_i32)}
        assert launcher.members == [part] and launcher.next_launcher is None
    finally:
        gc.enable()


@pytest.mark.parametrize("make", [copy.deepcopy, lambda m: pickle.loads(pickle.dumps(m))])
def test_a_copied_model_has_launchers_of_its_own(make):
    model = patched()
    other = make(model)
    del model
    launchers = []
    for li in range(2):
        for p in ToyDecoder.PROJ:
            w = other.proj(li, p)
            gl = w.group_launcher
            assert gl.usable and any(m is w for m in gl.members) and gl._sizes == {}
            if gl.members[0] is w:
                launchers.append(gl)
    assert len(launchers) == 8 and all(a.next_launcher is b for a, b in zip(launchers, launchers[1:] + launchers[:1]))


def test_room_for_r_that_a_graph_was_captured_with_stays(monkeypatch):
    capturing = [False]
    monkeypatch.setattr(K, "_is_capturing", lambda: capturing[0])
    monkeypatch.setattr(K, "current_stream_ptr", lambda device: 7)
    monkeypatch.setattr(K, "current_device", lambda: 0)
    device = SimpleNamespace(type="cuda", index=0)
    monkeypatch.setattr(K.torch, "zeros", lambda n, dtype, device, zeros=torch.zeros: zeros(n, dtype=dtype))
    cache, model = MiniGroupCache(), patched()
    cache._buf = model.proj(0, "mlp.down_proj")._own_r = None      # as a file of an earlier form has them
    for room in (cache.buffer, model.proj(0, "mlp.down_proj")._private_r):
        warm = room(5, 16, device)
        assert warm.shape == (5, 16) and warm.dtype == torch.float16 and room(5, 16, device) is warm
        capturing[0] = True
        captured = room(5, 16, device)
        capturing[0] = False
        assert captured.data_ptr() == warm.data_ptr()
        at = {room(m, 16, device).data_ptr() for m in (5, 16, 17, 300)}
        capturing[0] = True
        assert room(5, 16, device).data_ptr() == warm.data_ptr() not in at
        capturing[0] = False


@pytest.mark.gpu
@pytest.mark.parametrize("fuse", ["1", "0"])
@pytest.mark.parametrize("m", [1, 5, 20, 100])
def test_a_captured_step_beside_other_calls(m, fuse, monkeypatch):
    """A step in a graph, replayed on one stream while calls of other sizes, and of its own, run on another."""
    monkeypatch.setenv("GLOWQ_FUSE_GROUPS", fuse)
    sizes = dict(hidden=2048, kv=512, inter=8192)
    model, x = patched("cuda", rank=64, **sizes), inputs(m, 2048, 8192)
    other = {n: inputs(n, 2048, 8192, seed=n) for n in (m, 3, 33, 300)}
    with torch.no_grad():
        fresh = patched("cuda", rank=64, **sizes)
        want = [y.clone() for y in forward(fresh, *x)]
        want_other = {n: [y.clone() for y in forward(fresh, *other[n])] for n in other}
        for _ in range(2):
            forward(model, *x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = forward(model, *x)
        forward(model, *other[300])
        torch.cuda.synchronize()
        side, got = torch.cuda.Stream(), []
        for rep in range(6):
            for o in outs:
                o.fill_(float("nan"))
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                graph.replay()
            for n in other:
                got.append((n, forward(model, *other[n])))
            torch.cuda.current_stream().wait_stream(side)
            assert all(torch.equal(y, z) for y, z in zip(outs, want)), rep
        assert all(torch.equal(y, z) for n, ys in got for y, z in zip(ys, want_other[n]))
    ext = model.proj(0, "self_attn.q_proj").inner._get_ext()
    status = ext.lib.glowq_w4a16_read_status
    stream = torch.cuda.current_stream().cuda_stream
    mods = [model.proj(li, p) for li in range(2) for p in ToyDecoder.PROJ]
    used = [piece for w in mods for piece in pieces(w.group_launcher) + pieces(w.inner)]
    assert used and {status(piece.data_ptr(), stream) for piece in used} == {0}


@pytest.mark.gpu
def test_what_is_left_of_a_group(m=5):
    """A member whose wrapper is gone: the others launch for themselves, the producer first."""
    model, x = patched("cuda"), inputs(m)
    with torch.no_grad():
        want = [y.clone() for y in forward(model, *x)]
        model.model.layers[0].self_attn.k_proj = nn.Identity()
        model.model.layers[1].self_attn.q_proj = nn.Identity()
        got = forward(model, *x)
    for li in range(2):
        for i, p in enumerate(ToyDecoder.PROJ):
            if not isinstance(model.proj(li, p), nn.Identity):
                torch.testing.assert_close(got[7 * li + i], want[7 * li + i], rtol=1e-4, atol=1e-4)
