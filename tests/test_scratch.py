"""What the launches of a module work in: pieces per stream, what a captured graph keeps, and results that have no history."""
import copy
import pickle
import threading

import pytest
import torch

from glowq_b200.cuda_w4a16 import kernels as K
from glowq_b200.cuda_w4a16.linear import CudaW4A16Linear

CPU = torch.device("cpu")


@pytest.fixture
def capturing(monkeypatch):
    state = [False]
    monkeypatch.setattr(K, "_is_capturing", lambda: state[0])
    return state


def test_a_stream_keeps_its_piece_until_a_larger_one_is_needed(capturing):
    s = K.Scratch()
    a = s.get(1000, CPU, 1)
    assert s.get(10, CPU, 1) is a and s.get(1000, CPU, 2) is not a and not a.any()
    b = s.get(1001, CPU, 1)
    assert b is not a and b.numel() == 1500 and s.get(1500, CPU, 1) is b
    assert s.get(1, CPU, 3).numel() == 256


def test_a_capture_takes_over_the_warm_ups_piece_and_keeps_it(capturing):
    s = K.Scratch()
    warm = s.get(1000, CPU, 0)
    capturing[0] = True
    assert s.get(1000, CPU, 7) is warm and s.get(10, CPU, 7) is warm     # every launch of the capture, every capture of the stream
    capturing[0] = False
    eager = s.get(1000, CPU, 0)
    assert eager is not warm and s.get(1000, CPU, 7) is not warm
    larger = s.get(5000, CPU, 0)                                          # calls outgrow their piece, not the captures'
    capturing[0] = True
    assert s.get(1000, CPU, 7) is warm
    assert s.get(5000, CPU, 7) is larger
    capturing[0] = False
    ref = [p.data_ptr() for p in s._kept]
    assert ref == [warm.data_ptr()]                                       # still held: the first graph has its address


def test_a_capture_without_a_warm_up_of_its_thread_keeps_nothing(capturing):
    s, made = K.Scratch(), []
    t = threading.Thread(target=lambda: made.append(s.get(1000, CPU, 5)))
    t.start()
    t.join()
    small = s.get(300, CPU, 0)
    capturing[0] = True
    for _ in range(2):
        got = s.get(1000, CPU, 5)
        assert got is not made[0] and got is not small and got.numel() == 1000
    capturing[0] = False
    assert s.get(1000, CPU, 5) is made[0] and s.get(300, CPU, 0) is small and s._kept == []


def test_the_default_stream_is_not_asked_whether_it_captures(monkeypatch):
    monkeypatch.setattr(K, "_is_capturing", lambda: 1 / 0)
    assert K.Scratch().get(300, CPU, 0).numel() == 300


def test_what_is_held_is_bounded(capturing):
    s = K.Scratch()
    for stream in range(1, 40):
        s.get(1000, CPU, stream)
    assert len(s._pieces) == K.Scratch.MAX_STREAMS
    s, n = K.Scratch(), 300
    while n < 300000:                                   # graphs of ever larger batches, each with its warm-up
        s.get(n, CPU, 0)
        capturing[0] = True
        s.get(n, CPU, 7)
        capturing[0] = False
        n = n * 21 // 20
    assert sum(p.numel() for p in s._kept) <= 3 * s._largest and s._largest <= 3 * n // 2


def test_a_copied_scratch_is_empty(capturing):
    s = K.Scratch()
    s.get(1000, CPU, 0)
    assert copy.deepcopy(s)._pieces == {} and pickle.loads(pickle.dumps(s))._pieces == {}


def _plain(oc, ic, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lin = torch.nn.Linear(ic, oc, bias=False, device="meta", dtype=torch.float16)
    lin.weight = torch.nn.Parameter(torch.randn(oc, ic, generator=gen, device="cuda", dtype=torch.float16) * 0.02, requires_grad=False)
    return CudaW4A16Linear.from_float(lin, 128), lambda m: torch.randn(m, ic, generator=gen, device="cuda", dtype=torch.float16)


def _status(mod):
    ext = K.load_w4a16_extension()
    return [ext.lib.glowq_w4a16_read_status(p.data_ptr(), torch.cuda.current_stream().cuda_stream)
            for p in list(mod._scratch._pieces.values()) + mod._scratch._kept]


@pytest.mark.gpu
@pytest.mark.parametrize("m,warm", [(5, True), (5, False), (1, True), (33, True), (100, True)])
def test_a_captured_call_survives_larger_ones(m, warm):
    """A K-sliced plain call from a graph: the memory it was captured with is its own after larger calls and whatever else is
    allocated, and with a call of the same module between two replays."""
    mod, act = _plain(3584, 18944)
    x, big = act(m), act(300)
    ref = _plain(3584, 18944)[0]          # the same weights, memory of its own
    with torch.no_grad():
        want, want_big = ref(x).clone(), ref(big).clone()
        if warm:
            mod(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = mod(x)
        held = []
        for n in (64, 300):
            mod(act(n))
            held.append([torch.full((1 << 18,), 0x7FFFFFFF, dtype=torch.int32, device="cuda") for _ in range(64)])
        for _ in range(3):
            out.fill_(float("nan"))
            graph.replay()
            got_big = mod(big)
            assert torch.equal(out, want) and torch.equal(got_big, want_big) and torch.equal(mod(x), want)
        torch.cuda.synchronize()
        assert set(_status(mod)) == {0}
        assert all(bool((t == 0x7FFFFFFF).all()) for ts in held for t in ts)


@pytest.mark.gpu
def test_one_module_on_two_streams():
    """Calls on two streams, neither waiting for the other: every one gives the bits of a call alone."""
    mod, act = _plain(3584, 18944, 1)
    xs = [act(5), act(64)]
    with torch.no_grad():
        want = [mod(x) for x in xs]
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        outs = [[], []]
        for _ in range(50):
            for i, s in enumerate(streams):
                with torch.cuda.stream(s):
                    outs[i].append(mod(xs[i]))
        torch.cuda.synchronize()
    assert all(torch.equal(o, want[i]) for i in (0, 1) for o in outs[i])
    assert set(_status(mod)) == {0}


@pytest.mark.gpu
def test_results_do_not_depend_on_the_calls_before():
    mod, act = _plain(2048, 8192, 2)
    x = {m: act(m) for m in (1, 3, 8, 20, 70, 300)}
    with torch.no_grad():
        first = {m: _plain(2048, 8192, 2)[0](x[m]) for m in x}
        for m in (300, 1, 70, 8, 20, 3, 300, 1, 3):
            assert torch.equal(mod(x[m]), first[m]), m
