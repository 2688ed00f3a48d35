"""The product of CTA pairs (65 tokens and more) at the sizes where it can go wrong."""
import numpy as np
import pytest
import torch

from glowq_b200.cuda_w4a16 import kernels as K
from gpu_helpers import Linear, assert_close, dev, ext, make_group, new_out, run_group, status_ok
from test_workspace_layout import BEHIND_THE_WEIGHTS

pytestmark = pytest.mark.gpu


# token tiles of 64 to 256 rows and their edges, one and several of them; output columns below, at and above the 128 rows of a CTA
# and the 256 of a pair, members that share a pair; K of a partial group, of one group, odd numbers of groups (scales in loads of
# 1, 2, 4 and 8); K slices; ranks below, at and above the 64 and 128 columns of a correction step
@pytest.mark.parametrize("M,ocs,ic,rank,alpha,bias,f32", [
    (65, [128], 128, 8, 1.0, False, False), (100, [72, 130], 136, 64, 1.0, True, False), (127, [257], 1032, 72, 0.5, True, False),
    (200, [40, 128, 100], 2048, 64, 0.5, True, True), (220, [5000], 1408, 48, 1.0, True, False), (256, [640], 3584, 128, 1.0, True, True),
    (300, [1152], 3200, 136, 1.0, False, False), (513, [3072], 256, 128, 1.0, True, False), (777, [512, 96], 5120, 16, 1.0, True, True),
    (1000, [640], 6144, 264, 0.5, False, False), (2500, [1024, 1024], 1024, 64, 0.5, True, False)])
def test_against_the_oracle(M, ocs, ic, rank, alpha, bias, f32):
    rng = np.random.default_rng(M * 1000 + ic)
    lins = [Linear(rng, oc, ic, bias=bias, rank=rank, quantize=ic % 128 != 0) for oc in ocs]
    R = (rng.standard_normal((rank, ic)) * 0.01).astype(np.float16)
    x = rng.standard_normal((M, ic)).astype(np.float16)
    dt = K.OUT_F32 if f32 else K.OUT_F16
    seen, ws = [], None
    for corrected in (False, True, True):
        outs = [new_out(M, l, dt) for l in lins]
        kw = dict(R_d=dev(R), r_buf=torch.zeros(M, rank, dtype=torch.float16, device="cuda"), r_mode=K.R_COMPUTE,
                  alpha=alpha, ws=ws) if corrected else {}
        g = make_group(dev(x), lins, outs, out_dtype=dt, **kw)
        assert run_group(g) == 0 and status_ok(g) == 0
        for l, o in zip(lins, outs):
            assert_close(o, l.oracle(x, R if corrected else None, alpha=alpha), tag=f"{M}x{l.oc}x{ic} corrected={corrected}")
        if corrected:
            ws = g._keep[5]
            assert int(ws[256:1280].count_nonzero()) == 0 and int(ws[34048:38144].count_nonzero()) == 0
        seen.append([o.cpu() for o in outs])
    assert all(torch.equal(a, b) for a, b in zip(seen[1], seen[2]))     # slices are added in slice order: the same bits


@pytest.mark.parametrize("M,ocs,ic,alpha,f32", [(15000, [384], 128, 1.0, False), (12000, [128, 200], 128, 0.5, False),
                                                (15000, [330], 128, 1.0, True), (9000, [40, 300, 300], 256, 1.0, False)])
def test_output_stages_of_warps_with_and_without_columns(M, ocs, ic, alpha, f32):
    """Short tiles one after another, and warps whose columns lie inside the outputs in one tile and past the end in the next: a stage
    is written again only when the copy engine has read it."""
    rng = np.random.default_rng(M)
    lins = [Linear(rng, oc, ic, rank=16, quantize=False) for oc in ocs]
    x_d, R_d = dev(rng.standard_normal((M, ic)).astype(np.float16)), dev((rng.standard_normal((16, ic)) * 0.01).astype(np.float16))
    dt, seen, want = K.OUT_F32 if f32 else K.OUT_F16, [], [l.oracle(x_d.cpu().numpy(), R_d.cpu().numpy(), alpha=alpha) for l in lins]
    for _ in range(5):
        outs = [new_out(M, l, dt) for l in lins]
        g = make_group(x_d, lins, outs, R_d=R_d, r_buf=torch.zeros(M, 16, dtype=torch.float16, device="cuda"), r_mode=K.R_COMPUTE,
                       alpha=alpha, out_dtype=dt)
        assert run_group(g) == 0 and status_ok(g) == 0
        for o, w in zip(outs, want):
            assert_close(o, w)
        seen.append([o.cpu() for o in outs])
    assert all(torch.equal(a, b) for s in seen[1:] for a, b in zip(s, seen[0]))


@pytest.mark.parametrize("M,oc,ic,rank,r_mode", BEHIND_THE_WEIGHTS)
@pytest.mark.parametrize("alpha", [0.5, 1.0])
def test_slices_that_start_behind_the_weights(M, oc, ic, rank, r_mode, alpha):
    """K slices of nothing but correction steps, and not the first of them: with a factor other than 1 they accumulate beside the
    weights' products, and with 1 among them."""
    rng = np.random.default_rng(M + rank)
    lin = Linear(rng, oc, ic, rank=rank, bias=True, quantize=False)
    x = rng.standard_normal((M, ic)).astype(np.float16)
    R = (rng.standard_normal((rank, ic)) * 0.01).astype(np.float16)
    r_buf = torch.zeros(M, rank, dtype=torch.float16, device="cuda")
    if r_mode == K.R_LOAD:
        r_buf.copy_(dev(x.astype(np.float32) @ R.astype(np.float32).T))
    want, seen = lin.oracle(x, R, alpha=alpha), []
    for _ in range(2):
        out = new_out(M, lin, K.OUT_F32)
        g = make_group(dev(x), [lin], [out], R_d=dev(R), r_buf=r_buf, r_mode=r_mode, alpha=alpha, out_dtype=K.OUT_F32)
        assert run_group(g) == 0 and status_ok(g) == 0
        assert_close(out, want, tag=f"alpha {alpha}")
        seen.append(out.cpu())
    assert torch.equal(*seen)


def test_other_layouts_and_scarce_workspaces():
    """Rows of a wider output (no copies of whole rows), a workspace without slots, one without counters (r in front of the members,
    every tile a cluster of its own)."""
    rng = np.random.default_rng(3)
    lin = Linear(rng, 200, 4096, rank=40)
    R = (rng.standard_normal((40, 4096)) * 0.01).astype(np.float16)
    x = rng.standard_normal((150, 4096)).astype(np.float16)
    wide = torch.full((150, 203), float("nan"), dtype=torch.float16, device="cuda")
    for nbytes in (None, 64 << 10, 1024):
        ws = None if nbytes is None else torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
        for kw in ({}, dict(R_d=dev(R), r_buf=torch.zeros(150, 40, dtype=torch.float16, device="cuda"), r_mode=K.R_COMPUTE)):
            g = make_group(dev(x), [lin], [wide], ws=ws, **kw)
            assert run_group(g) == 0 and status_ok(g) == 0
            assert_close(wide[:, :200], lin.oracle(x, R if kw else None))
            assert wide[:, 200:].isnan().all()


@pytest.mark.parametrize("M,alpha,use_L", [(150, [1.0, 0.5, 0.0], None), (300, [1.0, 1.0, 1.0], [False, True, False])])
def test_corrected_and_uncorrected_members_in_one_launch(M, alpha, use_L):
    """Members that share a pair, one of them without a correction, with and without a second accumulator."""
    rng = np.random.default_rng(M)
    lins = [Linear(rng, oc, 640, rank=72, bias=True) for oc in (384, 100, 130)]
    R = (rng.standard_normal((72, 640)) * 0.01).astype(np.float16)
    x = rng.standard_normal((M, 640)).astype(np.float16)
    outs = [new_out(M, l, K.OUT_F32) for l in lins]
    g = make_group(dev(x), lins, outs, R_d=dev(R), r_buf=torch.zeros(M, 72, dtype=torch.float16, device="cuda"), r_mode=K.R_COMPUTE,
                   alpha=alpha, use_L=use_L, out_dtype=K.OUT_F32)
    assert run_group(g) == 0 and status_ok(g) == 0
    for i, (l, o) in enumerate(zip(lins, outs)):
        on = alpha[i] != 0 and (use_L is None or use_L[i])
        assert_close(o, l.oracle(x, R if on else None, alpha=alpha[i]), tag=f"member {i}")


@pytest.mark.parametrize("M,ocs,ic,use_L", [(100, [384, 200, 128], 4096, [True, False, True]), (300, [128, 640], 640, [False, True]),
                                            (70, [100, 100, 300, 40], 1024, [True, False, False, True]),
                                            (700, [384, 130], 2048, [False, True])])
def test_an_overflow_of_r_stays_with_the_corrected_members(M, ocs, ic, use_L):
    """r is fp16 and may hold infinities: the tokens' results of the members without a correction do not depend on it, wherever their
    column tiles lie."""
    rng = np.random.default_rng(M)
    lins = [Linear(rng, oc, ic, rank=72, bias=True, quantize=False) for oc in ocs]
    x = rng.standard_normal((M, ic)).astype(np.float16)
    R = (rng.standard_normal((72, ic)) * 0.01).astype(np.float16)
    r_buf = dev((x.astype(np.float32) @ R.astype(np.float32).T).astype(np.float16))
    r_buf[3, 5], r_buf[M - 1, 71] = float("inf"), float("-inf")
    outs = [new_out(M, l) for l in lins]
    g = make_group(dev(x), lins, outs, R_d=dev(R), r_buf=r_buf, r_mode=K.R_LOAD, use_L=use_L)
    assert run_group(g) == 0 and status_ok(g) == 0
    finite = [t for t in range(M) if t not in (3, M - 1)]
    for i, (l, o) in enumerate(zip(lins, outs)):
        want = l.oracle(x, R if use_L[i] else None)
        if use_L[i]:
            assert not o[3].isfinite().any()
            assert_close(o[finite], want[finite], tag=f"member {i}")
        else:
            assert_close(o, want, tag=f"member {i}")


@pytest.mark.parametrize("M,ocs,ic,rank,launches", [(211, [5120], 5120, 256, 100), (600, [3072, 1024, 1024], 3072, 64, 60),
                                                    (1300, [2048], 8192, 64, 40), (90, [1024], 18944, 128, 100)])
def test_launches_back_to_back_on_one_workspace(M, ocs, ic, rank, launches):
    """Tickets, counters, slots and r of one workspace through launches that overlap: every launch gives the same bits."""
    rng = np.random.default_rng(M)
    lins = [Linear(rng, oc, ic, rank=rank, quantize=False) for oc in ocs]
    R_d = dev((rng.standard_normal((rank, ic)) * 0.01).astype(np.float16))
    x_d = dev(rng.standard_normal((M, ic)).astype(np.float16))
    ws, groups = None, []
    for _ in range(launches):
        outs = [new_out(M, l) for l in lins]
        g = make_group(x_d, lins, outs, R_d=R_d, r_buf=torch.zeros(M, rank, dtype=torch.float16, device="cuda"), r_mode=K.R_COMPUTE,
                       ws=ws)
        ws = g._keep[5]
        groups.append((g, outs))
    torch.cuda.synchronize()
    many = (K.Group * len(groups))(*[g for g, _ in groups])
    assert K.load_w4a16_extension().lib.glowq_w4a16_group_forward_many(many, len(groups)) == 0
    torch.cuda.synchronize()
    assert status_ok(groups[0][0]) == 0
    for l, o in zip(lins, groups[0][1]):
        assert_close(o, l.oracle(x_d.cpu().numpy(), R_d.cpu().numpy()), tol_abs=5e-2)   # K = 18944: outputs of 3.7 rms, fp16 ulp 2^-8
    for g, outs in groups[1:]:
        assert torch.equal(g._keep[4], groups[0][0]._keep[4])
        assert all(torch.equal(a, b) for a, b in zip(outs, groups[0][1]))


def test_a_wait_that_runs_out_is_reported_and_leaves_the_device_usable():
    """The count of finished r tiles starts at a value that it cannot reach: the CTAs that wait for r give up, let what they have in
    flight finish and return; the status word says so, and launches on another workspace are right."""
    rng = np.random.default_rng(21)
    lin = Linear(rng, 2048, 2048, rank=64)
    R = (rng.standard_normal((64, 2048)) * 0.01).astype(np.float16)
    x = rng.standard_normal((100, 2048)).astype(np.float16)
    kw = dict(R_d=dev(R), r_mode=K.R_COMPUTE)
    g = make_group(dev(x), [lin], [new_out(100, lin)], r_buf=torch.zeros(100, 64, dtype=torch.float16, device="cuda"), **kw)
    g._keep[5][256:1280].view(torch.int32)[73] = 1 << 20
    assert run_group(g) == 0                      # (the stream runs to its end)
    assert status_ok(g) == 7 and status_ok(g) == 0
    out = new_out(100, lin)
    g = make_group(dev(x), [lin], [out], r_buf=torch.zeros(100, 64, dtype=torch.float16, device="cuda"), **kw)
    assert run_group(g) == 0 and status_ok(g) == 0
    assert_close(out, lin.oracle(x, R))


_LATE_SCRIPT = r"""
import numpy as np, torch
from glowq_b200.cuda_w4a16 import kernels as K
from gpu_helpers import Linear, assert_close, dev, ext, make_group, new_out, status_ok
lib, stream = ext().lib, torch.cuda.current_stream().cuda_stream
p, mem, flags = K.Peers(), [torch.zeros(4096, dtype=torch.float16, device="cuda") for _ in range(2)], torch.zeros(64, dtype=torch.int32, device="cuda")
for r in range(2):                           # "rank 1" is local memory that nobody ever writes flags into
    p.buf[r], p.flag[r] = mem[r].data_ptr(), flags.data_ptr() + 16 * r
p.epoch, p.status = flags.data_ptr() + 64, flags.data_ptr() + 128
p.world, p.rank, p.sites, p.max_n = 2, 0, 2, 1024
v = torch.ones(1024, dtype=torch.float16, device="cuda")
rng = np.random.default_rng(5)
lin = Linear(rng, 5120, 1024, quantize=False)
x = rng.standard_normal((1000, 1024)).astype(np.float16)
late, right = [make_group(dev(x), [lin], [new_out(1000, lin)]) for _ in range(2)]
assert lib.glowq_w4a16_group_forward(right) == 0 and status_ok(right) == 0    # (the kernel is loaded)
torch.cuda.synchronize()
assert lib.glowq_w4a16_allreduce_f16(p, v.data_ptr(), 1024, 0, stream) == 0 and lib.glowq_w4a16_group_forward(late) == 0
torch.cuda.synchronize()
print("LATE", status_ok(late), int(flags[32]))
assert lib.glowq_w4a16_group_forward(right) == 0
torch.cuda.synchronize()
assert_close(right._keep[2][0], lin.oracle(x))
print("RIGHT", status_ok(right))
"""


def test_a_launch_whose_first_waits_run_out():
    """The warps that run ahead of the kernel before wait for their first item, which comes by ticket when that kernel is complete.  One
    that lasts longer than their waits (an all-reduce whose second rank never arrives, with a poll limit of some seconds) makes them
    give up before they have read an item: status 7, nothing faults, and launches on another workspace are right."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    root = os.path.dirname(here)
    env = dict(os.environ, GLOWQ_AR_SPIN_LIMIT="6000000", PYTHONPATH=os.pathsep.join((root, here, os.path.join(root, "oracle"))))
    r = subprocess.run([sys.executable, "-c", _LATE_SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "LATE 7 4" in r.stdout and "RIGHT 0" in r.stdout, r.stdout


def test_on_a_few_SMs():
    """A stream of 8 SMs: items are taken in order, so no CTA waits for one that cannot start.  The same bits as on the whole device."""
    green = pytest.importorskip("torch.cuda.green_contexts")
    if not green.SUPPORTED:
        pytest.skip("PyTorch without green contexts")
    rng = np.random.default_rng(23)
    for rank, M in ((128, 100), (256, 700)):
        lin = Linear(rng, 2048, 5120, rank=rank, quantize=False)
        x_d, R_d = dev(rng.standard_normal((M, 5120)).astype(np.float16)), dev((rng.standard_normal((rank, 5120)) * 0.01).astype(np.float16))
        outs = [new_out(M, lin) for _ in range(2)]
        rs = [torch.zeros(M, rank, dtype=torch.float16, device="cuda") for _ in range(2)]
        ctx = green.GreenContext.create(8, 0)
        few = ctx.Stream()
        for i in range(2):
            torch.cuda.synchronize()
            g = make_group(x_d, [lin], [outs[i]], R_d=R_d, r_buf=rs[i], r_mode=K.R_COMPUTE)
            torch.cuda.synchronize()
            if i == 1:
                g.stream = few.cuda_stream
                ctx.set_context()
            try:
                rc = run_group(g)
                assert rc == 0 and status_ok(g) == 0, (i, rc, ext().lib.glowq_w4a16_last_cuda_error())
            finally:
                if i == 1:
                    ctx.pop_context()
        assert_close(outs[0], lin.oracle(x_d.cpu().numpy(), R_d.cpu().numpy()))
        assert torch.equal(outs[0], outs[1]) and torch.equal(rs[0], rs[1])
