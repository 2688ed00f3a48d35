"""The product with the weights in tensor memory (9 to 64 tokens) at the sizes where it can go wrong."""
import numpy as np
import pytest
import torch

from glowq_b200.cuda_w4a16 import kernels as K
from gpu_helpers import Linear, assert_close, dev, ext, make_group, new_out, run_group, status_ok

pytestmark = pytest.mark.gpu


# token tiles of 16 / 32 / 48 / 64 rows and their edges; output columns below, at and above a 128-row tile; K of a partial group,
# of one group, of fewer groups than stages; K slices (2048 columns and more); ranks below, at and above a 64-column step
@pytest.mark.parametrize("M,ocs,ic,rank,alpha,bias,f32", [
    (9, [128], 128, 8, 1.0, False, False), (16, [72, 130], 136, 64, 1.0, True, False), (17, [257], 1032, 72, 0.5, True, False),
    (33, [40, 128, 100], 2048, 64, 0.5, True, True), (48, [1152], 3200, 136, 1.0, False, False),
    (63, [512, 96], 5120, 16, 1.0, True, True), (64, [640], 6144, 264, 0.5, False, False), (64, [3072], 256, 128, 1.0, True, False)])
def test_against_the_oracle(M, ocs, ic, rank, alpha, bias, f32):
    rng = np.random.default_rng(M * 1000 + ic)
    lins = [Linear(rng, oc, ic, bias=bias, rank=rank) for oc in ocs]
    R = (rng.standard_normal((rank, ic)) * 0.01).astype(np.float16)
    x = rng.standard_normal((M, ic)).astype(np.float16)
    dt = K.OUT_F32 if f32 else K.OUT_F16
    seen = []
    for corrected in (False, True, True):
        outs = [new_out(M, l, dt) for l in lins]
        kw = dict(R_d=dev(R), r_buf=torch.zeros(M, rank, dtype=torch.float16, device="cuda"), r_mode=K.R_COMPUTE,
                  alpha=alpha) if corrected else {}
        g = make_group(dev(x), lins, outs, out_dtype=dt, **kw)
        assert run_group(g) == 0 and status_ok(g) == 0
        for l, o in zip(lins, outs):
            assert_close(o, l.oracle(x, R if corrected else None, alpha=alpha), tag=f"{M}x{l.oc}x{ic} corrected={corrected}")
        seen.append([o.cpu() for o in outs])
    assert all(torch.equal(a, b) for a, b in zip(seen[1], seen[2]))     # slices are added in slice order: the same bits


def test_strided_output_and_a_scarce_workspace():
    """Rows of a wider output (no 16-byte stores), and a workspace without room for slices: one CTA walks all of K."""
    rng = np.random.default_rng(3)
    lin = Linear(rng, 200, 4096)
    x = rng.standard_normal((24, 4096)).astype(np.float16)
    wide = torch.full((24, 203), float("nan"), dtype=torch.float16, device="cuda")
    for ws in (None, torch.zeros(64 << 10, dtype=torch.uint8, device="cuda")):
        g = make_group(dev(x), [lin], [wide], ws=ws, kernel=K.KERNEL_GEMM)
        assert run_group(g) == 0 and status_ok(g) == 0
        assert_close(wide[:, :200], lin.oracle(x))
        assert wide[:, 200:].isnan().all()


@pytest.mark.parametrize("M,ocs,ic,rank,launches", [(16, [3072, 1024, 1024], 3072, 64, 24), (64, [640], 18944, 128, 600),
                                                    (64, [4736], 3584, 128, 300), (32, [2048], 2048, 256, 24)])
def test_launches_back_to_back_on_one_workspace(M, ocs, ic, rank, launches):
    """Counters, slots and r of one workspace through launches that overlap (short slices reach their epilogue before the launch
    before is complete): every launch gives the same bits.  At 64 tokens the packed ring is shorter than the stages plus two, and
    without the wait for a stage's previous use about one launch in some hundred was wrong: hence the number of launches there."""
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
    many = (K.Group * len(groups))(*[g for g, _ in groups])
    assert K.load_w4a16_extension().lib.glowq_w4a16_group_forward_many(many, len(groups)) == 0
    torch.cuda.synchronize()
    assert status_ok(groups[0][0]) == 0
    for l, o in zip(lins, groups[0][1]):
        assert_close(o, l.oracle(x_d.cpu().numpy(), R_d.cpu().numpy()), tol_abs=5e-2)   # K = 18944: outputs of 3.7 rms, fp16 ulp 2^-8
    for g, outs in groups[1:]:
        assert torch.equal(g._keep[4], groups[0][0]._keep[4])
        assert all(torch.equal(a, b) for a, b in zip(outs, groups[0][1]))


def test_narrow_and_wide_launches_take_turns_on_one_workspace():
    """Calls of different widths, token counts and ranks share a workspace (and w4a16_*_forward_cuda share one per device): each
    gives the bits it gives on a workspace of its own, whatever the one before left in its slots, and the counters stay zero."""
    rng = np.random.default_rng(17)
    lins = {oc: Linear(rng, oc, 5120, rank=128, quantize=False) for oc in (512, 1024, 5120, 18944)}
    down = Linear(rng, 3584, 18944, quantize=False)           # at one token: K slices of the weight-streaming kernel
    x = {ic: dev(rng.standard_normal((64, ic)).astype(np.float16)) for ic in (5120, 18944)}
    R_d = dev((rng.standard_normal((128, 5120)) * 0.01).astype(np.float16))

    def call(oc, M, corrected, ws):
        lin = lins.get(oc, down)
        out = new_out(M, lin)
        kw = dict(R_d=R_d, r_buf=torch.zeros(M, 128, dtype=torch.float16, device="cuda"), r_mode=K.R_COMPUTE) if corrected else {}
        g = make_group(x[lin.ic][:M], [lin], [out], ws=ws, **kw)
        assert run_group(g) == 0 and status_ok(g) == 0, (oc, M, corrected)
        return out

    calls = [(18944, 16, False), (512, 16, False), (18944, 16, False), (1024, 64, True), (18944, 64, False), (512, 16, False),
             (3584, 1, False), (5120, 1, True), (18944, 16, True), (5120, 8, True), (5120, 33, True), (1024, 16, False), (3584, 1, False),
             (18944, 64, True)]
    nbytes = max(K.load_w4a16_extension().workspace_bytes(M, lins.get(oc, down).ic, oc, 128, 1) for oc, M, _ in calls)
    fresh = lambda: torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    want = {c: call(*c, fresh()) for c in set(calls)}
    ws = fresh()
    for c in calls:
        assert torch.equal(call(*c, ws), want[c]), c
        assert int(ws[256:1280].count_nonzero()) == 0 and int(ws[34048:38144].count_nonzero()) == 0, c
    e = K.load_w4a16_extension()
    for oc, M in ((18944, 16), (512, 16), (18944, 16), (3584, 1), (1024, 16), (18944, 16), (512, 16), (3584, 1)):
        lin = lins.get(oc, down)
        fn = e.w4a16_gemv_forward_cuda if M == 1 else e.w4a16_gemm_forward_cuda
        y = fn(x[lin.ic][:M], lin.d_qweight, lin.d_scales, lin.d_qzeros, 128)
        torch.testing.assert_close(y, want[oc, M, False], rtol=2e-3, atol=4e-3)   # (scratch of another size: other slices; an fp16 ulp)
    assert e.lib.glowq_w4a16_read_status(e._ws["cuda", 0].data_ptr(), torch.cuda.current_stream().cuda_stream) == 0


def test_more_sliced_tiles_than_the_workspace_has_counters():
    """Slices on request of more than 1024 row tiles: the launch brings counters of its own and clears them, also where the call
    before left partial sums."""
    rng = np.random.default_rng(18)
    lin = Linear(rng, 33024, 4096, quantize=False)
    x = rng.standard_normal((2, 4096)).astype(np.float16)
    ws = torch.full((64 << 20,), 255, dtype=torch.uint8, device="cuda")
    ws[:38144] = 0
    for _ in range(2):
        out = new_out(2, lin)
        g = make_group(dev(x), [lin], [out], split_k=4, ws=ws)
        assert run_group(g) == 0 and status_ok(g) == 0
        assert_close(out, lin.oracle(x))


@pytest.mark.parametrize("M,ocs,ic,rank,alpha,use_L", [
    (16, [128, 128], 128, 448, [1.0, 0.0], None), (9, [200, 136], 256, 1024, [0.5, 1.0], [True, False]),
    (64, [512, 96, 128], 5120, 128, [1.0, 0.5, 0.0], None), (33, [640, 640], 2048, 64, [1.0, 1.0], [False, True])])
def test_corrected_and_uncorrected_members_in_one_launch(M, ocs, ic, rank, alpha, use_L):
    """K slices of members with different numbers of steps: a member without a correction (alpha 0, no L) is the shortest, down
    to one step beside sixteen of the correction; with and without a second accumulator.  Two passes on one workspace."""
    rng = np.random.default_rng(M + rank)
    lins = [Linear(rng, oc, ic, rank=rank, bias=True) for oc in ocs]
    R = (rng.standard_normal((rank, ic)) * 0.01).astype(np.float16)
    x = rng.standard_normal((M, ic)).astype(np.float16)
    ws = None
    for _ in range(2):
        outs = [new_out(M, l, K.OUT_F32) for l in lins]
        g = make_group(dev(x), lins, outs, R_d=dev(R), r_buf=torch.zeros(M, rank, dtype=torch.float16, device="cuda"), ws=ws,
                       r_mode=K.R_COMPUTE, alpha=alpha, use_L=use_L, out_dtype=K.OUT_F32)
        ws = g._keep[5]
        assert run_group(g) == 0 and status_ok(g) == 0
        for i, (l, o) in enumerate(zip(lins, outs)):
            on = alpha[i] != 0 and (use_L is None or use_L[i])
            assert_close(o, l.oracle(x, R if on else None, alpha=alpha[i]), tag=f"member {i}")


def test_a_wait_that_runs_out_is_reported_and_leaves_the_device_usable():
    """The count of finished parts of r starts at a value it cannot reach: the CTAs that wait for r give up, let what they have
    in flight finish and return; the status word says so, and launches on another workspace are right."""
    rng = np.random.default_rng(21)
    lin = Linear(rng, 2048, 2048, rank=64)
    R = (rng.standard_normal((64, 2048)) * 0.01).astype(np.float16)
    x = rng.standard_normal((16, 2048)).astype(np.float16)
    kw = dict(R_d=dev(R), r_mode=K.R_COMPUTE)
    g = make_group(dev(x), [lin], [new_out(16, lin)], r_buf=torch.zeros(16, 64, dtype=torch.float16, device="cuda"), **kw)
    g._keep[5][256:1280].view(torch.int32)[64] = 1 << 20
    assert run_group(g) == 0                      # (the stream runs to its end)
    assert status_ok(g) == 7 and status_ok(g) == 0
    out = new_out(16, lin)
    g = make_group(dev(x), [lin], [out], r_buf=torch.zeros(16, 64, dtype=torch.float16, device="cuda"), **kw)
    assert run_group(g) == 0 and status_ok(g) == 0
    assert_close(out, lin.oracle(x, R))


def test_r_on_fewer_SMs_than_its_CTAs_need():
    """A stream of 8 SMs holds 16 CTAs of the launch, of which 20 compute r (and a second R tile's 20 more): none of them may
    wait for another one to be resident.  The same bits as on the whole device."""
    green = pytest.importorskip("torch.cuda.green_contexts")
    if not green.SUPPORTED:
        pytest.skip("PyTorch without green contexts")
    rng = np.random.default_rng(23)
    for rank, M in ((128, 16), (256, 50)):
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
