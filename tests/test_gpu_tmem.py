"""The product with the weights in tensor memory (9 to 64 tokens) at the sizes where it can go wrong."""
import numpy as np
import pytest
import torch

from glowq_b200.cuda_w4a16 import kernels as K
from gpu_helpers import Linear, assert_close, dev, make_group, new_out, run_group, status_ok

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


@pytest.mark.parametrize("M,ocs,ic,rank", [(16, [3072, 1024, 1024], 3072, 64), (64, [640], 18944, 128), (32, [2048], 2048, 256)])
def test_launches_back_to_back_on_one_workspace(M, ocs, ic, rank):
    """Counters, slots and r of one workspace through launches that overlap (short slices reach their epilogue before the launch
    before is complete; at 64 tokens the packed ring is shorter than the stages): every launch gives the same bits."""
    rng = np.random.default_rng(M)
    lins = [Linear(rng, oc, ic, rank=rank, quantize=False) for oc in ocs]
    R_d = dev((rng.standard_normal((rank, ic)) * 0.01).astype(np.float16))
    x_d = dev(rng.standard_normal((M, ic)).astype(np.float16))
    ws, groups = None, []
    for _ in range(24):
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
