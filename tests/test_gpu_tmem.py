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
