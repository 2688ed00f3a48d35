"""2 to 8 tokens on the tensor cores with exact integer weights, and the launches around it whose route a cost decides."""
import copy
import ctypes

import numpy as np
import pytest
import torch

import glowq_oracle as O
from glowq_b200.cuda_w4a16 import kernels as K
from gpu_helpers import Linear, assert_close, dev, make_group, new_out, run_group, status_ok
from test_workspace_layout import Map

pytestmark = pytest.mark.gpu


def exact_and_bound(lin, x, r, alpha):
    """The product in 64 bits with the launch's own r, and what fp32 accumulation of its exact products may lose: a group of 128 is
    eight MMAs whose 16 products and accumulator meet at the largest one's exponent, then one FMA a group, an MMA for 16 ranks, the
    bias and the sum of slices and warps.  (The streaming kernel stages x / 16: elements below 2^-10 keep 2^-21.)"""
    G, gid = -(-lin.ic // 128), np.arange(lin.ic) // 128
    q = O.unpack_int4_i32(lin.qweight, lin.ic).astype(np.float64)
    z = O.unpack_int4_i32(lin.qzeros, G).astype(np.float64)
    w = (q - z[:, gid]) * lin.scales[:, :G].astype(np.float64)[:, gid]
    # the streaming kernel takes codes and zero-points apart: what is rounded is up to codes plus zero-points large
    both = (q + z[:, gid]) * lin.scales[:, :G].astype(np.float64)[:, gid]
    xd = x.astype(np.float64)
    y, size, rank = xd @ w.T, np.abs(xd) @ both.T, 0
    lost = 2.0 ** -21 * (np.abs(xd) < 2.0 ** -10) @ both.T
    if r is not None:
        rd, L, rank = r.astype(np.float64), lin.L.astype(np.float64), r.shape[1]
        y, size = y + alpha * rd @ L.T, size + abs(alpha) * np.abs(rd) @ np.abs(L).T
    if lin.bias is not None:
        y, size = y + lin.bias.astype(np.float64), size + np.abs(lin.bias.astype(np.float64))
    return y, (8 * 17 + G + 17 * -(-rank // 16) + 32) * 2.0 ** -24 * size + lost


def route(g):
    """The kernel that this very call takes on this device."""
    out = Map()
    fn = K.load_w4a16_extension().lib.glowq_internal_workspace_map
    fn.argtypes = [ctypes.POINTER(K.Group), ctypes.c_int, ctypes.POINTER(Map)]
    assert fn(g, torch.cuda.get_device_properties(0).multi_processor_count, out) == 0
    return out.kernel


def rounded(lin):
    """The weights as fp16 numbers, scale included: what the exact form is there to avoid."""
    gid = np.arange(lin.ic) // 128
    q = O.unpack_int4_i32(lin.qweight, lin.ic).astype(np.float32)
    z = O.unpack_int4_i32(lin.qzeros, -(-lin.ic // 128)).astype(np.float32)
    return ((q - z[:, gid]).astype(np.float16) * lin.scales[:, gid]).astype(np.float64)


# rows below, at and above a tile of 128; a partial group, one group, an odd number of groups, K slices; ranks below, at and above a
# 64-column step; members without a correction
@pytest.mark.parametrize("M,ocs,ic,rank,alpha,bias", [
    (2, [257], 18944, 72, 1.0, True), (4, [40, 128, 100], 12296, 64, 0.5, False), (5, [72, 130], 8200, 264, 1.0, True),
    (8, [128], 128, 8, 1.0, False), (8, [3072], 256, 128, 0.5, True), (8, [1152], 3200, 136, 1.0, False),
    (7, [640], 5120, 16, 0.5, True)])
def test_exact_form_against_64_bits(M, ocs, ic, rank, alpha, bias):
    """Every element within what fp32 accumulation may lose, and in the 2-norm of the error (fp32 outputs) no further off than the
    streaming kernel on the same inputs by more than half, which is a tenth of the way to weights rounded to fp16 at most."""
    rng = np.random.default_rng(M * 1000 + ic)
    lins = [Linear(rng, oc, ic, bias=bias, rank=rank, quantize=ic % 128 != 0) for oc in ocs]
    R, x = (rng.standard_normal((rank, ic)) * 0.01).astype(np.float16), rng.standard_normal((M, ic)).astype(np.float16)
    use_L = [i != 1 for i in range(len(ocs))]
    fp16_off = [np.linalg.norm(x.astype(np.float64) @ rounded(l).T - exact_and_bound(copy_without_bias(l), x, None, 1.0)[0]) for l in lins]
    for dt, corrected in ((K.OUT_F32, False), (K.OUT_F32, True), (K.OUT_F16, True)):
        for r_mode in ((K.R_COMPUTE, K.R_LOAD) if corrected else (K.R_NONE,)):
            seen, off = [], []
            for kernel in (K.KERNEL_AUTO, K.KERNEL_AUTO, K.KERNEL_GEMV):
                r_buf = torch.zeros(M, rank, dtype=torch.float16, device="cuda")
                if r_mode == K.R_LOAD:
                    r_buf.copy_(dev((x.astype(np.float32) @ R.astype(np.float32).T).astype(np.float16)))
                outs = [new_out(M, l, dt) for l in lins]
                kw = dict(R_d=dev(R), r_buf=r_buf, r_mode=r_mode, alpha=alpha, use_L=use_L) if corrected else {}
                g = make_group(dev(x), lins, outs, out_dtype=dt, kernel=kernel, **kw)
                assert route(g) == (1 if kernel == K.KERNEL_AUTO else 0), (M, ocs, r_mode)
                assert run_group(g) == 0 and status_ok(g) == 0
                r = r_buf.cpu().numpy()
                if corrected:
                    want_r = x.astype(np.float64) @ R.astype(np.float64).T
                    lost = (ic + 16) * 2.0 ** -24 * (np.abs(x.astype(np.float64)) @ np.abs(R.astype(np.float64)).T)
                    assert (np.abs(r - want_r) <= lost + np.abs(want_r) * 2.0 ** -11 + 2.0 ** -24).all()
                off.append([])
                for l, o, c in zip(lins, outs, use_L):
                    y, bound = exact_and_bound(l, x, r if corrected and c else None, alpha)
                    if dt == K.OUT_F16:
                        bound = bound + np.abs(y) * 2.0 ** -11 + 2.0 ** -24
                    err = np.abs(o.double().cpu().numpy() - y)
                    assert (err <= bound).all(), (M, l.oc, kernel, r_mode, float((err / bound).max()))
                    off[-1].append(float(np.linalg.norm(err)))
                seen.append([o.cpu() for o in outs] + [r_buf.cpu()])
            assert all(torch.equal(a, b) for a, b in zip(seen[0], seen[1]))
            if dt == K.OUT_F32:
                for exact, stream, fp16 in zip(off[0], off[2], fp16_off):
                    assert exact <= 1.5 * stream and 10 * exact <= fp16, (M, ocs, r_mode, exact, stream, fp16)


def copy_without_bias(lin):
    c = copy.copy(lin)
    c.bias = None
    return c


@pytest.mark.parametrize("ms", [(8, 1, 5, 16, 2, 8, 1, 3), (5, 5, 1, 8, 33, 8, 8, 2)])
def test_exact_and_streaming_launches_take_turns_on_one_workspace(ms):
    """Both forms, their counters and their slots, back to back without a wait in between: each call gives the bits of a workspace
    of its own."""
    rng = np.random.default_rng(7)
    lins = {(oc, ic): Linear(rng, oc, ic, rank=128, quantize=False) for oc, ic in ((3584, 18944), (9472, 2560))}
    R = {ic: dev((rng.standard_normal((128, ic)) * 0.01).astype(np.float16)) for _, ic in lins}
    x = {ic: dev(rng.standard_normal((33, ic)).astype(np.float16)) for _, ic in lins}
    fresh = lambda: torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")

    def group(lin, M, ws):
        return make_group(x[lin.ic][:M], [lin], [new_out(M, lin)], R_d=R[lin.ic], r_mode=K.R_COMPUTE, ws=ws,
                          r_buf=torch.zeros(M, 128, dtype=torch.float16, device="cuda"))

    want = {}
    for M in set(ms):
        for key, lin in lins.items():
            g = group(lin, M, fresh())
            assert run_group(g) == 0 and status_ok(g) == 0
            want[key, M] = g._keep[2][0]
    ws, groups = fresh(), []
    for M in ms * 6:
        for key, lin in lins.items():
            groups.append((key, M, group(lin, M, ws)))
    many = (K.Group * len(groups))(*[g for _, _, g in groups])
    assert K.load_w4a16_extension().lib.glowq_w4a16_group_forward_many(many, len(groups)) == 0
    torch.cuda.synchronize()
    assert status_ok(groups[0][2]) == 0
    for key, M, g in groups:
        assert torch.equal(g._keep[2][0], want[key, M]), (key, M)


# one token, 12 chunks of 1024 columns and more: no slices, two, three, a last slice that is short; rows that do not fill a tile;
# fewer, as many and more row tiles than CTA slots; R units in several rounds
@pytest.mark.parametrize("oc,ic,rank", [(1530, 12288, 64), (3584, 13824, 128), (5120, 17408, 256), (7168, 12416, 16), (4096, 12288, 64)])
def test_one_token_on_long_rows(oc, ic, rank):
    rng = np.random.default_rng(oc + ic)
    lin = Linear(rng, oc, ic, rank=rank, quantize=False)
    R, xs = (rng.standard_normal((rank, ic)) * 0.01).astype(np.float16), rng.standard_normal((2, ic)).astype(np.float16)
    R_d, rows = dev(R), np.arange(0, oc, 5) if oc > 2000 else np.arange(oc)     # (64 bits of every fifth row: coprime to the tiles)
    some = copy.copy(lin)
    some.qweight, some.qzeros, some.scales, some.L = lin.qweight[rows], lin.qzeros[rows], lin.scales[rows], lin.L[rows]
    for M in (1, 2):
        for r_mode in (K.R_NONE, K.R_COMPUTE, K.R_COMPUTE):
            r_buf, out = torch.zeros(M, rank, dtype=torch.float16, device="cuda"), new_out(M, lin, K.OUT_F32)
            g = make_group(dev(xs[:M]), [lin], [out], out_dtype=K.OUT_F32,
                           **(dict(R_d=R_d, r_buf=r_buf, r_mode=r_mode) if r_mode != K.R_NONE else {}))
            assert run_group(g) == 0 and status_ok(g) == 0
            y, bound = exact_and_bound(some, xs[:M], r_buf.cpu().numpy() if r_mode != K.R_NONE else None, 1.0)
            assert out.isfinite().all() and (np.abs(out.double().cpu().numpy()[:, rows] - y) <= bound).all()


# slots of r at 9 to 64 tokens: as many as one, two and four lanes per four elements add in a round; at 65 tokens and more: 16
@pytest.mark.parametrize("M,ocs,ic,rank", [(9, [128], 12288, 64), (64, [384], 18944, 8), (33, [2048], 6144, 256), (17, [128], 18944, 128),
                                           (211, [256], 17408, 256), (70, [640], 18944, 8)])
def test_r_in_many_slices(M, ocs, ic, rank):
    rng = np.random.default_rng(M + ic)
    lins = [Linear(rng, oc, ic, rank=rank, quantize=False) for oc in ocs]
    R, x = (rng.standard_normal((rank, ic)) * 0.01).astype(np.float16), rng.standard_normal((M, ic)).astype(np.float16)
    r_buf = torch.zeros(M, rank, dtype=torch.float16, device="cuda")
    outs = [new_out(M, l) for l in lins]
    g = make_group(dev(x), lins, outs, R_d=dev(R), r_buf=r_buf, r_mode=K.R_COMPUTE)
    assert run_group(g) == 0 and status_ok(g) == 0
    want = x.astype(np.float64) @ R.astype(np.float64).T
    lost = (ic + 16) * 2.0 ** -24 * (np.abs(x.astype(np.float64)) @ np.abs(R.astype(np.float64)).T)
    assert (np.abs(r_buf.cpu().numpy() - want) <= lost + np.abs(want) * 2.0 ** -11 + 2.0 ** -24).all()
    for l, o in zip(lins, outs):
        assert_close(o, l.oracle(x, R), tol_abs=5e-2)   # K = 18944: outputs of 3.7 rms, fp16 ulp 2^-8
