"""Where launches keep their counters and partial results in a workspace that calls of all widths may share (no GPU: the
planner of the library is host arithmetic)."""
import ctypes
import itertools

import pytest

from glowq_b200.cuda_w4a16 import kernels as K


class Map(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("kernel", "ksplit", "whole_tiles", "sliced_tiles", "r_ctas", "shortest")] + [
        (n, ctypes.c_ulonglong) for n in ("ctr_begin", "ctr_end", "slots_begin", "slots_end")]


def workspace_map(M, ic, ocs, rank=0, alphas=None, nbytes=1 << 28, kernel=K.KERNEL_AUTO, split_k=0, sms=148, rc=0,
                  r_mode=K.R_COMPUTE):
    """The map of a call; every address is a placeholder."""
    at, g = 1 << 20, K.Group()
    g.x, g.M, g.IC, g.x_stride, g.group_size = at, M, ic, ic, 128
    g.kernel, g.split_k, g.n_members = kernel, split_k, len(ocs)
    g.workspace, g.workspace_bytes = at, nbytes
    if rank:
        g.r_mode, g.rank, g.r_buf, g.R, g.R_stride = r_mode, rank, at, at, ic
    groups = -(-ic // 128)
    for i, oc in enumerate(ocs):
        m = g.members[i]
        m.qweight = m.scales = m.qzeros = m.out = at
        m.OC = m.out_stride = oc
        m.weight_stride_i32, m.scale_stride, m.zero_stride_i32 = groups * 16, groups, -(-groups // 8)
        m.alpha = 1.0 if alphas is None else alphas[i]
        if rank:
            m.L, m.L_stride = at, rank
    out = Map()
    fn = K.load_w4a16_extension().lib.glowq_internal_workspace_map
    fn.argtypes = [ctypes.POINTER(K.Group), ctypes.c_int, ctypes.POINTER(Map)]
    assert fn(g, sms, out) == rc
    return out


WIDTHS = [[128], [512], [1024], [3584], [5120], [18944], [65536], [151936], [5120] * 3, [3072, 1024, 1024], [17408] * 2]


def test_counters_of_any_call_lie_in_front_of_the_slots_of_every_other():
    """A call leaves bits of partial sums in its slots and takes its counters to be zero, so no call's counters may lie where
    another one keeps slots: narrow before wide, 9 to 64 tokens before one token, and the other way around."""
    counters = slots = 0
    for ocs, ic, M, rank in itertools.product(WIDTHS, (128, 2048, 5120, 18944), (1, 5, 8, 9, 16, 33, 64, 100, 300), (0, 64, 1024)):
        for split_k in ((0, 4) if M <= 8 else (0,)):
            m = workspace_map(M, ic, ocs, rank, split_k=split_k)
            tag = (ocs, ic, M, rank, split_k)
            assert m.slots_begin <= m.slots_end and m.slots_begin >= 38144, tag
            if m.ctr_end > m.ctr_begin:
                counters += 1
                assert m.ctr_begin == 34048 and m.ctr_end <= 38144, tag
            slots += m.slots_end > m.slots_begin
    assert counters > 100 and slots > 500


def test_a_launch_with_more_sliced_tiles_than_counters_brings_its_own():
    """Slices on request and more than 32768 output rows: the counters lie among the slots (the launch clears them)."""
    m = workspace_map(1, 4096, [32768], split_k=4)
    assert m.ksplit == 4 and m.sliced_tiles == 1024 and (m.ctr_begin, m.ctr_end) == (34048, 38144)
    m = workspace_map(1, 4096, [32800], split_k=4)
    assert m.ksplit == 4 and m.sliced_tiles == 1025 and m.ctr_end == 0 and m.slots_begin == 38144
    # the size grows with the rows whether or not K is sliced: 2^26 of them do not fit the scratch of 4 MiB + 4 KiB that is
    # part of the library
    workspace_map(1, 128, [1 << 26], nbytes=(4 << 20) + 4096, rc=4)
    workspace_map(1, 128, [(1 << 25) - (1 << 15)], nbytes=(4 << 20) + 38144)


@pytest.mark.parametrize("M,ic,oc,rank", [(16, 5120, 5120, 128), (64, 5120, 15360, 128), (1, 18944, 3584, 128), (33, 8192, 3072, 64)])
def test_the_reported_size_holds_the_slices(M, ic, oc, rank):
    """With exactly the bytes glowq_w4a16_workspace_bytes asks for, a launch takes the slices it takes with any amount."""
    e = K.load_w4a16_extension()
    exact = workspace_map(M, ic, [oc], rank, nbytes=e.workspace_bytes(M, ic, oc, rank, 1))
    ample = workspace_map(M, ic, [oc], rank)
    assert (exact.ksplit, exact.whole_tiles, exact.sliced_tiles) == (ample.ksplit, ample.whole_tiles, ample.sliced_tiles)
    assert exact.ksplit > 1


@pytest.mark.parametrize("ic,rank", [(128, 448), (128, 1024), (256, 1024), (640, 1024), (5120, 256)])
@pytest.mark.parametrize("M", [9, 16, 33, 64])
def test_no_slice_of_a_group_of_unlike_members_is_empty(M, ic, rank):
    """Each member is cut by its own K steps: the one without a correction has the fewest, and no more slices than that."""
    for ocs in ([128, 128], [1024, 1024], [5120, 5120, 5120], [128, 8192]):
        for alphas in ([1.0, 0.0, 0.5], [0.0, 1.0, 1.0], [0.5, 0.0, 0.0]):
            m = workspace_map(M, ic, ocs, rank, alphas=alphas[:len(ocs)])
            assert m.kernel == 1 and m.shortest == -(-ic // 128) and m.ksplit <= m.shortest, (ocs, alphas, m.ksplit)


# calls of the CTA pairs with ranks above 512 against a short K: (tokens, columns, K, rank, how r comes)
BEHIND_THE_WEIGHTS = [(65, 19200, 1408, 1016, K.R_COMPUTE), (128, 19072, 2560, 976, K.R_COMPUTE), (200, 10240, 2560, 960, K.R_COMPUTE),
                      (256, 20224, 1536, 1024, K.R_LOAD), (100, 512, 1536, 1024, K.R_LOAD), (65, 128, 1152, 648, K.R_LOAD)]


@pytest.mark.parametrize("M,oc,ic,rank,r_mode", BEHIND_THE_WEIGHTS)
def test_the_plans_have_slices_that_start_behind_the_weights(M, oc, ic, rank, r_mode):
    nbytes = K.load_w4a16_extension().workspace_bytes(M, ic, oc, rank, 1)
    m = workspace_map(M, ic, [oc], rank, alphas=[0.5], nbytes=nbytes, r_mode=r_mode)
    groups, steps = -(-ic // 128), -(-ic // 128) + -(-rank // 128)
    assert m.kernel == 2 and m.ksplit > 1 and steps * (m.ksplit - 1) // m.ksplit > groups


@pytest.mark.parametrize("M", [2, 3, 5, 8])
def test_what_the_exact_form_takes_and_what_stays_with_the_streaming_kernel(M):
    """Only calls that the streaming kernel would take as well (its scratch, its layouts), and none that ask for something of its own."""
    for ocs, ic, rank in itertools.product(([128], [72, 130], [5120], [3584, 512, 512], [18944] * 2), (128, 2048, 8200, 18944), (0, 64, 264)):
        m = workspace_map(M, ic, ocs, rank)
        assert m.kernel in (0, 1)
        assert workspace_map(M, ic, ocs, rank, kernel=K.KERNEL_GEMV).kernel == 0
        assert workspace_map(M, ic, ocs, rank, split_k=2).kernel == 0
        e = K.load_w4a16_extension()
        need = e.workspace_bytes(M, ic, sum(ocs), rank, len(ocs))
        exact = workspace_map(M, ic, ocs, rank, nbytes=need)
        assert (exact.kernel, exact.ksplit, exact.slots_end <= need) == (m.kernel, m.ksplit, True)
        stream = workspace_map(M, ic, ocs, rank, kernel=K.KERNEL_GEMV)
        if stream.slots_end > 38144:
            workspace_map(M, ic, ocs, rank, nbytes=stream.slots_end - 1, rc=4)
    assert workspace_map(8, 18944, [3584], 128).kernel == 1 and workspace_map(1, 18944, [3584], 128).kernel == 0


def test_one_token_on_long_rows_takes_no_more_scratch_than_its_most_slices():
    """The cost of a one-token launch may choose fewer slices than fit; the scratch asked for does not depend on the choice."""
    seen = set()
    for oc, ic, rank in itertools.product((32, 1536, 2048, 3584, 5120, 7168, 9216, 9472), (12288, 13824, 17408, 18944, 32768, 65536), (0, 16, 128, 1024)):
        m = workspace_map(1, ic, [oc], rank)
        seen.add(m.ksplit)
        assert m.kernel == 0 and m.slots_end >= m.slots_begin + m.sliced_tiles * m.ksplit * 1024
        workspace_map(1, ic, [oc], rank, nbytes=m.slots_end - 1, rc=4)
        need = K.load_w4a16_extension().workspace_bytes(1, ic, oc, rank, 1)
        assert workspace_map(1, ic, [oc], rank, nbytes=need).ksplit == m.ksplit
    assert {1, 2, 3, 4} <= seen


# tokens, columns, K, rank (0: no correction), microseconds streamed and in the exact form on B200, call after call
MEASURED = [(4, [4224], 12416, 256, 33.6, 16.0), (6, [4480], 4992, 256, 17.7, 11.6), (7, [16768, 16768], 4992, 0, 40.8, 28.5),
            (5, [3840], 3840, 256, 15.1, 11.1), (4, [2048], 9600, 0, 12.3, 9.5), (5, [13696, 13696], 3456, 0, 24.3, 18.9),
            (7, [1920, 1408, 1408], 2304, 128, 12.3, 9.8), (3, [9856, 9856], 4608, 128, 20.6, 26.7),
            (3, [12544, 12544], 2432, 64, 13.9, 17.0), (2, [3840] * 3, 3328, 256, 11.3, 13.8), (2, [3584] * 3, 2560, 128, 9.6, 11.0),
            (3, [10624, 10624], 4736, 64, 23.4, 26.5)]


@pytest.mark.parametrize("M,ocs,ic,rank,stream,exact", MEASURED)
def test_two_to_eight_tokens_take_the_kernel_that_was_measured_faster(M, ocs, ic, rank, stream, exact):
    nbytes = K.load_w4a16_extension().workspace_bytes(M, ic, sum(ocs), rank, len(ocs))
    assert workspace_map(M, ic, ocs, rank, nbytes=nbytes).kernel == (1 if exact < stream else 0)


def test_two_to_eight_tokens_ask_for_the_slices_they_take():
    """With the reported bytes a call is cut as with any amount, in the form the library chooses and in the one asked for, whatever
    its members' sizes; and it is not asked for much more."""
    e, layer = K.load_w4a16_extension(), 0
    groups = [([5120] * 3, 5120), ([5120], 5120), ([13824] * 2, 5120), ([5120], 13824)]
    others = [([3000, 500, 501, 1], 2176), ([129, 127], 18944), ([1], 640), ([9856] * 2, 4608), ([200, 200, 200, 200], 8200)]
    for (ocs, ic), rank, kernel in itertools.product(groups + others, (0, 16, 128, 1024), (K.KERNEL_AUTO, K.KERNEL_GEMM)):
        need = e.workspace_bytes(6, ic, sum(ocs), rank, len(ocs))
        for r_mode in (K.R_COMPUTE, K.R_LOAD):
            a, b = (workspace_map(6, ic, ocs, rank, nbytes=n, kernel=kernel, r_mode=r_mode) for n in (need, 1 << 28))
            assert (a.kernel, a.ksplit, a.whole_tiles, a.sliced_tiles) == (b.kernel, b.ksplit, b.whole_tiles, b.sliced_tiles)
    for ocs, ic in groups:
        layer += e.workspace_bytes(8, ic, sum(ocs), 128, len(ocs))
    assert layer < 9e6


# outputs, K, rank (0: no correction), the number of slices that was fastest on B200, its microseconds and those of another number
SLICES = [(2304, 14208, 40, 3, 12.2, 15.3), (2944, 16256, 40, 3, 14.3, 22.2), (5760, 16256, 64, 3, 21.1, 27.7),
          (4992, 13440, 40, 3, 17.4, 19.2), (3584, 16256, 0, 4, 14.2, 18.9), (3584, 17920, 128, 1, 15.7, 17.6), (3584, 13824, 0, 1, 10.8, 14.2),
          (7168, 12288, 64, 1, 17.3, 22.6), (5120, 17408, 256, 3, 24.4, 29.2)]


@pytest.mark.parametrize("oc,ic,rank,slices,us,other", SLICES)
def test_one_token_on_long_rows_takes_the_slices_that_were_measured_fastest(oc, ic, rank, slices, us, other):
    nbytes = K.load_w4a16_extension().workspace_bytes(1, ic, oc, rank, 1)
    assert us < other and workspace_map(1, ic, [oc], rank, nbytes=nbytes).ksplit == slices
