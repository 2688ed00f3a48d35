"""Loader of the sm_100a C-ABI library and torch-tensor front ends of its entry points.

Counterpart of GlowQ's ``cuda_w4a16/kernels.py`` (``load_w4a16_extension``, src/cuda_w4a16/kernels.py:16-59)
and of the three names its pybind module exports (src/cuda_w4a16/csrc/pybind.cpp:19-34).  There is no JIT
fallback and no other backend: if the library is missing or the device is not sm_100, calls raise."""
from __future__ import annotations

import ctypes
import os
import struct
import threading
from typing import Optional

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
_LIB_NAME = "libglowq_w4a16.so"

GLOWQ_OK = 0
ERR_DEVICE_TIMEOUT = 7
OUT_F16, OUT_F32 = 0, 1
R_NONE, R_COMPUTE, R_LOAD = 0, 1, 2
KERNEL_AUTO, KERNEL_GEMV, KERNEL_GEMM = 0, 1, 2
MAX_MEMBERS = 4
ABI_VERSION = 2


class Member(ctypes.Structure):
    _fields_ = [("qweight", ctypes.c_void_p), ("scales", ctypes.c_void_p), ("qzeros", ctypes.c_void_p),
                ("bias", ctypes.c_void_p), ("L", ctypes.c_void_p), ("out", ctypes.c_void_p),
                ("OC", ctypes.c_int32), ("weight_stride_i32", ctypes.c_int32), ("zero_stride_i32", ctypes.c_int32),
                ("scale_stride", ctypes.c_int32), ("L_stride", ctypes.c_int32), ("out_stride", ctypes.c_int32),
                ("alpha", ctypes.c_float), ("reserved", ctypes.c_int32)]


class Group(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("R", ctypes.c_void_p), ("r_buf", ctypes.c_void_p),
                ("workspace", ctypes.c_void_p), ("workspace_bytes", ctypes.c_size_t), ("stream", ctypes.c_void_p),
                ("M", ctypes.c_int32), ("IC", ctypes.c_int32), ("x_stride", ctypes.c_int32),
                ("R_stride", ctypes.c_int32), ("rank", ctypes.c_int32), ("group_size", ctypes.c_int32),
                ("r_mode", ctypes.c_int32), ("out_dtype", ctypes.c_int32), ("kernel", ctypes.c_int32),
                ("n_members", ctypes.c_int32), ("split_k", ctypes.c_int32), ("reserved", ctypes.c_int32),
                ("next", ctypes.c_void_p),     # address of the Group that follows on the stream, or None
                ("push", ctypes.c_void_p),     # address of a Peers struct: push the result to every rank (row-split TP)
                ("push_site", ctypes.c_int32), ("reserved2", ctypes.c_int32),
                ("norm_weight", ctypes.c_void_p), ("residual", ctypes.c_void_p), ("hidden_out", ctypes.c_void_p),
                ("norm_eps", ctypes.c_float), ("reserved3", ctypes.c_int32),
                ("members", Member * MAX_MEMBERS)]


MAX_RANKS = 8


class Peers(ctypes.Structure):
    _fields_ = [("buf", ctypes.c_void_p * MAX_RANKS), ("flag", ctypes.c_void_p * MAX_RANKS), ("epoch", ctypes.c_void_p),
                ("status", ctypes.c_void_p), ("world", ctypes.c_int32), ("rank", ctypes.c_int32),
                ("sites", ctypes.c_int32), ("max_n", ctypes.c_int32), ("ll_buf", ctypes.c_void_p * MAX_RANKS)]


# The same layouts for struct.pack: filling a descriptor field by field through ctypes cost 6 of the 23 microseconds of a module call.
PACK_GROUP = struct.Struct("@6P12i2P2i3Pfi")     # a Group up to its members
PACK_MEMBER = struct.Struct("@6P6ifi")
assert PACK_GROUP.size == Group.members.offset and PACK_MEMBER.size == ctypes.sizeof(Member)

EXPORTS = ("glowq_w4a16_version", "glowq_w4a16_strerror", "glowq_w4a16_last_cuda_error", "glowq_w4a16_dequant",
           "glowq_w4a16_gemv_forward", "glowq_w4a16_gemm_forward", "glowq_w4a16_group_forward",
           "glowq_w4a16_group_forward_many", "glowq_w4a16_group_forward_host", "glowq_w4a16_workspace_bytes",
           "glowq_w4a16_read_status", "glowq_w4a16_gemv_forward_static", "glowq_w4a16_allreduce_f16",
           "glowq_w4a16_allreduce_finish_f16", "glowq_w4a16_quantize", "glowq_w4a16_quantize_indexed")


def library_path() -> str:
    env = os.environ.get("GLOWQ_W4A16_LIB")
    cands = ([env] if env else []) + [os.path.join(_HERE, _LIB_NAME), os.path.join(os.path.dirname(_HERE), _LIB_NAME)]
    for c in cands:
        if c and os.path.exists(c):
            return c
    raise RuntimeError(
        f"{_LIB_NAME} not found (looked in {cands}). Build it with `python -m glowq_b200.build`; "
        "this package has no JIT, Triton or CPU fallback.")


class _Ext:
    """What ``load_w4a16_extension()`` returns: the reference's three callables on torch tensors, plus ``lib``
    (the raw ctypes library) for the fused entry points."""

    def __init__(self, lib: ctypes.CDLL):
        self.lib = lib
        vp, i32, sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
        lib.glowq_w4a16_version.restype = i32
        lib.glowq_w4a16_strerror.restype = ctypes.c_char_p
        lib.glowq_w4a16_strerror.argtypes = [i32]
        lib.glowq_w4a16_last_cuda_error.restype = i32
        lib.glowq_w4a16_dequant.argtypes = [vp, vp, vp, vp, i32, i32, i32, i32, i32, i32, vp]
        lib.glowq_w4a16_quantize.argtypes = [vp, vp, vp, vp, i32, i32, i32, ctypes.c_longlong, vp]
        lib.glowq_w4a16_quantize_indexed.argtypes = [vp, vp, vp, vp, vp, i32, i32, i32, ctypes.c_longlong, vp]
        lib.glowq_w4a16_gemv_forward.argtypes = [vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, i32, i32, vp, sz, vp]
        lib.glowq_w4a16_gemm_forward.argtypes = [vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, i32, i32, i32, vp, sz, vp]
        lib.glowq_w4a16_group_forward.argtypes = [ctypes.POINTER(Group)]
        lib.glowq_w4a16_group_forward_many.argtypes = [ctypes.POINTER(Group), i32]
        lib.glowq_w4a16_group_forward_host.argtypes = [ctypes.POINTER(Group), vp, ctypes.POINTER(vp)]
        lib.glowq_w4a16_workspace_bytes.restype = sz
        lib.glowq_w4a16_workspace_bytes.argtypes = [i32, i32, i32, i32, i32]
        lib.glowq_w4a16_read_status.argtypes = [vp, vp]
        lib.glowq_w4a16_gemv_forward_static.argtypes = [vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, i32, i32, vp]
        lib.glowq_w4a16_allreduce_f16.argtypes = [ctypes.POINTER(Peers), vp, i32, i32, vp]
        lib.glowq_w4a16_allreduce_finish_f16.argtypes = [ctypes.POINTER(Peers), vp, i32, i32, vp]
        if lib.glowq_w4a16_version() != ABI_VERSION:
            raise RuntimeError("libglowq_w4a16.so ABI version mismatch; rebuild with `python -m glowq_b200.build`")
        self._ws = {}               # per device: the piece that the last plain call worked in
        self._pieces = Scratch()
        # the group call on a descriptor that struct.pack made (bytes)
        self.group_forward_packed = ctypes.CFUNCTYPE(i32, ctypes.c_char_p)(("glowq_w4a16_group_forward", lib))

    # ------------------------------------------------------------------ helpers
    def check(self, rc: int, what: str = "glowq_w4a16") -> None:
        if rc != GLOWQ_OK:
            msg = self.lib.glowq_w4a16_strerror(rc).decode()
            if rc == 6:
                msg += f" [cudaError {self.lib.glowq_w4a16_last_cuda_error()}]"
            raise RuntimeError(f"{what}: {msg} (status {rc})")

    def workspace_bytes(self, M: int, IC: int, OC_total: int, rank: int, n_members: int) -> int:
        return int(self.lib.glowq_w4a16_workspace_bytes(M, IC, OC_total, rank, n_members))

    def new_workspace(self, nbytes: int, device) -> torch.Tensor:
        """Zero-initialised workspace (the kernels re-arm their counters themselves after every launch)."""
        return torch.zeros(max(int(nbytes), 256), dtype=torch.uint8, device=device)

    def _scratch(self, device, nbytes: int) -> torch.Tensor:
        ws = self._ws[device.type, device.index] = self._pieces.get(nbytes, device, current_stream_ptr(device))
        return ws

    @staticmethod
    def _check_inputs(x, qweight, scales, qzeros, group_size):
        for t, name in ((x, "inputs"), (qweight, "qweight"), (scales, "scales"), (qzeros, "qzeros")):
            if not t.is_cuda:
                raise RuntimeError(f"{name} must be CUDA")
        if x.dtype != torch.float16:
            raise RuntimeError("inputs must be fp16")
        if qweight.dtype != torch.int32:
            raise RuntimeError("qweight must be int32 (8x int4 packed)")
        if scales.dtype != torch.float16:
            raise RuntimeError("scales must be fp16")
        if qzeros.dtype != torch.int32:
            raise RuntimeError("qzeros must be int32 (8x int4 packed)")
        if x.dim() != 2 or qweight.dim() != 2 or scales.dim() != 2 or qzeros.dim() != 2:
            raise RuntimeError("inputs must be [M, IC]; qweight [OC, packed]; scales [OC, groups]; qzeros [OC, groups_packed]")
        if group_size <= 0 or group_size % 8 != 0:
            raise RuntimeError("group_size must be > 0 and a multiple of 8")
        if scales.size(0) != qweight.size(0) or qzeros.size(0) != qweight.size(0):
            raise RuntimeError("scales / qzeros OC mismatch")

    def _plain(self, fn_name, x, qweight, scales, qzeros, group_size, extra=()):
        self._check_inputs(x, qweight, scales, qzeros, group_size)
        x, qweight, scales, qzeros = (t.contiguous() for t in (x, qweight, scales, qzeros))
        M, IC = x.shape
        OC = qweight.size(0)
        out = torch.empty((M, OC), dtype=torch.float16, device=x.device)
        if M == 0:
            return out
        with torch.cuda.device(x.device):
            need = self.workspace_bytes(M, IC, OC, 0, 1)
            ws = self._scratch(x.device, need)
            stream = torch.cuda.current_stream(x.device).cuda_stream
            fn = getattr(self.lib, fn_name)
            rc = fn(x.data_ptr(), qweight.data_ptr(), scales.data_ptr(), qzeros.data_ptr(), out.data_ptr(), M, IC, OC,
                    int(group_size), *extra, qweight.size(1), qzeros.size(1), scales.size(1), ws.data_ptr(), need, stream)
        self.check(rc, fn_name)
        return out

    # ------------------------------------------------------------------ the reference's three exports
    def w4a16_gemv_forward_cuda(self, x, qweight, scales, qzeros, group_size: int) -> torch.Tensor:
        """[M, OC] fp16 = x . dequant(Q)^T (csrc/gemv_w4a16.cu:146-214)."""
        return self._plain("glowq_w4a16_gemv_forward", x, qweight, scales, qzeros, group_size)

    gemv_w4a16_asym = w4a16_gemv_forward_cuda

    def w4a16_gemm_forward_cuda(self, x, qweight, scales, qzeros, group_size: int, split_k_iters: int = 1) -> torch.Tensor:
        """Same product through the tensor-core kernel (csrc/gemm_w4a16.cu:76-135); split_k_iters is ignored."""
        return self._plain("glowq_w4a16_gemm_forward", x, qweight, scales, qzeros, group_size, (int(split_k_iters),))

    def dequant(self, qweight, scales, qzeros, in_features: int, group_size: int) -> torch.Tensor:
        """[OC, in_features] fp16 dequantised weight, bit-exact with ``_dequant_chunk`` (linear.py:248-253)."""
        qweight, scales, qzeros = (t.contiguous() for t in (qweight, scales, qzeros))
        out = torch.empty((qweight.size(0), in_features), dtype=torch.float16, device=qweight.device)
        with torch.cuda.device(qweight.device):
            rc = self.lib.glowq_w4a16_dequant(qweight.data_ptr(), scales.data_ptr(), qzeros.data_ptr(), out.data_ptr(),
                                              qweight.size(0), in_features, int(group_size), qweight.size(1),
                                              qzeros.size(1), scales.size(1),
                                              torch.cuda.current_stream(qweight.device).cuda_stream)
        self.check(rc, "glowq_w4a16_dequant")
        return out

    def quantize(self, weight, group_size: int):
        """(qweight_i32, qzeros_i32, scales_f16) of a [OC, IC] fp16 weight with unit column stride, in one launch."""
        return self.quantize_indexed(weight, group_size, False)[:3]

    def quantize_indexed(self, weight, group_size: int, index: bool = True):
        """``quantize`` and the group index of every column (int64 [IC]; None unless asked for), in the same launch."""
        oc, ic = weight.shape
        groups = -(-ic // group_size)
        qweight = torch.empty((oc, groups * (group_size // 8)), dtype=torch.int32, device=weight.device)
        qzeros = torch.empty((oc, (groups + 7) // 8), dtype=torch.int32, device=weight.device)
        scales = torch.empty((oc, groups), dtype=torch.float16, device=weight.device)
        gid = torch.empty(ic, dtype=torch.int64, device=weight.device) if index else None
        args = (weight.data_ptr(), qweight.data_ptr(), qzeros.data_ptr(), scales.data_ptr(),
                gid.data_ptr() if index else None, oc, ic, int(group_size), max(weight.stride(0), ic), current_stream_ptr(weight.device))
        if current_device() == weight.device.index:
            rc = self.lib.glowq_w4a16_quantize_indexed(*args)
        else:
            with torch.cuda.device(weight.device):
                rc = self.lib.glowq_w4a16_quantize_indexed(*args)
        self.check(rc, "glowq_w4a16_quantize")
        return qweight, qzeros, scales, gid


def int32(v: int) -> int:
    """What a c_int32 field keeps of ``v`` (the stride of a single row may be anything)."""
    return v if -0x80000000 <= v <= 0x7FFFFFFF else ctypes.c_int32(v).value


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def current_stream_ptr(device: torch.device) -> int:
    """The cudaStream_t that PyTorch's current stream of ``device`` stands for."""
    if _raw_stream is not None:
        return _raw_stream(device.index)
    return torch.cuda.current_stream(device).cuda_stream


current_device = getattr(torch._C, "_cuda_getDevice", torch.cuda.current_device)   # (where CUDA is in use already)
_is_capturing = getattr(torch._C, "_cuda_isCurrentStreamCapturing", torch.cuda.is_current_stream_capturing)


class Scratch:
    """Zeroed device memory that one module's launches work in: counters, which every launch leaves at zero, and partial sums.

    Launches on one stream take turns on one piece, whatever their sizes; every stream has a piece of its own.  A CUDA graph
    keeps the addresses it was captured with, so what a capture has used belongs to the captures of that stream from then on
    and is held as long as this object, and other calls get another piece.  A capture takes over a piece that its thread's
    calls have used before (the warm-up), whose counters are zero; where there is none, a captured launch gets memory of the
    graph's own, which the graph zeroes.  Graphs captured on one stream share a piece: they are not to be replayed at the same time."""

    __slots__ = ("_pieces", "_makers", "_kept", "_largest")
    MAX_STREAMS = 8      # streams that keep a piece; beyond, the oldest is given back (its memory is freed in its stream's order)

    def __init__(self):
        self._pieces = {}      # (device, stream, capturing): uint8 tensor
        self._makers = {}      # the same keys: the thread that asked for the piece
        self._kept = []        # pieces of captures that later ones outgrew
        self._largest = 0

    def __reduce__(self):      # a copied or loaded module starts without any
        return Scratch, ()

    def get(self, nbytes: int, device: torch.device, stream: int) -> torch.Tensor:
        """At least ``nbytes`` for a launch on ``stream``, the current stream of ``device``, which is the current device."""
        key = (device.index, stream, stream != 0 and _is_capturing())   # (the default stream, 0, cannot be captured)
        piece = self._pieces.get(key)
        if piece is None or piece.numel() < nbytes:
            piece = self._more(nbytes, device, key)
        return piece

    def _more(self, nbytes: int, device: torch.device, key) -> torch.Tensor:
        pieces, me = self._pieces, threading.get_ident()
        if key[2]:
            mine = [k for k, p in list(pieces.items())
                    if not k[2] and k[0] == key[0] and p.numel() >= nbytes and self._makers.get(k) == me]
            mine.sort(key=lambda k: k[1] != key[1])
            piece = pieces.pop(mine[0], None) if mine else None
            if piece is None:
                return torch.zeros(nbytes, dtype=torch.uint8, device=device)
            if key in pieces:
                self._kept.append(pieces[key])
        else:
            # (sizes that outgrow one another grow by half at least, so that what captures hold on to is a few times the largest)
            size = max(nbytes, 256)
            if size > self._largest:
                self._largest = size = max(size, self._largest * 3 // 2)
            piece = torch.zeros(size, dtype=torch.uint8, device=device)
            streams = [k for k in list(pieces) if not k[2] and k != key]
            if len(streams) >= self.MAX_STREAMS:
                pieces.pop(streams[0], None)
        self._makers[key] = me
        pieces[key] = piece
        return piece


class RRows:
    """Room for r = B x, [tokens, rank] fp16, as ``Scratch`` gives it: by streams, and a captured graph's own."""

    __slots__ = ("_scratch", "_last")

    def __init__(self):
        self._scratch = Scratch()
        self._last = None

    def __reduce__(self):
        return RRows, ()

    def rows(self, m: int, rank: int, device: torch.device) -> torch.Tensor:
        stream = 0
        if device.type == "cuda":
            if current_device() != device.index:     # (whether the stream captures is asked of the current device)
                with torch.cuda.device(device):
                    return self.rows(m, rank, device)
            stream = current_stream_ptr(device)
        piece = self._scratch.get(2 * max(m, 16) * rank, device, stream)
        last = self._last
        if last is None or last[0] is not piece or last[1] != (m, rank):
            self._last = last = (piece, (m, rank), piece[:2 * m * rank].view(torch.float16).view(m, rank))
        return last[2]


_ext: Optional[_Ext] = None


def load_w4a16_extension(verbose: Optional[bool] = None) -> _Ext:
    """Load (once) and return the kernel library front end (src/cuda_w4a16/kernels.py:16-59)."""
    global _ext
    if _ext is None:
        path = library_path()
        try:
            lib = ctypes.CDLL(path)
        except OSError as exc:
            raise RuntimeError(f"failed to load {path}: {exc}. Rebuild with `python -m glowq_b200.build`.") from exc
        missing = [n for n in EXPORTS if not hasattr(lib, n)]
        if missing:
            raise RuntimeError(f"{path} lacks symbols {missing}")
        _ext = _Ext(lib)
        if verbose:
            print(f"[glowq_b200] loaded {path}")
    return _ext


__all__ = ["load_w4a16_extension"]
