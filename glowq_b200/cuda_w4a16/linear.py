"""Drop-in ``cuda_w4a16.linear``: RTN uint4 quantiser/packer, the replacement module ``CudaW4A16Linear``
(same constructor, buffers, attributes and ``from_float`` as src/cuda_w4a16/linear.py:91-276) and the
model-conversion pass ``convert_to_cuda_w4a16`` (linear.py:279-293), on top of the sm_100a C-ABI library.

Differences from the reference, all on the host side of the same interface:
* forward runs only on CUDA tensors of an sm_100 device; there is no pure-torch or CPU path;
* the kernel choice knobs W4A16_KERNEL_OUT_DTYPE / W4A16_GEMV_M_MAX / W4A16_FORCE_GEMM / W4A16_FORCE_GEMV are
  read once when the module is built (the reference re-reads the environment on every call, linear.py:172-177);
  W4A16_GEMV_M_MAX has no built-in default of 128 here: unset, the library switches kernels where it measured the
  cross-over (2 to 8 tokens by an estimate of both, tensor cores above);
  the dequant-cache / chunk / JIT knobs belong to fallbacks that do not exist here;
* output and scratch buffers are caller-side torch tensors; the library allocates nothing.
"""
from __future__ import annotations

import math
import os
from typing import Optional

import torch
import torch.nn as nn

from . import kernels as K
from .kernels import load_w4a16_extension

_TRUE = {"1", "true", "yes", "y", "on"}


def _env_flag(*names: str) -> bool:
    for n in names:
        v = os.environ.get(n)
        if v is not None:
            return v.lower() in _TRUE
    return False


def _env_int(*names: str, default: int) -> int:
    for n in names:
        v = os.environ.get(n)
        if v:
            return int(v)
    return int(default)


def _get_kernel_out_dtype() -> torch.dtype:
    """W4A16_KERNEL_OUT_DTYPE (legacy MIXED_KERNEL_OUT_DTYPE), default fp32 (linear.py:29-39)."""
    v = os.environ.get("W4A16_KERNEL_OUT_DTYPE", os.environ.get("MIXED_KERNEL_OUT_DTYPE", "fp32")).lower()
    return torch.float16 if v in ("fp16", "float16", "half") else torch.float32


def _pack_int4_to_int32(u4: torch.Tensor) -> torch.Tensor:
    """[..., 8] uint8 codes -> [...] int32 with code j in bits [4j, 4j+4) (linear.py:42-46)."""
    if u4.dtype != torch.uint8 or u4.shape[-1] != 8:
        raise ValueError("expected uint8 codes with a trailing axis of 8")
    word = torch.zeros(u4.shape[:-1], dtype=torch.int32, device=u4.device)
    for j in range(8):
        word |= u4[..., j].to(torch.int32) << (4 * j)   # bit 31 wraps into the sign, as int32 arithmetic does
    return word


def _unpack_int4_i32(packed_i32: torch.Tensor, total_vals: int) -> torch.Tensor:
    """Row-wise inverse of the packer (linear.py:49-54)."""
    p = packed_i32.contiguous().to(torch.int32)
    cols = [((p >> (4 * j)) & 0xF).to(torch.uint8) for j in range(8)]
    return torch.stack(cols, dim=-1).reshape(p.size(0), -1)[:, :total_vals].contiguous()


def _device_quantises(device: torch.device) -> bool:
    """The library's kernels run on compute capability 10.0 alone (sm_100a code).  Converting a model needs no library: where
    it is missing or of another version, the forward call says so and the quantiser is the torch expression."""
    if torch.cuda.get_device_capability(device) != (10, 0):
        return False
    try:
        load_w4a16_extension()
    except RuntimeError:
        return False
    return True


def _kernel_quantises(weight: torch.Tensor, group_size: int) -> bool:
    """The one-launch quantiser takes what a conversion hands over: a plain fp16 matrix on an sm_100 device in groups of
    128.  Everything else (CPU tensors, other types, group sizes and devices, no library) is the torch expression, the same bits.
    Measured for the seven linears of a Llama-2-13B layer: 29.1 ms with the torch expression and the buffers of the
    module made on the host, 0.27 ms with this launch (0.21 ms of it on the GPU; the modules are built around its buffers)."""
    return (group_size == 128 and weight.is_cuda and weight.dtype == torch.float16 and type(weight) is torch.Tensor
            and not weight.requires_grad and weight.numel() > 0 and weight.stride(1) == 1
            and weight.stride(0) >= weight.shape[1] and _device_quantises(weight.device))


def _quantize_per_group_w4(weight: torch.Tensor, group_size: int):
    """RTN asymmetric uint4 per (row, group) in the weight's own (fp16) arithmetic; returns
    (qweight_i32 [OC, ICp/8], qzeros_i32 [OC, ceil(G/8)], scales_f16 [OC, G], ICp) exactly as
    src/cuda_w4a16/linear.py:57-88 does: scale = (max-min)/15, zero = round(-min/scale) clamped to [0,15],
    code = round(w/scale + zero) clamped to [0,15]; columns padded with zeros to a whole group; unused
    zero-point nibbles hold 8."""
    if group_size % 8 != 0:
        raise ValueError("group_size must be multiple of 8 for int32 int4 packing")
    oc, ic = weight.shape
    if _kernel_quantises(weight, group_size):
        qweight, qzeros, scales = load_w4a16_extension().quantize(weight, group_size)
        return qweight, qzeros, scales, scales.shape[1] * group_size
    rem = ic % group_size
    if rem:
        weight = torch.nn.functional.pad(weight, (0, group_size - rem))
        ic = weight.shape[1]
    n_groups = ic // group_size
    grouped = weight.reshape(oc, n_groups, group_size)
    lo = grouped.amin(dim=-1)
    hi = grouped.amax(dim=-1)
    scales = ((hi - lo) / 15.0).clamp(min=1e-8)
    zeros = (-lo / scales).round().clamp(0, 15)
    codes = (grouped / scales[..., None] + zeros[..., None]).round().clamp(0, 15).to(torch.uint8)
    qweight = _pack_int4_to_int32(codes.view(oc, n_groups, group_size // 8, 8)).reshape(oc, ic // 8)

    words = (n_groups + 7) // 8
    z8 = torch.nn.functional.pad(zeros.to(torch.uint8), (0, words * 8 - n_groups), value=8)
    qzeros = _pack_int4_to_int32(z8.view(oc, words, 8))
    return qweight.contiguous(), qzeros.contiguous(), scales.to(torch.float16).contiguous(), ic


class CudaW4A16Linear(nn.Module):
    """W4A16 linear on packed int4 weights (src/cuda_w4a16/linear.py:91-276)."""

    def __init__(self, in_features: int, out_features: int, group_size: int = 128, bias: bool = False):
        super().__init__()
        self._configure(in_features, out_features, group_size)
        self.register_buffer("qweight_i32", torch.empty(self.out_features, (self.in_features + 7) // 8, dtype=torch.int32))
        self.register_buffer("qzeros_i32", torch.empty(self.out_features, max(1, self.groups_packed), dtype=torch.int32))
        self.register_buffer("scales_f16", torch.empty(self.out_features, self.groups, dtype=torch.float16))
        self.register_buffer("gid", torch.arange(self.in_features, dtype=torch.long) // self.group_size, persistent=False)
        self.bias = nn.Parameter(torch.empty(self.out_features, dtype=torch.float16)) if bias else None

    def _configure(self, in_features: int, out_features: int, group_size: int) -> None:
        """Sizes and knobs.  (Plain values go to the module's dictionary at once: nn.Module.__setattr__ takes microseconds each.)"""
        in_features, out_features, group_size = int(in_features), int(out_features), int(group_size)
        if group_size <= 0 or group_size % 8 != 0:
            raise ValueError("group_size must be > 0 and a multiple of 8 for GlowQ int32 int4 packing")
        groups = math.ceil(in_features / group_size)
        self.__dict__.update(
            in_features=in_features, out_features=out_features, group_size=group_size, groups=groups, groups_packed=(groups + 7) // 8,
            _ext=None,
            # -1: the knob is unset and the library's own switch-over applies
            _gemv_threshold=_env_int("W4A16_GEMV_M_MAX", "CUDA_MIXED_GEMV_M_MAX", default=-1),
            _force_gemm=_env_flag("W4A16_FORCE_GEMM", "CUDA_MIXED_FORCE_GEMM"),
            _force_gemv=_env_flag("W4A16_FORCE_GEMV", "CUDA_MIXED_FORCE_GEMV") or _env_flag("W4A16_USE_GEMV"),
            _out_dtype=_get_kernel_out_dtype(), _check_status=_env_flag("GLOWQ_CHECK_STATUS"))

    def extra_repr(self) -> str:
        return (f"in_features={self.in_features}, out_features={self.out_features}, "
                f"group_size={self.group_size}, bias={self.bias is not None}")

    # ------------------------------------------------------------------ plumbing
    def _get_ext(self):
        if self._ext is None:
            self._ext = load_w4a16_extension()
        return self._ext

    def kernel_choice(self, m: int) -> int:
        """Which kernel a call with ``m`` tokens asks for (linear.py:172-181): a FORCE knob wins; otherwise an
        explicitly set W4A16_GEMV_M_MAX sends ``m <= W4A16_GEMV_M_MAX`` to the weight-streaming kernel and anything
        larger to the tensor-core kernel; with the knob unset the library's own switch-over (2 to 8 tokens) applies."""
        if self._force_gemm:
            return K.KERNEL_GEMM
        if self._force_gemv:
            return K.KERNEL_GEMV
        if self._gemv_threshold >= 0:
            return K.KERNEL_GEMV if m <= self._gemv_threshold else K.KERNEL_GEMM
        return K.KERNEL_AUTO

    def _flatten_input(self, x: torch.Tensor):
        if x.shape[-1] != self.in_features:
            raise ValueError(f"Input dim mismatch: got {x.shape[-1]}, expected {self.in_features}")
        if not x.is_cuda:
            raise RuntimeError("CudaW4A16Linear runs on CUDA (sm_100) tensors only; there is no CPU path")
        x2d = x if x.dim() == 2 else x.reshape(-1, x.shape[-1])
        if x2d.dtype != torch.float16:
            x2d = x2d.to(torch.float16)
        return x2d.contiguous()

    def fill_member(self, mem: "K.Member", out: torch.Tensor, L: Optional[torch.Tensor] = None, alpha: float = 0.0):
        """Fill a descriptor's ``Member`` in place."""
        K.PACK_MEMBER.pack_into(mem, 0, *self.pack_member(out, L, float(alpha)))

    def pack_member(self, out: torch.Tensor, L: Optional[torch.Tensor] = None, alpha: float = 0.0) -> tuple:
        """The fields of a ``Member`` in order (``kernels.PACK_MEMBER``).  Buffers are looked up in their dictionary:
        ``nn.Module.__getattr__`` takes half a microsecond each."""
        bufs = self._buffers
        try:
            qw, sc, qz = bufs["qweight_i32"], bufs["scales_f16"], bufs["qzeros_i32"]
        except KeyError:
            qw, sc, qz = self.qweight_i32, self.scales_f16, self.qzeros_i32
        bias = self._parameters["bias"] if "bias" in self._parameters else self.bias
        # (stride()[0]: half the time of stride(0))
        return (qw.data_ptr(), sc.data_ptr(), qz.data_ptr(), bias.data_ptr() if bias is not None else 0,
                L.data_ptr() if L is not None else 0, out.data_ptr(), self.out_features, qw.stride()[0], qz.stride()[0],
                sc.stride()[0], L.stride()[0] if L is not None else 0, out.stride()[0], alpha, 0)

    def _work(self, m: int, rank: int, device, stream: int):
        """What a call on ``stream`` works in, and how much of it is this call's: the slices of K follow from the size, so that a
        larger call before leaves the results as they are."""
        own = self.__dict__
        needs = own.get("_needs")
        if needs is None:
            needs = own.setdefault("_needs", {})
        need = needs.get((m, rank))
        if need is None:
            if len(needs) > 4096:
                needs.clear()
            need = needs[m, rank] = self._get_ext().workspace_bytes(m, self.in_features, self.out_features, rank, 1)
        scratch = own.get("_scratch")
        if scratch is None:
            scratch = own.setdefault("_scratch", K.Scratch())
        return scratch.get(need, device, stream), need

    def workspace_for(self, m: int, rank: int, device) -> torch.Tensor:
        return self._work(m, rank, device, K.current_stream_ptr(device))[0]

    def launch(self, x2d: torch.Tensor, *, L=None, R=None, r_buf=None, r_mode=K.R_NONE, alpha=0.0, push=None,
               push_site: int = 0) -> torch.Tensor:
        """One library call: this linear, optionally with its low-rank correction folded in.  ``push``: a
        ``glowq_b200.tp.PeerAllReduce`` - a row-split tensor-parallel shard then also stores its result into every
        rank's staging slot of ``push_site`` (complete the sum with ``push.finish(out, push_site)``)."""
        ext = self._get_ext()
        m, dev = x2d.size(0), x2d.device
        out = torch.empty(m, self.out_features, dtype=self._out_dtype, device=dev)
        if m == 0:
            return out
        if K.current_device() == dev.index:
            self._launch(ext, x2d, out, m, dev, L, R, r_buf, r_mode, alpha, push, push_site)
        else:
            with torch.cuda.device(dev):
                self._launch(ext, x2d, out, m, dev, L, R, r_buf, r_mode, alpha, push, push_site)
        return out

    def _launch(self, ext, x2d, out, m, dev, L, R, r_buf, r_mode, alpha, push, push_site) -> None:
        rank = r_ptr = r_stride = rb_ptr = 0
        if r_mode != K.R_NONE:
            rank = int(L.size(1))
            if R is not None:
                r_ptr, r_stride = R.data_ptr(), R.stride(0)
            rb_ptr = r_buf.data_ptr()
        else:
            L = None
        stream = K.current_stream_ptr(dev)
        ws, need = self._work(m, rank, dev, stream)
        grp = K.PACK_GROUP.pack(
            x2d.data_ptr(), r_ptr, rb_ptr, ws.data_ptr(), need, stream, m, self.in_features, K.int32(x2d.stride(0)), r_stride, rank,
            self.group_size, r_mode, K.OUT_F32 if self._out_dtype == torch.float32 else K.OUT_F16, self.kernel_choice(m), 1, 0, 0, 0,
            push.descriptor_address() if push is not None else 0, int(push_site) if push is not None else 0, 0, 0, 0, 0, 0.0, 0)
        ext.check(ext.group_forward_packed(grp + K.PACK_MEMBER.pack(*self.pack_member(out, L, alpha))), "glowq_w4a16_group_forward")
        if self._check_status:   # debugging aid: synchronises the stream after every launch
            ext.check(ext.lib.glowq_w4a16_read_status(ws.data_ptr(), stream), "device status")

    # ------------------------------------------------------------------ reference-named entry points
    def _run_cuda_gemv(self, x2d: torch.Tensor) -> torch.Tensor:
        return self._get_ext().w4a16_gemv_forward_cuda(x2d, self.qweight_i32, self.scales_f16, self.qzeros_i32,
                                                       int(self.group_size))

    def _run_cuda_gemm(self, x2d: torch.Tensor) -> torch.Tensor:
        return self._get_ext().w4a16_gemm_forward_cuda(x2d, self.qweight_i32, self.scales_f16, self.qzeros_i32,
                                                       int(self.group_size), _env_int("W4A16_SPLIT_K_ITERS", default=1))

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        out = self.launch(self._flatten_input(x))
        return out if x.dim() == 2 else out.reshape(*x.shape[:-1], self.out_features)

    def _dequant_full_weight_fallback(self) -> torch.Tensor:
        """[OC, in_features] fp16 dequantised weight (bit-exact with linear.py:240-253), on the device."""
        return self._get_ext().dequant(self.qweight_i32, self.scales_f16, self.qzeros_i32, self.in_features,
                                       self.group_size)

    @classmethod
    def from_float(cls, linear_layer: nn.Linear, group_size: int):
        dev = linear_layer.weight.device
        if cls is CudaW4A16Linear and cls.__init__ is _CONSTRUCTOR:
            # The same module without the buffers that the constructor makes only for them to be replaced: made on the host, moved
            # and replaced they took longer than quantising (140 us a module; 37 so, with the group index from the quantiser's launch).
            mod = cls.__new__(cls)
            nn.Module.__init__(mod)
            mod._configure(linear_layer.in_features, linear_layer.out_features, group_size)
            weight = linear_layer.weight.data.to(torch.float16)
            if weight.dim() == 2 and weight.shape[1] == mod.in_features and _kernel_quantises(weight, group_size):
                qweight, qzeros, scales, gid = load_w4a16_extension().quantize_indexed(weight, group_size)
            else:
                qweight, qzeros, scales, _ = _quantize_per_group_w4(weight, group_size)
                gid = torch.arange(mod.in_features, dtype=torch.long, device=dev) // mod.group_size
            if _BUFFER_HOOKS is not None and not _BUFFER_HOOKS:
                mod._buffers.update(qweight_i32=qweight, qzeros_i32=qzeros, scales_f16=scales, gid=gid)
                mod._non_persistent_buffers_set.add("gid")
            else:
                for name, t in (("qweight_i32", qweight), ("qzeros_i32", qzeros), ("scales_f16", scales)):
                    mod.register_buffer(name, t)
                mod.register_buffer("gid", gid, persistent=False)
            if linear_layer.bias is None:
                mod.__dict__["bias"] = None
            else:
                mod.bias = nn.Parameter(torch.empty(mod.out_features, dtype=torch.float16, device=dev))
                mod.bias.data.copy_(linear_layer.bias.data.to(torch.float16))
            return mod
        with torch.device(dev):    # a subclass, or a constructor put in the place of this one
            mod = cls(linear_layer.in_features, linear_layer.out_features, group_size,
                      bias=linear_layer.bias is not None).to(dev)
        mod.qweight_i32, mod.qzeros_i32, mod.scales_f16, _ = _quantize_per_group_w4(
            linear_layer.weight.data.to(torch.float16), group_size)
        if linear_layer.bias is not None:
            mod.bias.data.copy_(linear_layer.bias.data.to(torch.float16))
        return mod


_CONSTRUCTOR = CudaW4A16Linear.__init__
_BUFFER_HOOKS = getattr(nn.modules.module, "_global_buffer_registration_hooks", None)   # of register_module_buffer_registration_hook


def convert_to_cuda_w4a16(model: nn.Module, group_size: int = 128) -> nn.Module:
    """Replace every ``nn.Linear`` whose qualified name does not contain "lm_head" (linear.py:279-293).
    A layer whose conversion raises keeps its original module, as in the reference; the failures are
    collected in ``model._w4a16_conversion_errors`` instead of vanishing."""
    errors = {}
    targets = [(n, m) for n, m in model.named_modules() if isinstance(m, nn.Linear) and "lm_head" not in n]
    for name, lin in targets:
        parent = model
        *path, leaf = name.split(".")
        for part in path:
            parent = getattr(parent, part)
        try:
            setattr(parent, leaf, CudaW4A16Linear.from_float(lin, group_size))
        except Exception as exc:  # noqa: BLE001 - parity with the reference's keep-going behaviour
            errors[name] = repr(exc)
    try:
        model._w4a16_conversion_errors = errors
    except Exception:  # noqa: BLE001
        pass
    if torch.cuda.is_available():
        torch.cuda.empty_cache()
    return model
