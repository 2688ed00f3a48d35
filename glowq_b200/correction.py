"""Low-rank correction wrapper and patchers, same surface as GlowQ's step3 scripts
(``AddSVDCorrection``, ``MiniGroupCache``, ``patch_svd_correction_wrappers``: src/step3_eval_dataset.py:417-605;
``patch_svd_correction_wrappers_cumulative``, the GlowQ-S enable mask: src/restoration/step4_evaluate_cumulative.py:99-154).

The reference wrapper runs ``inner(x)``, then ``F.linear(x, B_q)`` (or a cache hit), ``F.linear(r, A_q)`` and an
in-place add: 3-4 launches.  Here the whole of ``z + alpha * (x B_q^T) A_q^T`` is ONE library launch per module: the
wrapper only decides, from the role and the cache state, whether that launch computes r = B_q x and leaves it in the
group's device buffer (roles q / gate / solo) or reads it from there (roles k / v / up on a hit)."""
from __future__ import annotations

import ctypes
import os
import warnings
import weakref
from typing import Dict, Optional, Set

import torch
import torch.nn as nn

from .cuda_w4a16 import kernels as K
from .cuda_w4a16.linear import CudaW4A16Linear

try:  # tqdm only decorates the patch loop, as in the reference
    from tqdm import tqdm as _tqdm
except Exception:  # noqa: BLE001
    def _tqdm(it, **_):
        return it

_pack_member_into, _MEMBER_BYTES, _MEMBERS_AT = K.PACK_MEMBER.pack_into, K.PACK_MEMBER.size, K.Group.members.offset

_ALL_CACHES: "weakref.WeakSet[MiniGroupCache]" = weakref.WeakSet()


def _fuse_enabled() -> bool:
    return os.environ.get("GLOWQ_FUSE_GROUPS", "1").lower() not in ("0", "false", "no", "off")


def clear_group_cache() -> None:
    """Invalidate every live group cache (a no-op placeholder in src/step3_eval_dataset.py:409-411)."""
    for c in list(_ALL_CACHES):
        c.clear()


def _x_key(x: torch.Tensor):
    return (x.data_ptr(), x.shape, x.dtype, x._version)


def _inner(w: "AddSVDCorrection") -> CudaW4A16Linear:
    """``w.inner`` (``nn.Module.__getattr__`` takes half a microsecond)."""
    inner = w._modules.get("inner")
    return w.inner if inner is None else inner


class MiniGroupCache:
    """Hand-off of r = B_shared . x between the members of a group (src/step3_eval_dataset.py:417-444):
    the producer (q / gate) calls ``set(r, uses)``; each consumer (k, v / up) calls ``consume()`` and gets
    ``(r, True)`` until ``uses`` run out.  Here r lives in a device buffer owned by the cache that the kernel
    writes and reads directly.  A consumer may pass the identity of its input; a hit then also requires that
    the producer saw the same tensor (the reference trusts call order alone)."""

    __slots__ = ("r", "valid", "uses_left", "_key", "_buf", "__weakref__")

    def __init__(self):
        self.r: Optional[torch.Tensor] = None
        self.valid: bool = False
        self.uses_left: int = 0
        self._key = None
        self._buf = K.RRows()
        _ALL_CACHES.add(self)

    def buffer(self, m: int, rank: int, device) -> torch.Tensor:
        if not isinstance(self._buf, K.RRows):      # loaded from a file of an earlier form
            self._buf = K.RRows()
        return self._buf.rows(m, rank, device)

    def set(self, r: torch.Tensor, uses: int, key=None):
        self.r = r
        self.valid = True
        self.uses_left = uses
        self._key = key

    def consume(self, key=None):
        if self.valid and self.uses_left > 0 and (key is None or self._key is None or key == self._key):
            self.uses_left -= 1
            out = self.r
            if self.uses_left == 0:
                self.valid = False
                self.r = None
            return out, True
        return None, False

    def clear(self):
        self.r = None
        self.valid = False
        self.uses_left = 0
        self._key = None


class GroupLauncher:
    """One library launch for all wrapped members of a group (q/k/v, gate/up) or for a solo member.

    HF decoder layers call the members of a group back to back on the same tensor (q, k, v:
    models/llama/modeling_llama.py, ``LlamaAttention.forward``; gate before up: ``LlamaMLP.forward``) - the order the
    reference's cache relies on (src/step3_eval_dataset.py:481-504).  The patchers therefore give every group a
    launcher: the FIRST member's forward issues ONE ``glowq_w4a16_group_forward`` for all members and keeps the other
    members' outputs; their forwards return them when they are called with the same tensor (identity, shape, dtype and
    version), and fall back to a launch of their own otherwise.  Outputs are fresh tensors on every call, as in the
    reference.  The workspace and r are one piece of scratch (``kernels.Scratch``) that launches of all token counts share:
    a piece for each of them would be 17 MB a group and prompt length.  ``next_launcher`` (set by the patchers in model
    order) names the launch that follows, for the library's ``next`` hint."""

    def __init__(self, members):
        members = list(members)               # AddSVDCorrection wrappers, first = producer (q / gate / solo)
        first = members[0]
        inner0 = first.inner
        self._reset(members, None, len(members) <= K.MAX_MEMBERS and all(
            w.inner.in_features == inner0.in_features and w.inner.group_size == inner0.group_size
            and w.inner._out_dtype == inner0._out_dtype and w.B_q.shape == first.B_q.shape
            and w.A_q.size(1) == first.A_q.size(1) for w in members))

    def _reset(self, members, next_launcher, usable: bool) -> None:
        # The wrappers hold their launcher, and it names them and its successor weakly: a model that is dropped gives its memory back
        # then and there, not when the cycle collector runs.
        self._refs = [weakref.ref(w) for w in members]
        self.next_launcher = next_launcher
        self.usable = usable
        self._scratch = K.Scratch()
        self._sizes: Dict[tuple, int] = {}    # the workspace's bytes by (tokens, device, rank)
        self._call: Optional[K.Group] = None  # the descriptor of the last launch, which the launch in front names as the one that follows
        self._call_key: Optional[tuple] = None
        self._call_r: Optional[tuple] = None
        self._call_weights: list = []         # (buffers, name, address) of the right factor and the packed weights
        self._pending: Dict[int, torch.Tensor] = {}
        self._pending_key = None

    @property
    def members(self) -> list:
        """The wrappers that are alive, the producer first."""
        return [w for w in (ref() for ref in self._refs) if w is not None]

    @property
    def next_launcher(self) -> Optional["GroupLauncher"]:
        return None if self._next is None else self._next()

    @next_launcher.setter
    def next_launcher(self, launcher: Optional["GroupLauncher"]) -> None:
        self._next = None if launcher is None else weakref.ref(launcher)

    def __getstate__(self):      # a copied or saved launcher has the same place in its model, and nothing of its launches
        return self.members, self.next_launcher, self.usable and len(self.members) == len(self._refs)

    def __setstate__(self, state):
        if isinstance(state, dict):      # saved when launchers named their members strongly
            state = state["members"], state["next_launcher"], state["usable"]
        self._reset(*state)

    def _describe(self, key: tuple, inners) -> None:
        """What calls of one size have in common: the descriptor's fixed fields."""
        m, dev, rank, dtype = key
        if self._call is None:
            call = K.Group()
            self._call_at = ctypes.addressof(call)
            self._call = call
        grp, lin = self._call, inners[0]
        grp.M, grp.IC, grp.rank, grp.group_size = m, lin.in_features, rank, lin.group_size
        grp.r_mode, grp.kernel, grp.n_members = K.R_COMPUTE, lin.kernel_choice(m), len(inners)
        grp.out_dtype = K.OUT_F32 if dtype == torch.float32 else K.OUT_F16
        need = self._sizes.get((m, dev, rank))
        if need is None:
            if len(self._sizes) > 4096:
                self._sizes.clear()
            need = lin._get_ext().workspace_bytes(m, lin.in_features, sum(i.out_features for i in inners), rank, len(inners))
            self._sizes[m, dev, rank] = need
        self._call_key, self._call_need, self._call_total = key, need, need + 2 * m * rank   # (a multiple of 256 bytes, and r)

    def descriptor_address(self, m: int, device, dtype=None) -> Optional[int]:
        """The descriptor of the last launch, for the ``next`` hint of the one in front.  None before a launch of so many tokens, and
        where the weights have moved since: what the descriptor points to may be unmapped by now."""
        key = self._call_key
        if key is None or key[1] != device.index or (m, key[1], key[2]) not in self._sizes:
            return None
        for buffers, name, at in self._call_weights:
            t = buffers.get(name)
            if t is None or t.data_ptr() != at:
                return None
        return self._call_at

    def run(self, x: torch.Tensor, members: Optional[list] = None) -> torch.Tensor:
        """Called by the first member: launch the whole group, keep the other members' outputs, return its own."""
        members = members or self.members
        first = members[0]
        inners = [_inner(w) for w in members]
        inner = inners[0]
        x2d = inner._flatten_input(x)
        m, dev, dtype = x2d.shape[0], x2d.device, inner._out_dtype
        outs = [torch.empty(m, lin.out_features, dtype=dtype, device=dev) for lin in inners]
        self._pending.clear()
        key = _x_key(x)
        if m > 0:
            if K.current_device() == dev.index:
                r = self._launch(x2d, members, inners, outs, m, dev, dtype)
            else:
                with torch.cuda.device(dev):
                    r = self._launch(x2d, members, inners, outs, m, dev, dtype)
            self._keep = x2d          # the launch reads x2d asynchronously
            if r is not None:
                first.group_cache.set(r, len(members) - 1, key)
        flat = x.dim() == 2
        for w, o in zip(members[1:], outs[1:]):
            self._pending[id(w)] = o if flat else o.reshape(*x.shape[:-1], o.size(1))
        self._pending_key = key
        return outs[0] if flat else outs[0].reshape(*x.shape[:-1], inner.out_features)

    def _launch(self, x2d, members, inners, outs, m, dev, dtype) -> Optional[torch.Tensor]:
        """The launch; r, where the members' cache hands it on."""
        first, inner = members[0], inners[0]
        factors, name = first._buffers, "B_q"
        R = factors.get(name)
        if R is None:
            factors, R = first._parameters, first.B_q
        rank = R.shape[0]
        key = (m, dev.index, rank, dtype)
        if key != self._call_key:
            self._describe(key, inners)
        grp, ext = self._call, inner._get_ext()
        stream = K.current_stream_ptr(dev)
        piece = self._scratch.get(self._call_total, dev, stream)
        at, R_at = piece.data_ptr(), R.data_ptr()
        grp.x, grp.x_stride = x2d.data_ptr(), x2d.stride()[0]
        grp.R, grp.R_stride = R_at, R.stride()[0]
        grp.workspace, grp.workspace_bytes, grp.r_buf, grp.stream = at, self._call_need, at + self._call_need, stream
        weights, place = [(factors, name, R_at)], _MEMBERS_AT
        for w, lin, o in zip(members, inners, outs):
            alpha = float(w.alpha_svd)
            if alpha != 0.0 and not w._mismatch:
                L = w._buffers.get("A_q")
                if L is None:
                    L = w.A_q
                fields = lin.pack_member(o, L, alpha)
                if fields[10] != rank and L.shape[1] != rank:      # (the row stride: other than the rank in a part of a larger factor)
                    raise RuntimeError(f"a left factor has rank {L.shape[1]}, the group's right factor {rank}")
            else:
                fields = lin.pack_member(o)
            _pack_member_into(grp, place, *fields)
            place += _MEMBER_BYTES
            weights.append((lin._buffers, "qweight_i32", fields[0]))
        self._call_weights = weights
        nxt = self._next and self._next()
        grp.next = nxt.descriptor_address(m, dev) if nxt is not None else None
        rc = ext.lib.glowq_w4a16_group_forward(grp)
        if rc:
            ext.check(rc, "glowq_w4a16_group_forward")
        if inner._check_status:
            ext.check(ext.lib.glowq_w4a16_read_status(at, stream), "device status")
        if not first.is_group or first.group_cache is None:
            return None
        r = self._call_r
        if r is None or r[0] is not piece or r[1] is not self._call_key:
            need, total = self._call_need, self._call_total
            self._call_r = r = (piece, self._call_key, piece[need:total].view(torch.float16).view(m, rank))
        return r[2]

    def forget(self) -> None:
        self._pending.clear()
        self._pending_key = None

    def take(self, wrapper: "AddSVDCorrection", x: torch.Tensor) -> Optional[torch.Tensor]:
        """A later member's output of the launch the first member issued for this very input, or None."""
        if self._pending_key is None or _x_key(x) != self._pending_key:
            return None
        out = self._pending.pop(id(wrapper), None)
        if out is not None and wrapper.group_cache is not None:
            wrapper.group_cache.consume(self._pending_key)     # the cache's use count follows the reference protocol
        return out


class AddSVDCorrection(nn.Module):
    """``inner(x) + alpha_svd * (x B_q^T) A_q^T`` (src/step3_eval_dataset.py:450-516), fused into one launch."""

    def __init__(self, inner: nn.Module, A_q: torch.Tensor, B_q: torch.Tensor, role: str, is_group: bool,
                 group_cache: Optional[MiniGroupCache], alpha_svd: float = 1.0):
        super().__init__()
        if not isinstance(inner, CudaW4A16Linear):
            raise TypeError("AddSVDCorrection wraps CudaW4A16Linear modules only (no Triton / dense backends here)")
        self.inner = inner
        self.register_buffer("A_q", A_q.to(torch.float16).contiguous(), persistent=False)
        self.register_buffer("B_q", B_q.to(torch.float16).contiguous(), persistent=False)
        self.role = role
        self.is_group = is_group
        self.group_cache = group_cache
        self.alpha_svd = alpha_svd
        self._own_r = K.RRows()
        self.group_launcher: Optional[GroupLauncher] = None     # installed by the patchers
        # The reference discovers a factor/linear shape mismatch as a RuntimeError inside forward and then
        # returns the uncorrected output (step3_eval_dataset.py:512-516); the same outcome, decided once, with a warning.
        self._mismatch = (A_q.dim() != 2 or B_q.dim() != 2 or A_q.size(0) != inner.out_features
                          or B_q.size(1) != inner.in_features or A_q.size(1) != B_q.size(0))
        if self._mismatch:
            warnings.warn(f"AddSVDCorrection: factor shapes A{tuple(A_q.shape)} B{tuple(B_q.shape)} do not fit "
                          f"linear {inner.in_features}->{inner.out_features}; correction disabled for this module")

    def _private_r(self, m: int, rank: int, device) -> torch.Tensor:
        if not isinstance(self._own_r, K.RRows):
            self._own_r = K.RRows()
        return self._own_r.rows(m, rank, device)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        gl = self.group_launcher
        if gl is not None and gl.usable and x.is_cuda:
            if gl._refs[0]() is self:
                members = [ref() for ref in gl._refs]
                if None not in members:      # (of a group of which only some are left, each launches for itself)
                    for w in members:
                        if w.alpha_svd != 0.0 and not w._mismatch:
                            return gl.run(x, members)
                gl.forget()      # nothing to correct in this group: outputs kept from an earlier call must not be served
            else:
                out = gl.take(self, x)
                if out is not None:
                    return out
        if self.alpha_svd == 0.0 or self._mismatch:
            return self.inner(x)
        inner = self.inner
        lead = x.shape[:-1]
        x2d = inner._flatten_input(x)
        m, rank, dev = x2d.size(0), self.A_q.size(1), x2d.device
        key = _x_key(x)
        cache = self.group_cache if self.is_group else None
        mode, r_buf = K.R_COMPUTE, None
        if cache is not None and self.role in ("k", "v", "up"):
            r_buf, hit = cache.consume(key)
            if hit and r_buf is not None and r_buf.size(0) == m and r_buf.device == dev:
                mode = K.R_LOAD
            else:
                r_buf = None
        if r_buf is None:
            if cache is not None and self.role in ("q", "gate"):
                r_buf = cache.buffer(m, rank, dev)
            else:
                r_buf = self._private_r(m, rank, dev)
        out = inner.launch(x2d, L=self.A_q, R=self.B_q, r_buf=r_buf, r_mode=mode, alpha=float(self.alpha_svd))
        if mode == K.R_COMPUTE and cache is not None and self.role in ("q", "gate"):
            cache.set(r_buf, 2 if self.role == "q" else 1, key)
        return out.reshape(*lead, inner.out_features)


def get_parent_module(model: nn.Module, name: str):
    parent = model
    *path, leaf = name.split(".")
    for part in path:
        parent = getattr(parent, part)
    return parent, leaf


def _role_from_suffix(sfx: str) -> str:
    for end, role in (("q_proj", "q"), ("k_proj", "k"), ("v_proj", "v"), ("gate_proj", "gate"), ("up_proj", "up")):
        if sfx.endswith(end):
            return role
    return "solo"


def _resolve(bkey: str, module_name: str):
    """(group key, A key, role, is_group) for one b_ref_map entry.  Grouped entries point at
    ``<gkey>.B_shared`` and take ``<gkey>.<module suffix>.A``; solo entries point at ``<module>.B`` and take
    ``<module>.A`` (key scheme written by src/step2_rsvd.py:487-522)."""
    if "B_shared" in bkey:
        gkey = bkey.replace(".B_shared", "")
        suffix = module_name.split(".")[-1]
        return gkey, f"{gkey}.{suffix}.A", _role_from_suffix(suffix), True
    gkey = bkey.rsplit(".", 1)[0] if bkey.endswith(".B") else bkey.replace(".B", "")
    return gkey, gkey + ".A", "solo", False


def _patch(model, shared, bmap, alpha_svd, groups_to_patch: Optional[Set[str]], verbose: bool):
    patched = skipped = 0
    wrapped = []
    caches: Dict[str, MiniGroupCache] = {}
    items = bmap.items()
    if verbose:
        items = _tqdm(items, desc="Patching SVD Correction")
    for weight_name, bkey in items:
        module_name = weight_name.replace(".weight", "")
        gkey, a_key, role, is_group = _resolve(bkey, module_name)
        if groups_to_patch is not None and gkey not in groups_to_patch:
            continue
        cache = caches.setdefault(gkey, MiniGroupCache()) if is_group else None
        A_q, B_q = shared.get(a_key), shared.get(bkey)
        if A_q is None or B_q is None:
            skipped += 1
            continue
        try:
            parent, leaf = get_parent_module(model, module_name)
            inner = getattr(parent, leaf)
        except (AttributeError, IndexError, KeyError) as exc:
            if verbose:
                print(f"AttributeError for {module_name}: {exc}")
            skipped += 1
            continue
        if not isinstance(inner, CudaW4A16Linear):
            skipped += 1
            continue
        dev = inner.qweight_i32.device
        wrapper = AddSVDCorrection(inner, A_q.to(dev), B_q.to(dev), role=role, is_group=is_group,
                                   group_cache=cache, alpha_svd=alpha_svd)
        setattr(parent, leaf, wrapper)
        wrapped.append((gkey, wrapper))
        patched += 1
    if verbose:
        print(f"SVD Correction Patching Summary: {patched} patched, {skipped} skipped")
    if _fuse_enabled():
        # launch order = module order of the model (q, k, v, o, gate, up, down within a layer), whatever the order of
        # the map's entries
        pos = {id(m): i for i, (_, m) in enumerate(model.named_modules())}
        wrapped.sort(key=lambda gw: pos.get(id(gw[1]), len(pos)))
        _install_launchers(wrapped)
    return model


def _install_launchers(wrapped) -> None:
    """``wrapped``: (group key, wrapper) in patch order = model order.  Members of a group share one launcher (the
    producer role first); every solo module gets its own; launchers are chained in model order."""
    order, by_key = [], {}
    for gkey, w in wrapped:
        key = gkey if w.is_group else (gkey, id(w))
        if key not in by_key:
            by_key[key] = []
            order.append(key)
        by_key[key].append(w)
    launchers = []
    for key in order:
        members = by_key[key]
        if members[0].is_group and members[0].role not in ("q", "gate"):
            continue                      # a group without its producer: the per-module protocol handles it
        gl = GroupLauncher(members)
        for w in members:
            w.group_launcher = gl
        launchers.append(gl)
    for a, b in zip(launchers, launchers[1:] + launchers[:1]):
        a.next_launcher = b


def patch_svd_correction_wrappers(model, shared, bmap, alpha_svd=1.0):
    """Wrap every module named in ``bmap`` whose factors exist (src/step3_eval_dataset.py:535-605)."""
    return _patch(model, shared, bmap, alpha_svd, None, True)


def patch_svd_correction_wrappers_cumulative(model, shared, bmap, groups_to_patch: set, alpha_svd=1.0):
    """GlowQ-S: wrap only modules whose group key (``layer{L}_qkv``, ``layer{L}_mlp`` or a solo module path) is in
    ``groups_to_patch``; every other module stays a bare CudaW4A16Linear
    (src/restoration/step4_evaluate_cumulative.py:99-154)."""
    return _patch(model, shared, bmap, alpha_svd, set(groups_to_patch), False)


__all__ = ["AddSVDCorrection", "MiniGroupCache", "GroupLauncher", "patch_svd_correction_wrappers",
           "patch_svd_correction_wrappers_cumulative", "clear_group_cache", "get_parent_module"]
