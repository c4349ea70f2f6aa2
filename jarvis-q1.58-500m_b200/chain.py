"""Whole layers in one ctypes call (jb200_forward_layers): the descriptor table of a list of blocks and its checks.

A forward is ~14 launches per layer.  Issued through ops.* each costs ~15 us of Python; here the loop over the layers
runs in C++ and Python pays for one call, a handful of allocations and the check that no parameter has changed.
"""
from __future__ import annotations

import ctypes as C
import math
import operator
import threading
import weakref
from typing import List, Optional

import torch

from . import _lib, ops

_data_ptr = torch.Tensor.data_ptr
_version = operator.attrgetter("_version")


# Methods of the stock classes that the native call stands for, by the part a module plays in a block: {name: function}, filled
# where the classes are.
_STOCK = {}


def stands_for(part, cls, *names):
    _STOCK[part] = {n: cls.__dict__[n] for n in names}


def _methods(block):
    """(module, name, stock function) of every method of the block's parts that the native call stands for."""
    at = block.attn
    parts = dict(block=block, attn=at, moe=block.moe, out_proj=getattr(at, "out_proj", None), rotary=getattr(at, "rotary", None))
    return [(m, n, fn) for part, m in parts.items() for n, fn in _STOCK[part].items()]


def _stock(block) -> bool:
    """Nothing of the block overrides what the native call stands for (a subclass that leaves those methods alone may)."""
    return all(getattr(type(m), n, None) is fn and n not in m.__dict__ for m, n, fn in _methods(block))


def supported(blocks) -> bool:
    """Blocks without overrides, of the shapes jb200_forward_layers takes: all parameters on one CUDA device and of the sizes the
    first block gives, since the native call knows nothing but their addresses."""
    if not all(map(_stock, blocks)):
        return False
    a = blocks[0].attn
    d_model = a.q_proj.weight.shape[1]
    hidden, E, dev = blocks[0].moe.w1[0].weight.shape[0], blocks[0].moe.num_experts, blocks[0].norm1.weight.device
    if d_model % 128 or d_model > 1024 or hidden % 128 or E not in (4, 8) or dev.type != "cuda":
        return False
    return all(_fits(b, a, d_model, hidden, E) and all(p.device == dev for p in b.parameters()) for b in blocks)


def _fits(b, a, d_model, hidden, E) -> bool:
    at, moe = b.attn, b.moe
    square, up, down = (d_model, d_model), (hidden, d_model), (d_model, hidden)
    return (at.n_heads == a.n_heads and at.head_dim == 64 and at.n_heads * 64 == d_model and at.rotary.base == a.rotary.base and
            at.gamma_raw.numel() == at.n_heads and moe.num_experts == E and moe.top_k == 2 and
            len(moe.w1) == len(moe.w2) == E and moe.router.weight.shape == (E, d_model) and
            b.norm1.weight.numel() == b.norm2.weight.numel() == d_model and b.liquid.var_scale.numel() == 1 and
            all(m.weight.shape == square for m in (at.q_proj, at.k_proj, at.v_proj, at.out_proj)) and
            all(m.weight.shape == up for m in moe.w1) and all(m.weight.shape == down for m in moe.w2))


_step_lock = threading.Lock()
_LAID_OUT = ("w_qkv", "a_qkv", "w_out", "a_out", "w1", "a1", "w2", "a2", "gamma")      # what a layer's second layout is made of


class LayerTable:
    """jb200_layer array of `blocks`, valid as long as every parameter it was built from is the same unmodified tensor in
    the same place (identity, storage and version are compared on every call: 16 tensors per layer, ~0.1 us each)."""

    def __init__(self, blocks, before: Optional["LayerTable"] = None):
        """before: the table that this one takes the place of; layers whose packed weights are still its keep their second layout."""
        from .modules import ReflectivePenalty, _f32
        blocks = list(blocks)
        # weak: a block may own its table, and a cycle would keep a dropped model's memory until the next collection
        self.blocks = [weakref.ref(b) for b in blocks]
        self.n = len(blocks)
        b0 = blocks[0]
        self.rotary = b0.attn.rotary
        self.C, self.H, self.E = b0.norm1.weight.numel(), b0.attn.n_heads, b0.moe.num_experts
        self.hidden = b0.moe.w1[0].weight.shape[0]
        self.device = b0.norm1.weight.device
        self.acc_bytes = _lib.load().jb200_accumulator_bytes(self.E)
        self.array = (_lib.Layer * self.n)()
        self._keep = []
        self._sizes = {}
        self._step = None
        self.has_reflect = all(type(b.reflect) is ReflectivePenalty for b in blocks)
        self._watch(blocks)
        for d, b in zip(self.array, blocks):
            at, moe, lq = b.attn, b.moe, b.liquid
            qkv, a_qkv = at.qkv_packed()
            out, a_out = at.out_proj.packed()
            (w1, a1), (w2, a2) = moe.packed()
            tensors = dict(w_norm1=_f32(b.norm1.weight), w_norm2=_f32(b.norm2.weight), w_router=_f32(moe.router.weight),
                           gamma=at.decays(), var_scale=_f32(lq.var_scale, scalar=True), w_qkv=qkv, a_qkv=a_qkv, w_out=out,
                           a_out=a_out, w1=w1, a1=a1, w2=w2, a2=a2)
            if self.has_reflect:
                tensors["mu"] = _f32(b.reflect.mu_t, scalar=True)
                d.reflect_lam, d.reflect_tau = b.reflect.lam, b.reflect.tau_max
            for name, t in tensors.items():
                setattr(d, name, t.data_ptr())
            self._keep.append(tensors)
            d.eps1, d.eps2, d.balance_alpha = b.norm1.eps, b.norm2.eps, moe.balance_alpha
            d.alpha_min, d.alpha_max = lq.alpha_min, lq.alpha_max
        self._laid = [None] * self.n
        if before is not None and before.device == self.device:
            same = [all(a[k] is b[k] for k in _LAID_OUT) for a, b in zip(self._keep, before._keep)]
            self._laid = [t if ok else None for t, ok in zip(before._laid, same)] + [None] * (self.n - len(same))

    def __reduce__(self):
        """Addresses mean nothing in a copy: a copied, saved or sent module makes its own table."""
        return type(None), ()

    def _watch(self, blocks):
        slots, mods, self._flags, self._consts = [], [], [], []
        for b in blocks:
            at, moe = b.attn, b.moe
            mods += [(b, "norm1"), (b, "norm2"), (b, "attn"), (b, "moe"), (b, "liquid"), (b, "reflect"), (moe, "router"),
                     (moe, "w1"), (moe, "w2")] + [(at, n) for n in ("q_proj", "k_proj", "v_proj", "out_proj", "rotary")]
            slots += [(m, "weight") for m in (b.norm1, b.norm2, moe.router, at.q_proj, at.k_proj, at.v_proj, at.out_proj)]
            slots += [(at, "gamma_raw"), (b.liquid, "var_scale")]
            for lst in (moe.w1, moe.w2):
                mods += [(lst, str(i)) for i in range(len(lst))]
                slots += [(m, "weight") for m in lst]
            self._flags.append((at.__dict__, moe.__dict__, b.reflect.__dict__))
            self._consts.append((b.norm1, b.norm2, moe, b.liquid, b.reflect))
        held = [h for b in blocks for h in _methods(b)]
        # instance overrides; not the blocks' own dictionaries, which may hold this table (`current` gets those to look at)
        own = set(map(id, blocks))
        self._dicts, self._names = zip(*((m.__dict__, n) for m, n, _ in held if id(m) not in own))
        self._block_names = [n for m, n, _ in held if m is blocks[0]]
        stock = {(type(m), n): fn for m, n, fn in held}                                           # and those of the classes
        self._types, self._methods = list(zip(*stock)), list(stock.values())
        slots = [(m._parameters, n) for m, n in slots]
        if self.has_reflect:
            slots += [(b.reflect._buffers, "mu_t") for b in blocks]
        self._slots, self._mods = list(zip(*slots)), list(zip(*((m._modules, n) for m, n in mods)))
        self._mod_objs = list(map(operator.getitem, *self._mods))
        self._params = list(map(operator.getitem, *self._slots))
        self._ptrs = list(map(_data_ptr, self._params))
        self._versions = list(map(_version, self._params))
        self._const_vals = self._read_consts()

    def _read_consts(self):
        return [(a.eps, b.eps, m.balance_alpha, q.alpha_min, q.alpha_max, getattr(r, "lam", None), getattr(r, "tau_max", None))
                for a, b, m, q, r in self._consts]

    def current(self, blocks) -> bool:
        try:
            now = list(map(operator.getitem, *self._slots))
            return (all(map(operator.is_, now, self._params)) and list(map(_data_ptr, now)) == self._ptrs and
                    list(map(_version, now)) == self._versions and
                    list(map(operator.getitem, *self._mods)) == self._mod_objs and      # modules compare by identity
                    not any(map(operator.contains, self._dicts, self._names)) and
                    not any(n in b.__dict__ for n in self._block_names for b in blocks) and
                    list(map(getattr, *self._types)) == self._methods and
                    self._read_consts() == self._const_vals)
        except (KeyError, AttributeError):
            return False

    def local(self) -> bool:
        """Nothing that needs the per-kernel path: statistics or experts shared with other GPUs, fused prologue, training, a
        penalty that has to be called (its running mean moves in training, hooks see its call)."""
        for at, moe, refl in self._flags:
            if moe["stats_group"] is not None or moe["_ep"] is not None or at["fuse_prologue"] or moe["training"]:
                return False
            if self.has_reflect and (refl["training"] or refl["_forward_hooks"] or refl["_forward_pre_hooks"] or "forward" in refl):
                return False
        return True

    def step_weights(self, B: int):
        """The layers' weights as the one-launch step of B sequences reads them (host array of device pointers), laid out when first
        wanted; None where there is no such step, or no memory for them when that was.  Not made inside a stream capture, which would
        only record the work."""
        lib = _lib.load()
        if B > lib.jb200_step_max_sequences():
            return None
        if self._step is None:
            nbytes = lib.jb200_step_weight_bytes(self.C, self.H, self.E, self.hidden)
            if not nbytes or torch.cuda.is_current_stream_capturing():
                return None
            with _step_lock:
                if self._step is None:
                    laid = list(self._laid)
                    new = [i for i, t in enumerate(laid) if t is None]
                    try:
                        buf = torch.empty((len(new), nbytes), dtype=torch.uint8, device=self.device)
                    except torch.OutOfMemoryError:       # the kernels need none; not tried again, a failing allocation is slow
                        self._step = (None,)
                        return None
                    for i, out in zip(new, buf):
                        _lib.check(lib.jb200_prepare_step_weights(C.byref(self.array[i]), self.C, self.H, self.E, self.hidden,
                                                                  out.data_ptr(), ops._stream()), "jb200_prepare_step_weights")
                        laid[i] = out
                    if new:
                        torch.cuda.current_stream(self.device).synchronize()      # any stream may be the next to read them
                    self._laid, self._step = laid, (_pointers(self.n, laid),)
        return self._step[0]

    def sizes(self, B: int, T: int):
        key = (B, T)
        got = self._sizes.get(key)
        if got is None:
            lib = _lib.load()
            off = (C.c_size_t * 7)()
            rb = lib.jb200_routing_layout(B * T, self.E, off)
            got = (lib.jb200_forward_workspace_bytes(B, T, self.C, self.H, self.E, self.hidden), rb, tuple(off))
            if len(self._sizes) >= 256:
                self._sizes.clear()
            self._sizes[key] = got
        return got


def table_of(owner, blocks) -> Optional[LayerTable]:
    """The (cached) table of `blocks`, kept on `owner`; None when they need the per-kernel path."""
    tab = owner.__dict__.get("_layer_table")
    if tab is None or tab.n != len(blocks) or any(r() is not b for r, b in zip(tab.blocks, blocks)) or not tab.current(blocks):
        if not supported(blocks):
            return None
        try:
            tab = LayerTable(blocks, tab)
        except KeyError:             # a weight that is no plain parameter (parametrised, pruned): read it anew on every call
            return None
        owner.__dict__["_layer_table"] = tab
    return tab if tab.local() else None


def _carried(ts, n: int, shape, dev, what: str, exact: bool = True, must_alias=None) -> List[Optional[torch.Tensor]]:
    """The carried states of n layers as contiguous f32 tensors (or None), checked: the native call reads and writes through
    their addresses.  exact: the shape itself and not just its number of elements.  must_alias(t): the caller's own tensor is
    to be updated, so one that would have to be converted is refused."""
    ts = list(ts)
    if len(ts) < n:
        raise RuntimeError(f"forward: {what} has {len(ts)} entries for {n} layers")
    out = []
    for t in ts[:n]:
        if t is not None:
            if t.device != dev:
                raise RuntimeError(f"forward: {what} on {t.device}, expected {dev} (this path has no CPU fallback)")
            if t.shape != shape and (exact or t.numel() != math.prod(shape)):
                raise RuntimeError(f"forward: {what} of shape {tuple(t.shape)}, expected {shape}")
            if t.dtype is not torch.float32 or not t.is_contiguous():
                if must_alias is not None and must_alias(t):
                    raise RuntimeError(f"forward: {what} updated in place must be contiguous f32, got {t.dtype} {tuple(t.stride())}")
                t = t.float().contiguous()
        out.append(t)
    return out


def _pointers(n, ts):
    return (C.c_void_p * n)(*[None if t is None else t.data_ptr() for t in ts])


def _results(n, given, inplace, shape, dev):
    """Where the states after the call go, one tensor per layer: the given ones (in place), new ones where there are none."""
    kept = given if inplace and given is not None else [None] * n
    missing = n if kept is not given else sum(t is None for t in kept)
    if not missing:
        return kept
    if n == 1:
        return [torch.empty(shape, dtype=torch.float32, device=dev)]
    new = iter(torch.empty((missing, *shape), dtype=torch.float32, device=dev).unbind(0))
    return [next(new) if t is None else t for t in kept]


class Result:
    """What a call leaves: h / S (lists, one tensor per layer; S None when not wanted), scalars f32 (n, 3), reflect f32 (n,)
    and hidden (normalised rows after the last layer, bf16).  scalars and reflect are views of aux (3 n, then n values), made when
    somebody looks: a view is a microsecond of a block's call."""
    __slots__ = ("h", "S", "aux", "has_reflect", "hidden")

    @property
    def scalars(self):
        return self.aux[:self.aux.numel() // 4 * 3].view(-1, 3)

    @property
    def reflect(self):
        return self.aux[self.aux.numel() // 4 * 3:] if self.has_reflect else None


def run(tab: LayerTable, x, B: int, T: int, *, ids=None, table=None, start_pos=0, max_position=None, h_in=None, s_in=None,
        want_state=False, inplace=False, final_norm=None) -> Result:
    """One jb200_forward_layers call on the current stream.  x: f32 (B*T, C), updated in place (written from `ids` and the
    embedding `table` when given).  h_in / s_in: lists with one tensor or None per layer, or None; inplace: layer by layer, the
    states that are given are updated."""
    n, dev = tab.n, tab.device
    if not (x.device == dev and x.dtype is torch.float32 and x.is_contiguous() and x.shape == (B * T, tab.C)):
        raise RuntimeError(f"forward: expected a contiguous f32 residual stream ({B * T}, {tab.C}) on {dev} (this path has no CPU fallback)")
    for t in (table, final_norm[0]) if final_norm is not None else (table,):
        if t is not None and (t.device != dev or t.shape[-1] != tab.C):
            raise RuntimeError(f"forward: embedding table or final norm ({t.device}, {tuple(t.shape)}): expected {tab.C} channels on {dev}")
    step = ids is not None and T == 1         # a model's single-token step
    if h_in is not None:
        # the tail of a single-token step leaves a new membrane where it cannot update the one it was given
        alias = (lambda t: t.dtype is torch.float32 or not step) if inplace else None
        h_in = _carried(h_in, n, (B, tab.C), dev, "the membrane", exact=step, must_alias=alias)
    if s_in is not None:
        s_in = _carried(s_in, n, (B, tab.H, 64, 64), dev, "the attention state")
    ws_bytes, routing_bytes, _ = tab.sizes(B, T)
    head = (n * tab.acc_bytes + 255) // 256 * 256
    work = torch.empty(head + ws_bytes, dtype=torch.uint8, device=dev)
    routing = torch.empty(n * routing_bytes, dtype=torch.uint8, device=dev)
    res = Result()
    aux = res.aux = torch.empty(4 * n, dtype=torch.float32, device=dev)
    res.has_reflect = tab.has_reflect
    f = _lib.Forward()
    f.B, f.T, f.C, f.H, f.E, f.hidden = B, T, tab.C, tab.H, tab.E, tab.hidden
    if ids is not None:
        f.ids, f.table, f.vocab = ids.data_ptr(), table.data_ptr(), table.shape[0]
    f.x = x.data_ptr()
    if torch.is_tensor(start_pos):
        if not (start_pos.device == dev and start_pos.dtype is torch.int32 and start_pos.is_contiguous() and start_pos.numel() >= B):
            raise RuntimeError(f"forward: per-sequence positions must be a contiguous int32 tensor on {dev} with one entry per sequence")
        # without the caller's bound the table is sized from the positions themselves (a host read)
        end = (max_position if max_position is not None else int(start_pos.max())) + T
        f.pos0 = start_pos.data_ptr()
    else:
        f.pos0_scalar = int(start_pos)
        end = f.pos0_scalar + T
    cos, sin = tab.rotary.half_tables(end, dev)
    f.cos_tab, f.sin_tab, f.n_pos = cos.data_ptr(), sin.data_ptr(), cos.shape[0]
    if h_in is not None:
        h_ptrs = _pointers(n, h_in)
        f.h_in = C.addressof(h_ptrs)
    if s_in is not None:
        s_ptrs = _pointers(n, s_in)
        f.s_in = C.addressof(s_ptrs)
    res.h = _results(n, h_in, inplace, (B, tab.C), dev)
    ho_ptrs = _pointers(n, res.h)
    f.h_out = C.addressof(ho_ptrs)
    res.S = None
    if want_state or (inplace and s_in is not None):
        res.S = _results(n, s_in, inplace, (B, tab.H, 64, 64), dev)
        so_ptrs = _pointers(n, res.S)
        f.s_out = C.addressof(so_ptrs)
    base = work.data_ptr()
    f.accumulators, f.workspace = base, base + head
    f.scalars, f.routing = aux.data_ptr(), routing.data_ptr()
    f.reflect = aux.data_ptr() + 12 * n if tab.has_reflect else None
    res.hidden = None
    if final_norm is not None:
        res.hidden = torch.empty((B * T, tab.C), dtype=torch.bfloat16, device=dev)
        f.w_final, f.eps_final, f.hidden_out = final_norm[0].data_ptr(), final_norm[1], res.hidden.data_ptr()
    # A lone token without any carried state is no decode loop: not worth a second layout of the weights.  From four sequences on the
    # one-launch step takes an attention state and leaves one.
    step = tab.step_weights(B) if T == 1 and (s_in is not None or (h_in is not None and B < 4)) else None
    _lib.check(_lib.load().jb200_forward_layers_prepared(tab.array, n, C.byref(f), step, ops._stream()), "jb200_forward_layers")
    for i, (_, moe, _) in enumerate(tab._flags):
        moe["_routing"] = RoutingSource((routing, i, B * T, tab.E))      # the views are built when somebody looks at them
    return res


class RoutingSource(tuple):
    """(routing buffer, layer, tokens, experts): where a layer's last routing is, for routing_views."""


def routing_views(src):
    """(topk_idx, gates, (counts, offsets, scatter, gather, gate_idx)) of one layer from its block of a call's routing buffer."""
    buf, layer, N, E = src
    off = (C.c_size_t * 7)()
    nbytes = _lib.load().jb200_routing_layout(N, E, off)

    def view(i, count, dtype, *shape):
        size = torch.empty((), dtype=dtype).element_size()
        at = layer * nbytes + off[i]
        return buf[at:at + count * size].view(dtype).view(*shape)
    i32 = torch.int32
    return (view(0, 2 * N, torch.int64, N, 2), view(1, 2 * N, torch.float32, N, 2),
            (view(2, E, i32, E), view(3, E + 1, i32, E + 1), view(4, 2 * N, i32, N, 2), view(5, 2 * N, i32, 2 * N),
             view(6, 2 * N, i32, 2 * N)))
