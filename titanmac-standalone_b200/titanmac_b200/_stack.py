"""The model as the flat table that the whole-model calls of libtmw take (``tmw_block`` / ``tmw_stack_desc``).

A step of a few rows is bound by its host work when every norm, product and attention call is issued from Python, so
``TitanMAC`` hands the library one table per call.  The table is built once and holds addresses and sizes only: before every
use everything that went into it is compared with the modules as they are, and it is rebuilt when a parameter has moved or
changed its layout, a module has been replaced or added, or an attribute has another value.  A model that the table cannot
describe - another type of module in a known place, hooks, a forward set on an instance, fp32, an active dropout - has no
table, and its modules are called one by one.
"""

from __future__ import annotations

import ctypes
import math
import operator
import weakref
from typing import List, Optional

import torch
import torch.nn as nn
from torch.nn.modules import module as _nn_module

from . import _native


_dtype_of, _nbytes_of = operator.attrgetter("dtype"), operator.attrgetter("nbytes")

def overrides(obj, base: type, *names: str) -> bool:
    """Whether the object, or the subclass of ``base`` that it is of, has methods of its own under these names."""
    cls, own = type(obj), obj.__dict__
    return any([n in own for n in names]) or (cls is not base and any([getattr(cls, n) is not getattr(base, n) for n in names]))


# What runs when a module is called beside its class's forward; the second pair only with a gradient to come.  (A forward set
# on the instance replaces the class's.)
_FORWARD_HOOKS = ("_forward_hooks", "_forward_pre_hooks")
_BACKWARD_HOOKS = ("_backward_hooks", "_backward_pre_hooks")


def _global_hooks(training: bool) -> bool:
    return bool(_nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks
                or (training and (_nn_module._global_backward_hooks or _nn_module._global_backward_pre_hooks)))


class ModelTable:
    """Addresses of a ``TitanMAC``'s parameters and how to tell that they still hold."""

    def __init__(self, model):
        self.ok = False
        # what holds() compares: (parameters of a module, name, address, strides, bytes, dtype), (children of a module, name,
        # child), (object, attribute, value), (parameters of a module, name, identity) where there should be none, and
        # (children of a ModuleList, how many); also what keeps the table from being built
        self._params: list = []
        self._children: list = []
        self._attributes: list = []
        self._absent: list = []
        self._lists: list = []
        self._module_dicts: list = []
        self._dropouts: list = []
        self._attentions: list = []
        self._places: list = []
        self.dtype = model.embed_tokens.weight.dtype
        self.device = model.embed_tokens.weight.device
        self.config = model.config
        self._build(model)
        columns = (lambda rows, n: tuple(list(col) for col in zip(*rows)) if rows else ([],) * n)  # noqa: E731
        self._params, self._children = columns(self._params, 6), columns(self._children, 3)
        self._attributes, self._absent = columns(self._attributes, 3), columns(self._absent, 3)

    def _build(self, model) -> None:
        from .attn.block_sparse_attention import BlockSparseAttention
        from .attn.windowed_attention import WindowedAttention
        from .blocks.titan_block import MLPBlock, RMSNorm, TitanBlock

        if self.dtype not in (torch.bfloat16, torch.float16) or self.device.type != "cuda":
            return
        c = model.config

        def take(parent: nn.Module, name: str, *types) -> Optional[nn.Module]:
            child = parent._modules.get(name)
            self._children.append((parent._modules, name, child))
            if type(child) not in types:
                return None
            if type(child) is nn.ModuleList:
                self._lists.append((child._modules, len(child)))
            if isinstance(child, nn.Dropout):
                self._dropouts.append(child)
            self._module_dicts.append(child.__dict__)
            return child

        def address(mod: nn.Module, name: str, shape) -> Optional[int]:
            d = mod._parameters
            prm = d.get(name)
            if prm is None:
                absent(mod, name)
                return None
            ptr, dtype = prm.data_ptr(), prm.dtype
            self._params.append((d, name, ptr, prm.stride(), prm.nbytes, dtype))
            ok = dtype is self.dtype and prm.shape == shape and prm.is_contiguous() and prm.device == self.device and ptr % 16 == 0
            return ptr if ok else None

        def absent(mod: nn.Module, name: str) -> bool:
            prm = mod._parameters.get(name)
            self._absent.append((mod._parameters, name, id(prm)))
            return prm is None

        def optional(mod: nn.Module, name: str, shape):
            if mod._parameters.get(name) is None:
                absent(mod, name)
                return 0
            return address(mod, name, shape)

        def attributes(obj, *names) -> tuple:
            values = tuple(getattr(obj, name) for name in names)
            self._attributes += zip((obj,) * len(names), names, values)
            return values

        D, V, d_head = c.d_model, c.vocab_size, c.d_head
        sizes = (c.n_heads, d_head, c.window_size, c.n_persistent)
        layers = take(model, "layers", nn.ModuleList)
        tops = (take(model, "embed_tokens", nn.Embedding), take(model, "embed_positions", nn.Embedding),
                take(model, "norm", RMSNorm), take(model, "lm_head", nn.Linear))
        if layers is None or len(layers) == 0 or any(t is None for t in tops) or not absent(tops[3], "bias"):
            return
        attributes(c, "d_model", "n_heads", "window_size", "n_persistent", "vocab_size", "max_seq_len", "norm_eps")
        F = layers[0].mlp.d_ff if type(layers[0]) is TitanBlock and type(layers[0].mlp) is MLPBlock else 0
        found: List[Optional[int]] = []
        self.blocks = (_native.Block * len(layers))()
        for i in range(len(layers)):
            block = take(layers, str(i), TitanBlock)
            if block is None:
                return
            attn, mlp = take(block, "attention", WindowedAttention, BlockSparseAttention), take(block, "mlp", MLPBlock)
            norms = (take(block, "norm_attn", RMSNorm), take(block, "norm_mlp", RMSNorm))
            if attn is None or mlp is None or None in norms or any(attributes(n, "eps") != (c.norm_eps,) for n in norms):
                return
            windowed = type(attn) is WindowedAttention
            if attributes(attn, "n_heads", "d_head", "window_size", "num_persistent" if windowed else "n_persistent") != sizes \
                    or mlp.d_ff != F:
                return
            kind = (0, 0)
            if not windowed:
                scale, block_size, use_conv = attributes(attn, "scale", "block_size", "use_conv")
                if scale != 1.0 / math.sqrt(d_head):
                    return
                kind = (block_size, attn.conv_q.kernel_size[0] if use_conv else 0)
            if i > 0 and kind != self.kind:
                return
            self.kind = kind
            self._attentions.append(attn)
            qkv, out = take(attn, "qkv_proj", nn.Linear), take(attn, "out_proj", nn.Linear)
            fc1, fc2 = take(mlp, "fc1", nn.Linear), take(mlp, "fc2", nn.Linear)
            if None in (qkv, out, fc1, fc2) or not absent(qkv, "bias") or not absent(out, "bias"):
                return
            if take(attn, "dropout", nn.Identity, nn.Dropout) is None or take(mlp, "dropout", nn.Identity, nn.Dropout) is None \
                    or take(mlp, "activation", nn.GELU) is None or attributes(mlp.activation, "approximate") != ("none",):
                return
            homes = [("norm_attn", norms[0], "scale", (D,)), ("norm_mlp", norms[1], "scale", (D,)), ("w_qkv", qkv, "weight", (3 * D, D)),
                     ("w_out", out, "weight", (D, D)), ("w_fc1", fc1, "weight", (F, D)), ("w_fc2", fc2, "weight", (D, F)),
                     ("b_fc1", fc1, "bias", (F,)), ("b_fc2", fc2, "bias", (D,))]
            for name in ("conv_q", "conv_k", "conv_v") if kind[1] else ():
                conv = take(attn, name, nn.Conv1d)
                if conv is None or not absent(conv, "bias"):
                    return
                homes.append((name, conv, "weight", (D, 1, kind[1])))
            b = self.blocks[i]
            for field, mod, key, shape in homes:
                value = (optional if key == "bias" else address)(mod, key, shape)
                found.append(value)
                setattr(b, field, value or None)
                self._places.append(((i, field), (mod._parameters, key)))
        d = self.desc = _native.StackDesc()
        top = (address(tops[0], "weight", (V, D)), address(tops[1], "weight", (c.max_seq_len, D)), address(tops[2], "scale", (D,)),
               address(tops[3], "weight", (V, D)))
        pers = 0
        if c.n_persistent > 0:
            pers = address(model, "persistent_tokens", (c.n_persistent, D))
        if None in found or None in top or pers is None or attributes(tops[2], "eps") != (c.norm_eps,) \
                or attributes(tops[0], "max_norm") != (None,) or attributes(tops[1], "max_norm") != (None,):
            return
        d.embed_tokens, d.embed_positions, d.norm, d.head = top
        tops_at = dict(embed_tokens=(tops[0], "weight"), embed_positions=(tops[1], "weight"), norm=(tops[2], "scale"),
                       head=(tops[3], "weight"))
        if pers:
            tops_at["persistent"] = (model, "persistent_tokens")
        self._places += [((-1, name), (m._parameters, key)) for name, (m, key) in tops_at.items()]
        d.persistent = pers or None
        d.block_size, d.conv_taps = self.kind
        d.dtype = _native._DTYPES[self.dtype]
        d.layers, d.d_model, d.heads, d.head_dim, d.d_ff = len(layers), D, c.n_heads, d_head, F
        d.window, d.n_persistent, d.vocab, d.max_positions, d.eps = c.window_size, c.n_persistent, V, c.max_seq_len, c.norm_eps
        # unique parameters as (dictionary, name), and each one's places in the structures: (layer or -1, field)
        self.slots, self.roles, at = [], [], {}
        for place, (d_, name) in self._places:
            prm = d_.get(name)
            if prm is not None:
                if id(prm) not in at:
                    at[id(prm)] = len(self.slots)
                    self.slots.append((d_, name))
                    self.roles.append([])
                self.roles[at[id(prm)]].append(place)
        self.geometry = sizes + (self.dtype,)
        self.decodes = d_head in (64, 128) and F % 32 == 0 and D <= 4096 and self.kind == (0, 0)
        self.forwards = V % 8 == 0 and F % 8 == 0 and D % 8 == 0 and d_head % 8 == 0 and self.kind[1] <= 8
        # the backward writes a gradient once per place; only for the table that is also the head it adds the places up
        # (and it knows nothing of an embedding table's options)
        options = [attributes(t, "padding_idx", "scale_grad_by_freq", "sparse") for t in tops[:2]]
        self.trains = self.forwards and D <= 2048 and options == [(None, False, False)] * 2 and all(
            len(places) == 1 or set(places) == {(-1, "embed_tokens"), (-1, "head")} for places in self.roles)
        self.workspace_bytes: dict = {}  # (batch, tokens) -> bytes; tokens = -1: a decode step
        self.ok = True

    def holds(self) -> bool:
        """Whether the modules, the attributes that went into the table and the parameters' places and layouts are still what
        it says.  Whole columns at a time: a model has some hundreds of each, and this is in front of every call."""
        get, tensor = dict.get, torch.Tensor
        dicts, names, children = self._children
        if not all(map(operator.is_, map(get, dicts, names), children)):
            return False
        for listed, n in self._lists:
            if len(listed) != n:
                return False
        objects, names, values = self._attributes
        if list(map(getattr, objects, names)) != values:
            return False
        dicts, names, ids = self._absent
        if list(map(id, map(get, dicts, names))) != ids:
            return False
        dicts, names, ptrs, strides, sizes, dtypes = self._params
        params = list(map(get, dicts, names))
        try:
            return (list(map(tensor.data_ptr, params)) == ptrs and list(map(tensor.stride, params)) == strides
                    and list(map(_nbytes_of, params)) == sizes and list(map(_dtype_of, params)) == dtypes)
        except TypeError:  # a parameter that is no more
            return False

    def plain_call(self, training: bool) -> bool:
        """Whether calling the modules would do nothing but compute: no hooks, no active dropout."""
        dicts = self._module_dicts
        for name in _FORWARD_HOOKS + _BACKWARD_HOOKS if training else _FORWARD_HOOKS:
            if any(map(operator.itemgetter(name), dicts)):
                return False
        if any(["forward" in d for d in dicts]):
            return False
        for m in self._dropouts:
            if m.training and m.p > 0:
                return False
        for m in self._attentions:
            if m.algo != _native.ALGO_AUTO or m.core_events is not None or not m.causal or (m.training and m.dropout_p > 0):
                return False
        return not _global_hooks(training)


# not an attribute of the model: copies and pickles of a model do not carry addresses
_tables: "weakref.WeakKeyDictionary[nn.Module, ModelTable]" = weakref.WeakKeyDictionary()


def table_of(model, training: bool = False) -> Optional[ModelTable]:
    """The model's table if it can be used right now (``training``: for a call with a gradient to come), else None."""
    table, weight = _tables.get(model), getattr(model.embed_tokens, "weight", None)
    if not isinstance(weight, torch.Tensor):  # another kind of embedding
        return None
    if table is None or weight.dtype is not table.dtype or weight.device != table.device or table.config is not model.config \
            or not table.holds():
        table = _tables[model] = ModelTable(model)
    return table if table.ok and table.plain_call(training) else None


def _attach(blocks, caches, geometry, device) -> bool:
    for b, c in zip(blocks, caches):
        if c.geometry != geometry or c.k_ring.device != device:
            return False
        b.k_ring, b.v_ring = c.k_ring.data_ptr(), c.v_ring.data_ptr()
        b.k_pers, b.v_pers = c.k_pers.data_ptr(), c.v_pers.data_ptr()
        b.cache_scale = c.scale
    return True


def forward(table: ModelTable, token_ids: torch.Tensor, caches=None) -> Optional[torch.Tensor]:
    """``tmw_stack_forward``: logits of every row (persistent rows first), or, with ``caches`` to fill, of the last one
    only; None where the arguments are not what that call takes."""
    device = table.device
    if not table.forwards or token_ids.dtype != torch.int64 or token_ids.dim() != 2 or token_ids.device != device:
        return None
    B, T = token_ids.shape
    d = _native.StackDesc.from_buffer_copy(table.desc)
    if B == 0 or T == 0 or T > d.max_positions or B * (T + d.n_persistent) >= 1 << 31:
        return None
    token_ids = token_ids.contiguous()
    blocks = type(table.blocks).from_buffer_copy(table.blocks)
    if caches is not None and (len(caches) != len(blocks) or not _attach(blocks, caches, (B,) + table.geometry, device)):
        return None
    d.batch = B
    lib = _native.lib()
    nbytes = table.workspace_bytes.get((B, T))
    if nbytes is None:
        if len(table.workspace_bytes) > 256:
            table.workspace_bytes.clear()
        nbytes = table.workspace_bytes[B, T] = lib.tmw_stack_workspace(ctypes.byref(d), T)
    workspace = torch.empty(nbytes, dtype=torch.uint8, device=device)
    shape = (B, d.vocab) if caches is not None else (B, T + d.n_persistent, d.vocab)
    logits = torch.empty(shape, dtype=table.dtype, device=device)
    with _native._on(device):
        _native.check(lib.tmw_stack_forward(ctypes.byref(d), blocks, token_ids.data_ptr(), T, int(caches is not None),
                                            logits.data_ptr(), workspace.data_ptr(), nbytes, _native._stream_ptr(device)))
    return logits


def _step_arguments(table: ModelTable, batch: int, caches):
    """``(StackDesc, blocks with the caches, workspace)`` of a decode step, or None where the table or the caches are not what
    the step takes."""
    device = table.device
    if not table.decodes or not 0 < batch <= 65535 or len(caches) != len(table.blocks):
        return None
    blocks = type(table.blocks).from_buffer_copy(table.blocks)  # (the table is shared by all threads)
    if not _attach(blocks, caches, (batch,) + table.geometry, device):
        return None
    d = _native.StackDesc.from_buffer_copy(table.desc)
    d.batch = batch
    nbytes = table.workspace_bytes.get((batch, -1))
    if nbytes is None:
        with _native._on(device):  # (what it takes depends on the device's SMs)
            nbytes = table.workspace_bytes[batch, -1] = _native.lib().tmw_decode_step_workspace(ctypes.byref(d))
    return d, blocks, torch.empty(nbytes, dtype=torch.uint8, device=device)


def decode_step(table: ModelTable, token_ids: torch.Tensor, pos: torch.Tensor, caches) -> Optional[torch.Tensor]:
    """``tmw_decode_step``; None where the arguments are not what that call takes."""
    B = token_ids.shape[0]
    device = table.device
    if (token_ids.dtype != torch.int64 or pos.dtype != torch.int32 or token_ids.dim() != 1 or pos.shape != (B,)
            or token_ids.device != device or pos.device != device):
        return None
    arguments = _step_arguments(table, B, caches)
    if arguments is None:
        return None
    d, blocks, workspace = arguments
    token_ids, pos = token_ids.contiguous(), pos.contiguous()
    logits = torch.empty((B, d.vocab), dtype=table.dtype, device=device)
    with _native._on(device):
        _native.check(_native.lib().tmw_decode_step(ctypes.byref(d), blocks, token_ids.data_ptr(), pos.data_ptr(), logits.data_ptr(),
                                                    workspace.data_ptr(), workspace.numel(), _native._stream_ptr(device)))
    return logits


def generate(table: ModelTable, input_ids: torch.Tensor, logits: torch.Tensor, caches, new_tokens: int) -> Optional[torch.Tensor]:
    """The prompt and its greedy continuation (``tmw_generate``) from the logits of its last token; None where the arguments
    are not what that call takes."""
    B, T = input_ids.shape
    device = table.device
    if input_ids.dtype != torch.int64 or input_ids.device != device or new_tokens < 0 or not logits.is_contiguous() \
            or logits.dtype != table.dtype:
        return None
    arguments = _step_arguments(table, B, caches)
    if arguments is None:
        return None
    d, blocks, workspace = arguments
    out = torch.empty((B, T + new_tokens), dtype=torch.int64, device=device)
    out[:, :T] = input_ids
    token = torch.empty(B, dtype=torch.int64, device=device)
    pos = torch.full((B,), T, dtype=torch.int32, device=device)
    with _native._on(device):
        _native.check(_native.lib().tmw_generate(ctypes.byref(d), blocks, logits.data_ptr(), new_tokens, token.data_ptr(),
                                                 pos.data_ptr(), out.data_ptr() + 8 * T, T + new_tokens, workspace.data_ptr(),
                                                 workspace.numel(), _native._stream_ptr(device)))
    return out


def _plain_weight(mod: nn.Module, kind, like: torch.Tensor, shape, training: bool) -> Optional[torch.Tensor]:
    """The weight of a submodule that is nothing but a ``kind`` without bias and hooks, contiguous, of that shape, and of
    ``like``'s dtype and device."""
    d = mod.__dict__
    if type(mod) is not kind or d["_forward_hooks"] or d["_forward_pre_hooks"] or "forward" in d \
            or (training and (d["_backward_hooks"] or d["_backward_pre_hooks"])):
        return None
    p = d["_parameters"]
    w = p.get("weight")  # (a tensor that is no parameter stands elsewhere)
    return w if w is not None and p.get("bias") is None and "bias" in p and w.dtype is like.dtype and w.shape == shape \
        and w.is_contiguous() and w.device == like.device else None


def attention_plan(attn: nn.Module, x: torch.Tensor, n_persistent: int, block_size: int, scale: float, training: bool = False):
    """``(AttentionDesc, w_qkv, w_out, convolution weights)`` if the module's forward on ``x`` is nothing but what the library
    computes in one call, else None.  The library takes every extent from the descriptor, so an input or a weight of another
    shape goes to the modules, which raise or, where they can, compute it."""
    dtype = x.dtype
    if (dtype is not torch.bfloat16 and dtype is not torch.float16) or attn.algo or attn.core_events is not None \
            or not x.is_contiguous():
        return None
    B, L, D = x.shape
    if D != attn.n_heads * attn.d_head or B * L == 0 or attn.d_head % 8 or _global_hooks(training):
        return None
    mods = attn._modules
    w_qkv = _plain_weight(mods["qkv_proj"], nn.Linear, x, (3 * D, D), training)
    w_out = _plain_weight(mods["out_proj"], nn.Linear, x, (D, D), training)
    if w_qkv is None or w_out is None:
        return None
    conv, taps = (), 0
    if block_size and attn.use_conv:
        taps = mods["conv_q"].weight.shape[-1]
        conv = tuple(_plain_weight(mods[n], nn.Conv1d, x, (D, 1, taps), training) for n in ("conv_q", "conv_k", "conv_v"))
        if not 1 <= taps <= 8 or any(w is None for w in conv):
            return None
    if (x.data_ptr() | w_qkv.data_ptr() | w_out.data_ptr()) % 16:
        return None
    return _native.AttentionDesc(_native._DTYPES[dtype], B, L, attn.n_heads, attn.d_head, attn.window_size, n_persistent, block_size,
                                 taps, scale), w_qkv, w_out, conv


def attention_forward(attn: nn.Module, x: torch.Tensor, n_persistent: int, block_size: int, scale: float) -> Optional[torch.Tensor]:
    """An attention module's forward as one ``tmw_attention_forward``; None where that call does not apply."""
    plan = attention_plan(attn, x, n_persistent, block_size, scale)
    if plan is None:
        return None
    d, w_qkv, w_out, conv = plan
    lib = _native.lib()
    ref = ctypes.byref(d)
    device = x.device
    nbytes = lib.tmw_attention_workspace(ref)
    y = torch.empty(x.shape, dtype=x.dtype, device=device)
    workspace = torch.empty(nbytes, dtype=torch.uint8, device=device)
    conv_ptrs = tuple(w.data_ptr() for w in conv) if conv else (None, None, None)
    with _native._on(device):
        _native.check(lib.tmw_attention_forward(ref, x.data_ptr(), w_qkv.data_ptr(), *conv_ptrs, w_out.data_ptr(), y.data_ptr(),
                                                workspace.data_ptr(), nbytes, _native._stream_ptr(device)))
    return y
