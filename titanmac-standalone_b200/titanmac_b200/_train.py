"""Training steps in 16-bit types as single autograd nodes over the whole-model and whole-module calls of libtmw.

``TitanMAC`` and the attention modules use them when every part is what the library computes (see ``_stack.ModelTable``);
anything else - fp32, frozen parameters, hooks, autocast - keeps the graph of the modules themselves.
"""

from __future__ import annotations

import ctypes
from typing import Optional

import torch
from torch.autograd.function import once_differentiable

from . import _native, _stack


def _autocast() -> bool:
    return torch.is_autocast_enabled("cuda")


def _aligned(grad: torch.Tensor) -> torch.Tensor:
    """The gradient contiguous and at an address the kernels take (autograd may hand over any part of a larger one)."""
    grad = grad.contiguous()
    return grad.clone() if grad.data_ptr() % 16 else grad


class _Rows:
    """The logits of all rows ``[B, Np + T, V]``, persistent rows first, and their gradient, around the sequence rows ``[B, T, V]``
    that the caller sees and the loss depends on.  Where the gradient of the sequence rows is the one that the loss's backward
    has just written inside a gradient of all rows, that one is taken as it is."""

    __slots__ = ("rows", "d_rows")

    def __init__(self, rows: Optional[torch.Tensor] = None):
        self.rows, self.d_rows = rows, None

    def gradient(self, d_logits: torch.Tensor, n_persistent: int) -> torch.Tensor:
        """Of all rows, contiguous; the persistent ones' is zero."""
        if n_persistent == 0:
            return d_logits
        d_rows, self.d_rows = self.d_rows, None  # (held until here: no other tensor can have its address)
        if d_rows is not None:
            own = d_rows[:, n_persistent:]
            if d_logits.data_ptr() == own.data_ptr() and d_logits.stride() == own.stride() and d_logits.shape == own.shape:
                return d_rows
        B, T, V = d_logits.shape
        d_rows = d_logits.new_empty((B, n_persistent + T, V))
        d_rows[:, :n_persistent] = 0
        d_rows[:, n_persistent:] = d_logits
        return d_rows


class _StackTrain(torch.autograd.Function):
    """``ids [B, T]`` → logits of the sequence rows ``[B, T, V]``; ``held`` gets those of all rows."""

    @staticmethod
    def forward(ctx, table, held: _Rows, ids: torch.Tensor, *params: torch.Tensor) -> torch.Tensor:
        d = _native.StackDesc.from_buffer_copy(table.desc)
        B, T = ids.shape
        d.batch = B
        lib, ref, device = _native.lib(), ctypes.byref(d), ids.device
        nbytes = lib.tmw_stack_train_saved(ref, T)
        saved = torch.empty(nbytes, dtype=torch.uint8, device=device)
        logits = torch.empty((B, T + d.n_persistent, d.vocab), dtype=table.dtype, device=device)
        with _native._on(device):
            _native.check(lib.tmw_stack_train_forward(ref, table.blocks, ids.data_ptr(), T, logits.data_ptr(), saved.data_ptr(),
                                                      nbytes, _native._stream_ptr(device)))
        ctx.desc, ctx.roles, ctx.held = d, table.roles, held
        ctx.save_for_backward(ids, saved, *params)
        held.rows = logits
        return logits[:, d.n_persistent:].detach() if d.n_persistent else logits  # (not a view to autograd: it may be changed)

    @staticmethod
    @once_differentiable
    def backward(ctx, d_logits: torch.Tensor):
        ids, saved, *params = ctx.saved_tensors
        d = _native.StackDesc.from_buffer_copy(ctx.desc)
        d_logits = _aligned(ctx.held.gradient(d_logits, d.n_persistent))
        # the parameters' addresses as they are now, and their gradients'
        blocks, block_grads = (_native.Block * d.layers)(), (_native.BlockGrads * d.layers)()
        grads, out = _native.StackGrads(), []
        for prm, roles in zip(params, ctx.roles):
            grad = torch.empty_like(prm, memory_format=torch.contiguous_format)
            out.append(grad)
            p, g = prm.data_ptr(), grad.data_ptr()
            for layer, name in roles:
                if layer < 0:
                    setattr(d, name, p)
                    setattr(grads, name, g)
                else:
                    setattr(blocks[layer], name, p)
                    setattr(block_grads[layer], name, g)
        lib, ref, device, T = _native.lib(), ctypes.byref(d), ids.device, ids.shape[1]
        nbytes = lib.tmw_stack_train_scratch(ref, T)
        scratch = torch.empty(nbytes, dtype=torch.uint8, device=device)
        with _native._on(device):
            _native.check(lib.tmw_stack_train_backward(ref, blocks, ctypes.byref(grads), block_grads, ids.data_ptr(), T,
                                                       d_logits.data_ptr(), saved.data_ptr(), scratch.data_ptr(), nbytes,
                                                       _native._stream_ptr(device)))
        return (None, None, None, *out)


def stack_forward(model, input_ids: torch.Tensor):
    """``(logits of the sequence rows with a gradient to every parameter, _Rows around them)``, or None where that takes the
    modules themselves."""
    table = _stack.table_of(model, training=True)
    # (tokens that repeat are added up with atomics: not in a fixed order, as the library's embedding backward does)
    if table is None or not table.trains or _autocast() or torch.are_deterministic_algorithms_enabled() \
            or input_ids.dtype != torch.int64 or input_ids.dim() != 2 or input_ids.device != table.device:
        return None
    B, T = input_ids.shape
    if B == 0 or T == 0 or T > table.desc.max_positions or B * (T + table.desc.n_persistent) >= (1 << 31) // 8:
        return None
    params = [d[name] for d, name in table.slots]
    if not all(p.requires_grad for p in params):
        return None
    held = _Rows()
    return _StackTrain.apply(table, held, input_ids.contiguous(), *params), held


class _SequenceRows(torch.autograd.Function):
    """The sequence rows of ``rows [B, Np + T, V]``, which the modules have made; a slice of them would cost a pass over the
    gradient of all rows on the way back."""

    @staticmethod
    def forward(ctx, rows: torch.Tensor, n_persistent: int, held: _Rows) -> torch.Tensor:
        ctx.n_persistent, ctx.held = n_persistent, held
        return rows[:, n_persistent:].detach()

    @staticmethod
    @once_differentiable
    def backward(ctx, d_logits: torch.Tensor):
        return ctx.held.gradient(d_logits, ctx.n_persistent), None, None


class _ShiftedCrossEntropy(torch.autograd.Function):
    """Mean cross-entropy of ``rows [B, Np + T, V]``, row ``Np + t`` against ``labels[:, t + 1]`` (-100: not counted).  The
    gradient goes to ``logits``, the sequence rows; ``held`` keeps it as part of a gradient of all rows."""

    @staticmethod
    def forward(ctx, logits: torch.Tensor, rows: torch.Tensor, labels: torch.Tensor, n_persistent: int, held: _Rows) -> torch.Tensor:
        B, L, V = rows.shape
        loss = torch.empty((), dtype=rows.dtype, device=rows.device)
        stats = torch.empty(4 + 2 * B * L, dtype=torch.float32, device=rows.device)
        with _native._on(rows.device):
            _native.check(_native.lib().tmw_cross_entropy(_native._DTYPES[rows.dtype], B, L - n_persistent, n_persistent, V,
                                                          rows.data_ptr(), labels.data_ptr(), loss.data_ptr(), stats.data_ptr(),
                                                          None, None, _native._stream_ptr(rows.device)))
        ctx.save_for_backward(rows, labels, stats)
        ctx.n_persistent, ctx.held = n_persistent, held
        return loss

    @staticmethod
    @once_differentiable
    def backward(ctx, grad: torch.Tensor):
        rows, labels, stats = ctx.saved_tensors
        B, L, V = rows.shape
        n = ctx.n_persistent
        d_rows = torch.empty_like(rows)
        grad = grad.contiguous()
        with _native._on(rows.device):
            _native.check(_native.lib().tmw_cross_entropy(_native._DTYPES[rows.dtype], B, L - n, n, V, rows.data_ptr(),
                                                          labels.data_ptr(), None, stats.data_ptr(), grad.data_ptr(),
                                                          d_rows.data_ptr(), _native._stream_ptr(rows.device)))
        if n == 0:
            return d_rows, None, None, None, None
        ctx.held.d_rows = d_rows
        return d_rows[:, n:], None, None, None, None


def shifted_cross_entropy(rows: torch.Tensor, labels: torch.Tensor, n_persistent: int, logits: Optional[torch.Tensor] = None,
                          held: Optional[_Rows] = None):
    """``(logits, loss)`` of ``rows``, every row's logits, persistent rows first: the sequence rows and their mean shifted
    cross-entropy, which depends on them (``logits`` and ``held``: from ``stack_forward``, else they are made here).  None
    where the library's kernel does not apply."""
    B, L, V = rows.shape
    if (rows.dtype not in (torch.bfloat16, torch.float16) or not rows.is_cuda or not rows.is_contiguous() or V % 8
            or rows.data_ptr() % 16 or labels.dtype != torch.int64 or labels.shape != (B, L - n_persistent)
            or labels.device != rows.device or B == 0 or L == n_persistent or _autocast()):
        return None
    if held is None:
        held = _Rows()
        if n_persistent == 0:
            logits = rows
        elif rows.requires_grad and torch.is_grad_enabled():
            logits = _SequenceRows.apply(rows, n_persistent, held)
        else:
            logits = rows[:, n_persistent:]
        rows = rows.detach()
    return logits, _ShiftedCrossEntropy.apply(logits, rows, labels.contiguous(), n_persistent, held)


class _AttentionTrain(torch.autograd.Function):
    """An attention module's forward and backward: ``x [B, L, D]``, its projections and (block-sparse) convolutions."""

    @staticmethod
    def forward(ctx, desc, x: torch.Tensor, w_qkv: torch.Tensor, w_out: torch.Tensor, *conv: torch.Tensor) -> torch.Tensor:
        lib, ref, device = _native.lib(), ctypes.byref(desc), x.device
        nbytes = lib.tmw_attention_train_saved(ref)
        saved = torch.empty(nbytes, dtype=torch.uint8, device=device)
        y = torch.empty_like(x)
        with _native._on(device):
            _native.check(lib.tmw_attention_train_forward(ref, x.data_ptr(), w_qkv.data_ptr(), *_conv_ptrs(conv), w_out.data_ptr(),
                                                          y.data_ptr(), saved.data_ptr(), nbytes, _native._stream_ptr(device)))
        ctx.desc = desc
        ctx.save_for_backward(x, saved, w_qkv, w_out, *conv)
        return y

    @staticmethod
    @once_differentiable
    def backward(ctx, dy: torch.Tensor):
        x, saved, w_qkv, w_out, *conv = ctx.saved_tensors
        dy = _aligned(dy)
        lib, ref, device = _native.lib(), ctypes.byref(ctx.desc), x.device
        nbytes = lib.tmw_attention_train_scratch(ref)
        scratch = torch.empty(nbytes, dtype=torch.uint8, device=device)
        need = ctx.needs_input_grad
        dx = torch.empty_like(x) if need[1] else None
        out = [torch.empty_like(w) if n else None for w, n in zip((w_qkv, w_out, *conv), need[2:])]
        grads = _native.BlockGrads()
        for name, g in zip(("w_qkv", "w_out", "conv_q", "conv_k", "conv_v"), out):
            if g is not None:  # (the library leaves out what is not wanted)
                setattr(grads, name, g.data_ptr())
        with _native._on(device):
            _native.check(lib.tmw_attention_train_backward(ref, x.data_ptr(), w_qkv.data_ptr(), *_conv_ptrs(conv), w_out.data_ptr(),
                                                           dy.data_ptr(), saved.data_ptr(), dx.data_ptr() if need[1] else None,
                                                           ctypes.byref(grads), scratch.data_ptr(), nbytes,
                                                           _native._stream_ptr(device)))
        return (None, dx, *out)


def _conv_ptrs(conv):
    return tuple(w.data_ptr() for w in conv) if conv else (None, None, None)


def attention_forward(attn, x: torch.Tensor, n_persistent: int, block_size: int, scale: float) -> Optional[torch.Tensor]:
    """The module's forward as one autograd node, or None where that takes its parts."""
    if _autocast():
        return None
    x = x.contiguous()
    plan = _stack.attention_plan(attn, x, n_persistent, block_size, scale, training=True)
    if plan is None:
        return None
    desc, w_qkv, w_out, conv = plan
    return _AttentionTrain.apply(desc, x, w_qkv, w_out, *conv)
