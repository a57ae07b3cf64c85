"""Packed variable-length sequences and grouped value heads on top of the primitive.

The reference lists both as not yet part of its specialisation (README.md:128-130, 297-299 of
the reference); callers that batch ragged sequences need them next to the operator:

``chunk_gdn2_varlen``    several sequences packed along the time axis of ``[1, total, H, 128]``
                         tensors, delimited by ``cu_seqlens`` (``[N + 1]`` cumulative lengths, as
                         in flash-attention style APIs), each with its own initial / final state
                         (``[N, H, 128, 128]``).  Every sequence is an independent recurrence; the
                         kernels of all of them are launched together (csrc/packed.cu), each
                         sequence on the kernels its length calls for.  One
                         ``autograd.Function`` spans the whole call, and backward writes every
                         sequence's gradients straight into the packed gradient tensors.
``expand_grouped_heads`` key-shaped tensors given for fewer heads than the value-shaped ones
                         (every group of value heads shares one q / k / g / beta head) expanded
                         to the value heads; gradients of the shared heads are summed by autograd.

A batch goes to the library in groups of consecutive sequences: at most 256 of them (their table
travels in the kernels' parameters) and no more than the scratch budget of ``chunk_kernels`` holds.
"""

from __future__ import annotations

import ctypes
import math
from dataclasses import dataclass

import torch

from . import _lib, _validate, chunk_kernels
from .ops import _prologue_flags
from .prologue import gate_prologue

_DIM = 128


def _bounds(cu_seqlens, total: int) -> tuple[int, ...]:
    if isinstance(cu_seqlens, torch.Tensor):
        if cu_seqlens.ndim != 1 or cu_seqlens.dtype not in (torch.int32, torch.int64):
            raise TypeError("cu_seqlens must be a rank-1 int32 or int64 tensor")
        values = [int(x) for x in cu_seqlens.tolist()]
    else:
        values = [int(x) for x in cu_seqlens]
    if len(values) < 2 or values[0] != 0 or values[-1] != total:
        raise ValueError("cu_seqlens must start at 0 and end at the packed length of the tensors")
    if any(b < a for a, b in zip(values, values[1:])):
        raise ValueError("cu_seqlens must be non-decreasing")
    return tuple(values)


_MAX_SEQUENCES = 256


@dataclass(frozen=True)
class _Group:
    """Consecutive sequences ``first .. last - 1`` handed to the library in one call."""

    first: int
    last: int
    bounds: ctypes.Array   # int64[last - first + 1], rows of the packed tensors
    chunks: int
    chunk_slots: int
    span_slots: int


def _plan_groups(bounds: tuple[int, ...], heads: int, training: bool) -> list[_Group]:
    per_unit = chunk_kernels.scratch_bytes(1, 64, 1, False)
    if training:
        per_unit = chunk_kernels.scratch_bytes(1, 64, 1, True) + 2 * 65536
    most = max(1, chunk_kernels.SCRATCH_BUDGET_BYTES // (per_unit * heads))
    groups, first, chunks = [], 0, 0
    for i in range(len(bounds) - 1):
        own = chunk_kernels.supported_tokens(bounds[i + 1] - bounds[i]) // 64
        if i > first and (i - first == _MAX_SEQUENCES or chunks + own > most):
            groups.append((first, i))
            first, chunks = i, 0
        chunks += own
    groups.append((first, len(bounds) - 1))
    out, sizes = [], [ctypes.c_int64() for _ in range(3)]
    for lo, hi in groups:
        part = (ctypes.c_int64 * (hi - lo + 1))(*bounds[lo:hi + 1])
        status = _lib.lib().gdn2_packed_sizes(part, hi - lo, bounds[-1], heads, *(ctypes.byref(x) for x in sizes))
        if status != 0:
            raise RuntimeError(f"gdn2_packed_sizes failed with status {status}")
        out.append(_Group(lo, hi, part, *(x.value for x in sizes)))
    return out


def _states(slots: int, heads: int, device):
    if not slots:
        return None
    return torch.empty((slots, heads, _DIM, _DIM), device=device, dtype=torch.float32)


def _bytes(size: int, device):
    return torch.empty(size, device=device, dtype=torch.uint8)


def _short_kernels(bounds, prologue: int) -> int:
    """Forward launches for the sequences shorter than a chunk: up to 9 tokens (raw inputs: 8) go token by token."""

    lengths, steps = [b - a for a, b in zip(bounds, bounds[1:])], 8 if prologue else 9
    return any(steps < n < 64 for n in lengths) + any(n <= steps for n in lengths)


def _packed_forward(seq, state, bounds, scale: float, training: bool, prologue: int = 0):
    """Forward over every packed sequence; returns output, final states and what backward needs: the
    groups and, for each, ``(workspace, chunk checkpoints, span checkpoints)``."""

    q = seq[0]
    n_seq, total, heads, device = len(bounds) - 1, q.shape[1], q.shape[2], q.device
    output = torch.empty_like(seq[2])
    final_state = torch.empty((n_seq, heads, _DIM, _DIM), device=device, dtype=torch.float32)
    if total == 0:
        final_state.zero_() if state is None else final_state.copy_(state)
        return output, final_state, [], []
    saved, groups = [], _plan_groups(bounds, heads, training)
    scale = _validate.float32_scale(scale)
    for group in groups:
        tokens = 64 * group.chunks
        workspace = scratch = chunk_states = span_states = None
        if tokens:
            size = chunk_kernels.workspace_bytes(1, tokens, heads, training)
            scratch_size = 0 if training else chunk_kernels.scratch_bytes(1, tokens, heads, False)
            slots = group.chunk_slots if training else 0
            chunk_kernels.check_memory(size + scratch_size + slots * heads * _DIM * _DIM * 4, device, "packed forward")
            workspace = _bytes(size, device)
            scratch = None if training else _bytes(scratch_size, device)
        if training:
            chunk_states = _states(group.chunk_slots, heads, device)
            span_states = _states(group.span_slots, heads, device)
        part = slice(group.first, group.last)
        _lib.call("gdn2_packed_forward", device, *(x.data_ptr() for x in seq),
                  None if state is None else state[part].data_ptr(), output.data_ptr(), final_state[part].data_ptr(),
                  _lib.ptr(chunk_states), _lib.ptr(span_states), _lib.ptr(workspace), _lib.ptr(scratch), group.bounds,
                  group.last - group.first, total, heads, int(training), _lib.dtype_code(q.dtype),
                  _lib.dtype_code(seq[3].dtype), scale, prologue, _lib.stream_ptr(device),
                  kernels=2 * (group.chunks > 0) + _short_kernels(group.bounds, prologue))
        saved.append((workspace, chunk_states, span_states))
    return output, final_state, groups, saved


class _ChunkGDN2Varlen(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, g, beta, w, initial_state, bounds, scale: float):
        seq = tuple(_validate.detached(x) for x in (q, k, v, g, beta, w))
        output, final_state, ctx.groups, saved = _packed_forward(seq, _validate.detached(initial_state), bounds, scale,
                                                                 True)
        ctx.present = [tuple(x is not None for x in item) for item in saved]
        ctx.save_for_backward(q, k, v, g, beta, w, *(x for item in saved for x in item if x is not None))
        ctx.set_materialize_grads(False)
        ctx.n_seq, ctx.scale = len(bounds) - 1, scale
        ctx.has_initial_state = initial_state is not None
        return output, final_state

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, d_output, d_final_state):
        q, k, v, g, beta, w, *rest = ctx.saved_tensors
        seq = tuple(_validate.detached(x) for x in (q, k, v, g, beta, w))
        total, heads, device = q.shape[1], q.shape[2], q.device
        d_output = torch.zeros_like(v) if d_output is None else _dense(d_output)
        d_final_state = None if d_final_state is None else _dense(d_final_state)
        grads = tuple(torch.empty_like(x) for x in seq)
        d_state = torch.empty((ctx.n_seq, heads, _DIM, _DIM), device=device, dtype=torch.float32)
        if total == 0:
            d_state.zero_() if d_final_state is None else d_state.copy_(d_final_state)
        scale, rest = _validate.float32_scale(ctx.scale), iter(rest)
        for group, present in zip(ctx.groups, ctx.present):
            workspace, chunk_states, span_states = (next(rest) if there else None for there in present)
            scratch = d_chunk_states = None
            if group.chunks:
                size = chunk_kernels.scratch_bytes(1, 64 * group.chunks, heads, True)
                chunk_kernels.check_memory(size + chunk_states.numel() * 4, device, "packed backward")
                scratch = _bytes(size, device)
                d_chunk_states = torch.empty_like(chunk_states)
            d_span_states = None if span_states is None else torch.empty_like(span_states)
            part = slice(group.first, group.last)
            _lib.call("gdn2_packed_backward", device, *(x.data_ptr() for x in seq), d_output.data_ptr(),
                      None if d_final_state is None else d_final_state[part].data_ptr(), _lib.ptr(chunk_states),
                      _lib.ptr(d_chunk_states), _lib.ptr(span_states), _lib.ptr(d_span_states), _lib.ptr(workspace),
                      _lib.ptr(scratch), *(x.data_ptr() for x in grads), d_state[part].data_ptr(), group.bounds,
                      group.last - group.first, total, heads, _lib.dtype_code(q.dtype), _lib.dtype_code(g.dtype),
                      scale, _lib.stream_ptr(device),
                      kernels=2 * (group.chunks > 0) + 2 * (group.span_slots > 0))
        return (*grads, d_state if ctx.has_initial_state else None, None, None)


def _dense(tensor):
    """Contiguous and 16-byte aligned, as the kernels' copies need it (nearly always already so)."""

    tensor = tensor if tensor.is_contiguous() else tensor.contiguous()
    return tensor if tensor.data_ptr() % 16 == 0 else tensor.clone()


def chunk_gdn2_varlen(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    g: torch.Tensor,
    beta: torch.Tensor,
    w: torch.Tensor,
    cu_seqlens,
    initial_state: torch.Tensor | None = None,
    *,
    scale: float | None = None,
    output_final_state: bool = False,
    use_qk_l2norm_in_kernel: bool = False,
    use_gate_in_kernel: bool = False,
) -> tuple[torch.Tensor, torch.Tensor | None]:
    """``chunk_gdn2`` over ``N`` sequences packed along time.

    Sequence tensors are contiguous ``[1, total, H, 128]`` (same dtype rules as ``chunk_gdn2``);
    ``cu_seqlens`` holds ``N + 1`` cumulative lengths (tensor or sequence of ints, read on the host);
    ``initial_state`` is ``None`` or fp32 ``[N, H, 128, 128]``.  Returns the packed output and,
    when asked for, the ``[N, H, 128, 128]`` final states.  Differentiable like ``chunk_gdn2``.
    """

    if not isinstance(q, torch.Tensor) or q.ndim != 4 or q.shape[0] != 1:
        raise ValueError("packed sequence tensors must have shape [1, total, H, 128]")
    bounds = _bounds(cu_seqlens, q.shape[1])
    output_scale = float(scale) if scale is not None else 1.0 / math.sqrt(_DIM)
    if not math.isfinite(output_scale):
        raise ValueError("scale must be finite")
    _validate.sequence_inputs(q, k, v, g, beta, w, need_alignment=True)
    n_seq, heads = len(bounds) - 1, q.shape[2]
    if initial_state is not None:
        _validate.state("initial_state", initial_state, n_seq, heads, q.device, need_alignment=True)
    wants_grad = torch.is_grad_enabled() and any(
        isinstance(t, torch.Tensor) and t.requires_grad for t in (q, k, v, g, beta, w, initial_state)
    )
    if wants_grad:
        # training: materialise the activated tensors once for the whole packed batch
        if use_qk_l2norm_in_kernel or use_gate_in_kernel:
            q, k, g, beta, w = gate_prologue(q, k, g, beta, w, normalize_qk=use_qk_l2norm_in_kernel,
                                             activate_gates=use_gate_in_kernel)
        output, final_state = _ChunkGDN2Varlen.apply(q, k, v, g, beta, w, initial_state, bounds, output_scale)
    else:
        seq = tuple(_validate.detached(x) for x in (q, k, v, g, beta, w))
        output, final_state, _, _ = _packed_forward(
            seq, _validate.detached(initial_state), bounds, output_scale, False,
            _prologue_flags(use_qk_l2norm_in_kernel, use_gate_in_kernel))
    return output, final_state if output_final_state else None


def expand_grouped_heads(q, k, g, beta, value_heads: int):
    """Expand key-shaped tensors ``[B, T, Hk, 128]`` to ``value_heads = Hk * r`` heads.

    Value head ``j`` uses key head ``j // r``.  Returns contiguous ``[B, T, value_heads, 128]``
    tensors; under autograd the gradients of the ``r`` value heads of a group add up in the shared
    key head."""

    key_heads = q.shape[2]
    if value_heads <= 0 or value_heads % key_heads:
        raise ValueError("value_heads must be a positive multiple of the number of key heads")
    repeat = value_heads // key_heads
    if repeat == 1:
        return q, k, g, beta
    return tuple(t.repeat_interleave(repeat, dim=2) for t in (q, k, g, beta))


__all__ = ["chunk_gdn2_varlen", "expand_grouped_heads"]
