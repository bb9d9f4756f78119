"""Recurrences over runs of many tokens in chunks of 64, as float32 matrix products: the matrix memory (csrc/recurrence.cuh, in the
library of csrc/ssm.cu) and the delta rule with one decay per head (csrc/delta_chunks.cu)."""
from __future__ import annotations

from ctypes import c_float, c_longlong, c_void_p
from functools import lru_cache
from typing import Optional, Sequence

import torch

from ..csrc.build import load_kernel
from ._call import KernelError, check, ints, ptr, stream, want_f32, want_int32
from .gemm_tc import status_word
from .ssm import ctypes_ptr

_LIB = "ssm"
CHUNK = 64               # csrc/chunks.cuh L
SIZES = (64, 128)        # key and value sizes the kernels are built for
# the most bytes of chunks' states a step holds at a time, 126 chunks of 16 heads of 128 x 129; longer steps go in groups of equal size
# (8,192 tokens of that layer: 780 us in one piece, 788 in two groups; of the delta rule, whose chunks take 130 KB a head, 1,102 and 1,163)
SCRATCH_BYTES = 128 << 20


def chunks_of(q_lens: Sequence[int], n_tokens: int, n_seqs: int) -> int:
    """Chunks of a step's runs (without the lengths on the host: at most)."""
    if len(q_lens) == n_seqs:
        return sum(-(-n // CHUNK) for n in q_lens)
    return n_tokens // CHUNK + n_seqs


def group_of(chunks: int, heads: int, dk: int, dv: int) -> int:
    """Chunks whose states a step holds at a time."""
    most = max(1, SCRATCH_BYTES // (4 * heads * ((dv + 1) * dk + 1)))
    return -(-chunks // -(-chunks // most)) if chunks else 1


def takes(dk: int, dv: int) -> bool:
    """Whether the kernels are built for keys and values of these sizes."""
    return dk in SIZES and dv in SIZES


def usable(dk: int, dv: int, rows: torch.Tensor, *offsets: int) -> bool:
    """Whether the kernels take this shape: sizes of 64 or 128, rows and offsets of whole 16 bytes."""
    return takes(dk, dv) and rows.shape[1] % 4 == 0 and all(o % 4 == 0 for o in offsets) \
        and rows.is_contiguous() and rows.data_ptr() % 16 == 0


def memory_chunks(rows: torch.Tensor, q_off: int, k_off: int, v_off: int, gates: torch.Tensor, state: torch.Tensor, y: torch.Tensor,
                  dots: torch.Tensor, chunks: int, heads: int, dk: int, dv: int, cu_seqlens: torch.Tensor, slots: torch.Tensor) -> None:
    """`kernels.ssm.memory_scan` with outputs, in chunks: state float32 [slots, heads, dv + 1, dk] (rows may be strided) is renewed,
    y [T, heads * dv], dots [T, heads].  chunks: at least the chunks of the runs (`chunks_of`), in groups of `group_of`."""
    for t, what in ((rows, "q, k and v"), (gates, "the gates"), (state, "the state"), (y, "the output"), (dots, "the dot products")):
        want_f32(t, what)
    for t, what in ((cu_seqlens, "cu_seqlens"), (slots, "slots")):
        want_int32(t, what)
    T, n_seqs = rows.shape[0], cu_seqlens.shape[0] - 1
    if not usable(dk, dv, rows, q_off, k_off, v_off) or tuple(state.shape[1:]) != (heads, dv + 1, dk) or not state[0].is_contiguous() \
            or y.numel() != T * heads * dv or dots.numel() != T * heads or gates.numel() != 2 * T * heads or slots.numel() < n_seqs \
            or max(q_off + heads * dk, k_off + heads * dk, v_off + heads * dv) > rows.shape[1]:
        raise KernelError("memory_chunks: sizes of 64 or 128, aligned rows that hold the heads, a state row of [heads, dv + 1, dk]")
    per_chunk, group = heads * (dv + 1) * dk, group_of(chunks, heads, dk, dv)
    scratch = torch.empty(group * (per_chunk + heads), dtype=torch.float32, device=rows.device)      # the chunks' states, then their decays
    at = scratch.data_ptr()
    lib = load_kernel(_LIB)
    check(_LIB, lib.tq_memory_chunks(
        ptr(rows), *ints(rows.shape[1], q_off, k_off, v_off), ptr(gates), ctypes_ptr(state), c_longlong(state.stride(0)), ptr(y), ptr(dots),
        c_void_p(at), c_void_p(at + 4 * group * per_chunk), *ints(chunks, group, n_seqs, heads, dk, dv), ptr(cu_seqlens), ptr(slots), stream()), kernels=3 * -(-chunks // group))


@lru_cache(maxsize=256)
def delta_bytes(group: int, heads: int, kv_heads: int, dk: int, dv: int) -> int:
    """Bytes of scratch that a group of the delta rule's chunks takes (csrc/delta_chunks.cu); as many times those of one chunk."""
    lib = load_kernel("delta_chunks")
    lib.tq_delta_chunks_bytes.restype = c_longlong
    return int(lib.tq_delta_chunks_bytes(*ints(group, heads, kv_heads, dk, dv)))


@lru_cache(maxsize=256)
def delta_rows_width(heads: int, kv_heads: int, dk: int) -> int:
    """Floats of a token's prepared row with one decay per head (csrc/ssm.cu)."""
    return int(load_kernel(_LIB).tq_delta_rows_width(*ints(heads, kv_heads, dk, 1)))


def delta_chunks(xqkv: torch.Tensor, q_off: int, k_off: int, v_off: int, proj: torch.Tensor, b_off: int, a_raw: torch.Tensor, a_off: int,
                 dt_bias: torch.Tensor, a_log: torch.Tensor, state: torch.Tensor, y: torch.Tensor, chunks: int, heads: int, kv_heads: int, dk: int,
                 dv: int, unit_eps: float, q_scale: float, cu_seqlens: torch.Tensor, slots: torch.Tensor,
                 status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """`kernels.ssm.delta_scan_runs` with one decay per head, in chunks: dk and dv 64 or 128 (`usable`); chunks: at least the chunks of the
    runs (`chunks_of`), as many at a time as SCRATCH_BYTES hold."""
    for t, what in ((xqkv, "q, k and v"), (proj, "the projection"), (a_raw, "the raw decays"), (dt_bias, "the decays' bias"),
                    (a_log, "the decay rates"), (state, "the state"), (y, "the output")):
        want_f32(t, what)
    for t, what in ((cu_seqlens, "cu_seqlens"), (slots, "slots")):
        want_int32(t, what)
    T, n_seqs = xqkv.shape[0], cu_seqlens.shape[0] - 1
    if not usable(dk, dv, xqkv, v_off) or tuple(state.shape[1:]) != (heads, dv, dk) or not state[0].is_contiguous() or y.numel() != T * heads * dv \
            or dt_bias.numel() != heads or a_log.numel() != heads or slots.numel() < n_seqs or y.data_ptr() % 16:
        raise KernelError("delta_chunks: sizes of 64 or 128, aligned rows, one decay per head, a state row of [heads, vdim, dim]")
    if chunks == 0:
        return y
    lib, at, st = load_kernel(_LIB), stream(), ptr(xqkv)
    each = delta_bytes(1, heads, kv_heads, dk, dv)
    group = -(-chunks // -(-chunks // max(1, SCRATCH_BYTES // each)))
    # one buffer: the chunks' scratch, then the prepared rows
    width = delta_rows_width(heads, kv_heads, dk)
    buf = torch.empty(group * each + 4 * T * width, dtype=torch.uint8, device=xqkv.device)
    rows = c_void_p(buf.data_ptr() + group * each)
    check(_LIB, lib.tq_delta_prepare(
        st, *ints(xqkv.shape[1], q_off, k_off), ptr(proj), *ints(proj.shape[1], b_off), ptr(a_raw), *ints(a_raw.shape[1], a_off, 1), ptr(dt_bias),
        ptr(a_log), rows, *ints(T, heads, kv_heads, dk), c_float(unit_eps), c_float(q_scale), at))
    check("delta_chunks", load_kernel("delta_chunks").tq_delta_chunks(
        rows, *ints(width), st, *ints(xqkv.shape[1], v_off), ctypes_ptr(state), c_longlong(state.stride(0)), ptr(y), ptr(buf),
        *ints(chunks, group, n_seqs, heads, kv_heads, dk, dv), ptr(cu_seqlens), ptr(slots), ptr(status if status is not None else status_word(xqkv.device)),
        at), kernels=3 * -(-chunks // group))
    return y
