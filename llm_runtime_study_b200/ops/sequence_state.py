"""Kernels of mixers that keep a state of fixed size per request: the linear scan (plain or delta
rule, constant or per-row decay), the short convolution's bookkeeping, and the gated group norm of
the read-out.  The state and everything that enters the recurrence are float32."""

from __future__ import annotations

from typing import Sequence

import torch

from ..errors import KernelError
from . import native
from .native import c_float, c_int, c_void_p, call, ptr, require, stream_ptr, tag

native.register_library(
    "b200_scan_chunks", ("scan_chunks.cu",),
    {"b200_scan_chunks": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, *[c_void_p] * 12, *[c_int] * 9, c_float, c_int, c_int, c_void_p],
     "b200_scan_chunks_record_floats": [c_int, c_int],
     "b200_scan_chunks_error": [],
     "b200_scan_single": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, *[c_void_p] * 11, *[c_int] * 6, c_float, c_int, c_int, c_void_p]},
)

native.register_error_probe("b200_scan_chunks", "b200_scan_chunks_error", "linear scan in chunks")

CHUNK_TOKENS, CHUNK_MAX_DIM = 16, 128     # tokens a chunk, largest key size of the chunked kernel
CHUNK_MIN_TOKENS = 48                     # tokens beyond one per request from which a batch may be scanned in chunks
CHUNK_MAX_NUMBERS = 1 << 28               # numbers in the records of a batch at most: a limit on work (2,048 tokens of 32 heads of 128: 1 << 24.7)
# Bytes of records that are there at once, in one launch.  2,048 tokens of 32 heads of 128 with the delta rule are 181 MB (a number is three bfloat16);
# cut in two the scan takes 20 to 30 us more, 32 portions of 34 tokens of 64 heads 1.4 times as long.
CHUNK_SLICE_BYTES = 1 << 28
MOST_RUNS = 4                             # launches a batch of long and short portions is cut into at most


def _lengths(lens: "Sequence[int] | None", n: int, entries: int) -> "Sequence[int] | None":
    """The entries' lengths, checked; those of a single entry are known without being told."""

    if lens is None:
        return [n] if entries == 1 else None
    if len(lens) != entries or sum(lens) != n or min(lens, default=0) < 0:
        raise KernelError(f"{len(lens)} lengths that add up to {sum(lens)} do not describe {n} rows of {entries} entries")
    return lens


def _record_numbers(n: int, entries: int, heads: int, dim: int) -> int:
    """How many numbers the records of a batch hold (the larger form, the delta rule's)."""

    dim = 32 if dim <= 32 else (64 if dim <= 64 else 128)
    return (n // CHUNK_TOKENS + entries) * heads * (3 * CHUNK_TOKENS * dim + 2 * CHUNK_TOKENS * CHUNK_TOKENS + dim)


def scans_in_chunks(n: int, entries: int, heads: int, dim: int, fixed_order: bool) -> bool:
    """Whether a batch of ``n`` tokens of ``entries`` requests can hold portions that are scanned sixteen tokens at a time
    (``csrc/scan_chunks.cu``; ``portion_in_chunks`` says which): batches with portions of prompts beside 16-bit activations.  With
    ``fixed_order`` a token's sums must not depend on where a step's chunks begin.  Batches of more than ``CHUNK_MAX_NUMBERS`` are scanned
    token by token (the memory that records take is bounded by ``CHUNK_SLICE_BYTES`` whatever the batch)."""

    return (not fixed_order and dim <= CHUNK_MAX_DIM and n - entries >= CHUNK_MIN_TOKENS
            and _record_numbers(n, entries, heads, dim) <= CHUNK_MAX_NUMBERS)


def portion_in_chunks(lens: "Sequence[int]", heads: int, dim: int, columns: int, delta: bool, row_gates: bool = False) -> int:
    """The number of tokens from which a portion of a batch is scanned in chunks (0: none is); ``columns``: of a head's state.

    ``row_gates``: the state has the normaliser as one more column.

    A chunk costs 1.6 us, 2.6 with the delta rule, behind some 8 us for the records; a token of a chain 0.2 us as long as the chains' CTAs of 8 columns
    all run at once, two an SM, and 0.3 to 0.5 us beyond that.  A chunk takes the same 0.04 us a head (0.06 with the
    delta rule) whether it holds sixteen tokens or one.  So what counts is the portion's own length, not the batch's.  Microseconds in
    chunks and as a chain, 128 x 128, one decay a head (delta rule, a decay per channel): 4 heads, one portion of 64 tokens 11.9, 13.8 (18.2, 19.5), of 96
    14.0, 19.3 (21.5, 27.8); 16 heads, 64 tokens 12.0, 15.8 (18.4, 24.3), 96 tokens 14.1, 22.2 (21.5, 34.9); 32 heads, eight of 24 28.7, 41.8 (41.5, 66.6), two of
    48 14.1, 29.5 (22.1, 50.3), eight of 48 37.0, 75.0 (61.7, 121.9), 64 of 2 167, 82 (224, 100).  With key sizes up to 64 and enough chains to
    fill the GPU with CTAs of 32 columns a chain is as fast or faster for short values (8 heads of 64, 64 portions of 64: 49.4, 38.1;
    82.7, 58.4).  Few chains beside requests of another kernel pay for that launch too (4 heads, 64 tokens beside one token: 15.3, 13.8).
    With row gates a head of 128 columns is five blocks of 32, and short portions pay only from 28 tokens on (16 heads, eight of 24 to 28 tokens 1.01 to
    0.91 of the chain's time) and where their CTAs are not just more than fit at once, two an SM (four of 32: 23.6, 21.8, six 0.76); with 96 rows of state, which
    are worked on as 128, not at all (four to 32 of 32 tokens: 0.90 to 1.40).  These lines hold with what runs today but lie on the chain's side: several short portions with the
    delta rule and single ones of 64 tokens would be faster in chunks."""

    sms = native.sm_count()
    if not delta and dim > 64:                 # many portions, each as long as two chunks or nearly
        least = 28 if row_gates else 24
        short = sum(m >= least for m in lens)
        ctas = short * heads * -(-columns // 32)
        if short >= 4 and short * heads * -(-columns // 8) > 4 * sms and not (row_gates and (dim <= 96 or 2 * sms < ctas <= 3 * sms)):
            return least
    long = sum(m >= 48 for m in lens)
    if not long or (dim <= 64 and long * heads * -(-columns // 32) >= 2 * sms):
        return 0
    ctas = long * heads * -(-columns // 8)
    if ctas > 2 * sms:
        return 48
    if ctas <= sms and long < len(lens):
        return 128 if delta else 96
    return 96 if delta else 64


def scan_runs(lens: "Sequence[int]", least: int) -> "list[tuple[str, int, int]]":
    """A batch as runs of neighbouring requests, ``(kind, first, last + 1)``: "chunks" for portions of ``least`` tokens and more,
    "single" for requests of one token each, "chain" for all others.  More than two runs are for portions of 128 tokens and more only
    (16 heads, requests of 1, 1, 1, 1, 60, 3 and 60 tokens: 49 us in four launches, 45 in one), and more than four are one chain."""

    runs: list[tuple[str, int, int]] = []
    at = 0

    def others(last: int) -> None:
        if at < last:
            runs.append(("single" if min(lens[at:last]) == max(lens[at:last]) == 1 else "chain", at, last))

    for i in [i for i, m in enumerate(lens) if m >= least] if least else ():
        if runs and runs[-1][0] == "chunks" and at == i:
            runs[-1] = ("chunks", runs[-1][1], i + 1)
        else:
            others(i)
            runs.append(("chunks", i, i + 1))
        at = i + 1
    others(len(lens))
    if len(runs) > 2 and least < 128:
        return scan_runs(lens, 128)
    return runs if len(runs) <= MOST_RUNS else [("chain", 0, len(lens))]


def _scan_plan(lens, n: int, entries: int, heads: int, dim: int, vdim: int, columns: int, delta: bool, fixed_order: bool):
    """The kernels of a batch, as ``scan_runs`` names them, with what is left of its choice: single tokens whose sizes their kernel
    does not take are chains.  Lengths that are not known are taken for equal ones, none of them for single tokens."""

    least = 0
    if scans_in_chunks(n, entries, heads, dim, fixed_order):
        least = portion_in_chunks(lens if lens else [n // entries] * entries, heads, dim, columns, delta, columns > vdim)
    if not lens:
        return [("chunks" if least and n >= least * entries else "chain", 0, entries)]
    singles = scans_single(1, 1, dim, vdim, fixed_order)
    return [("chain" if kind == "single" and not singles else kind, first, last) for kind, first, last in scan_runs(lens, least)]


def _parts(plan, lens, n: int):
    """The runs of a plan with their numbers of rows and of chunks (without lengths: at most so many, every request's last chunk
    may be short)."""

    for kind, first, last in plan:
        if lens:
            mine = lens[first:last]
            yield kind, first, last, sum(mine), sum(-(-m // CHUNK_TOKENS) for m in mine)
        else:
            yield kind, first, last, n, n // CHUNK_TOKENS + last - first


def chunk_slices(lens: "Sequence[int] | None", n: int, entries: int, chunks: int, chunk_bytes: int) -> "list[tuple[int, int, int]]":
    """The launches of portions scanned in chunks, ``(skip, most, chunks)``: of every request the tokens from ``skip`` on, ``most`` at
    most, ``chunks`` of them in all.  One launch as long as the records of all chunks take no more than ``CHUNK_SLICE_BYTES``, else as many
    tokens of every request at a time as fit (a chunk of each at least)."""

    fit = CHUNK_SLICE_BYTES // chunk_bytes
    if chunks <= fit:
        return [(0, max(n, 1), chunks)]
    most = CHUNK_TOKENS * max(1, fit // entries)
    longest = max(lens) if lens else n
    return [(skip, most, sum(-(-min(most, max(0, m - skip)) // CHUNK_TOKENS) for m in lens) if lens else most // CHUNK_TOKENS * entries)
            for skip in range(0, longest, most)]


def _scan_chunks(q, k, v, *, chunks, lens, heads, qk_heads, dim, vdim, state, q_start, slots, out, gate=None, decay=None, row_decay=None, row_gain=None,
                 beta=None, norm_state=None, norm_out=None, silu=False, q_scale=1.0) -> None:
    entries = slots.shape[0]
    floats = native.query("b200_scan_chunks_record_floats", dim, 0 if beta is None else 1)
    slices = chunk_slices(lens, q.shape[0], entries, chunks, heads * floats * 4)
    records = torch.empty(max(held for _, _, held in slices) * heads * floats, dtype=torch.float32, device=q.device)
    for skip, most, held in slices:
        call("b200_scan_chunks", ptr(q), ptr(k), ptr(v), q.stride(0), k.stride(0), v.stride(0), ptr(gate), ptr(decay), ptr(row_decay),
             ptr(row_gain), ptr(beta), ptr(state), ptr(norm_state), ptr(norm_out), ptr(out), ptr(records), ptr(q_start), ptr(slots), entries, held,
             skip, most, heads, qk_heads, dim, vdim, 1 if silu else 0, float(q_scale), tag(q.dtype), tag(v.dtype), stream_ptr(), launches=2)


def scans_single(n: int, entries: int, dim: int, vdim: int, fixed_order: bool, lens: "Sequence[int] | None" = None) -> bool:
    """Whether requests of one token each go to the kernel that holds a head's state in a CTA's registers: whole 16-byte
    columns, key sizes up to 128; faster at every batch from one request on (8 requests of 32 heads of 128: 7.9 us against 13.4).  (With
    ``fixed_order`` a token's sums are those of the token-by-token kernel.)  The kernel takes row ``q_start[e]`` of every entry and
    looks at no other, so as many tokens as requests is not enough: ``lens`` (the entries' lengths) must all be one."""

    return (not fixed_order and n == entries and (lens is None or all(m == 1 for m in lens)) and dim <= CHUNK_MAX_DIM
            and vdim % 4 == 0)


def _scan_single(q, k, v, *, heads, qk_heads, dim, vdim, state, q_start, slots, out, gate=None, decay=None, row_decay=None, row_gain=None,
                 beta=None, norm_state=None, norm_out=None, silu=False, q_scale=1.0) -> None:
    call("b200_scan_single", ptr(q), ptr(k), ptr(v), q.stride(0), k.stride(0), v.stride(0), ptr(gate), ptr(decay), ptr(row_decay),
         ptr(row_gain), ptr(beta), ptr(state), ptr(norm_state), ptr(norm_out), ptr(out), ptr(q_start), ptr(slots), slots.shape[0], heads, qk_heads,
         dim, vdim, 1 if silu else 0, float(q_scale), tag(q.dtype), tag(v.dtype), stream_ptr())


def _chunk_form(q: torch.Tensor, v: torch.Tensor, gate, decay, beta) -> bool:
    """Whether the kernels for chunks and for single tokens have this form of the scan: what bfloat16 models run."""

    if beta is not None:
        return decay is None and q.dtype == v.dtype == torch.float32
    return v.dtype == torch.bfloat16 and (decay is not None or (gate is not None and q.dtype == torch.bfloat16))


def linear_scan(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, heads: int, qk_heads: int, dim: int, vdim: int,
    state: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor, gate: torch.Tensor | None = None,
    decay: torch.Tensor | None = None, beta: torch.Tensor | None = None, silu: bool = False, q_scale: float = 1.0,
    fixed_order: bool = False, row_decay: torch.Tensor | None = None, lens: "Sequence[int] | None" = None,
) -> torch.Tensor:
    """Per request (entry ``e`` owns rows ``q_start[e] .. q_start[e+1]-1`` and the state row ``slots[e]``) and head,
    token after token: ``S <- D S + k u^T``, ``o = S^T q`` with ``D`` the head's constant ``decay`` or the row's
    ``gate`` factors (one per key channel) or, with ``beta``, the row's one factor per head ``row_decay`` (``[N, heads]``), and ``u = v``
    or, with ``beta``, ``beta (v - (D S)^T k)``.  ``q`` and
    ``k`` are ``[N, qk_heads * dim]`` column blocks (a row stride of their own is fine), ``v`` ``[N, heads * vdim]``;
    head ``h`` reads q/k head ``h // (heads / qk_heads)``.  ``silu`` applies SiLU to q, k and v as they are read;
    q is multiplied by ``q_scale`` then.  ``v`` may be bfloat16 beside float32 ``q`` and ``k`` (constant decay, no ``beta``).
    ``state`` is ``[slots, heads, dim, vdim]`` float32 and is updated in place.  ``fixed_order``: every sum is formed in
    an order that does not depend on the shape of the batch (the kernel otherwise spreads a column over more lanes when few
    requests bring long portions), so a token's bits do not depend on the cut.  ``lens``: the entries' numbers of rows on the host
    (what ``q_start`` holds on the device); known, they send single tokens, short and long portions each to a kernel of their
    own.  Returns float32 ``[N, heads * vdim]``."""

    n = q.shape[0]
    for t, name, width in ((q, "q", qk_heads * dim), (k, "k", qk_heads * dim), (v, "v", heads * vdim)):
        if t.device.type != "cuda" or t.dim() != 2 or t.shape != (n, width) or t.stride(1) != 1 or (name == "k" and t.dtype != q.dtype):
            raise KernelError(f"{name} must be CUDA rows [{n}, {width}] with unit column stride, q and k of one type")
    if v.dtype != q.dtype and (beta is not None or decay is None or q.dtype != torch.float32):
        raise KernelError("linear_scan takes v in another type than q and k with a constant decay and float32 q and k only")
    require(state, "state", dtype=torch.float32, dims=4)
    if tuple(state.shape[1:]) != (heads, dim, vdim):
        raise KernelError(f"state has shape {tuple(state.shape)}, expected [slots, {heads}, {dim}, {vdim}]")
    require(q_start, "q_start", dtype=torch.int32, dims=1)
    entries = q_start.shape[0] - 1
    require(slots, "slots", dtype=torch.int32, shape=(entries,))
    lens = _lengths(lens, n, entries)
    if sum(t is not None for t in (gate, decay, row_decay)) != 1:
        raise KernelError("linear_scan takes one of: gate factors per row and channel, one decay per row and head, one decay per head")
    if row_decay is not None:
        require(row_decay, "row_decay", dtype=torch.float32, shape=(n, heads))
        if beta is None:
            raise KernelError("linear_scan takes one decay per row and head with the delta rule only (linear_scan_row_gates otherwise)")
    elif gate is not None:
        require(gate, "gate", dtype=torch.float32, shape=(n, heads * dim))
    else:
        require(decay, "decay", dtype=torch.float32, shape=(heads,))
    if beta is not None:
        require(beta, "beta", dtype=torch.float32, shape=(n, heads))
    out = torch.empty((n, heads * vdim), dtype=torch.float32, device=q.device)
    plan = [("chain", 0, entries)]
    if _chunk_form(q, v, gate, decay, beta):
        plan = _scan_plan(lens, n, entries, heads, dim, vdim, vdim, beta is not None, fixed_order)
    for kind, first, last, rows, chunks in _parts(plan, lens, n):
        starts, at = (q_start, slots) if last - first == entries else (q_start[first : last + 1], slots[first:last])
        shared = dict(heads=heads, qk_heads=qk_heads, dim=dim, vdim=vdim, state=state, q_start=starts, slots=at, out=out, gate=gate, decay=decay,
                      row_decay=row_decay, beta=beta, silu=silu, q_scale=q_scale)
        if kind == "single" and state.data_ptr() % 16 == 0:
            _scan_single(q, k, v, **shared)
        elif kind == "chunks":
            _scan_chunks(q, k, v, chunks=chunks, lens=lens[first:last] if lens else None, **shared)
        else:
            call("b200_linear_scan", ptr(q), ptr(k), ptr(v), q.stride(0), k.stride(0), v.stride(0), ptr(gate), heads * dim, ptr(decay),
                 ptr(row_decay), ptr(beta), heads, ptr(state), ptr(out), heads * vdim, ptr(starts), ptr(at), last - first, rows, heads, qk_heads, dim, vdim,
                 1 if silu else 0, float(q_scale), 1 if fixed_order else 0, tag(q.dtype), tag(v.dtype), stream_ptr())
    return out


def linear_scan_row_gates(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, heads: int, dim: int, vdim: int, decay: torch.Tensor, gain: torch.Tensor,
    state: torch.Tensor, norm_state: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor, q_scale: float = 1.0,
    fixed_order: bool = False, lens: "Sequence[int] | None" = None,
) -> tuple[torch.Tensor, torch.Tensor]:
    """``linear_scan`` with one decay and one input gain per row and head, and a normaliser: ``S <- decay S + gain k v^T``,
    ``n <- decay n + gain k``; returns ``S^T q`` float32 ``[N, heads * vdim]`` and ``n . q`` float32 ``[N, heads]`` (q times
    ``q_scale`` as it is read).  ``state`` ``[slots, heads, dim, vdim]`` and ``norm_state`` ``[slots, heads, dim]`` float32 are
    updated in place; ``decay`` and ``gain`` are float32 ``[N, heads]``.  ``fixed_order`` and ``lens`` as for
    ``linear_scan``."""

    n = q.shape[0]
    for t, name, width in ((q, "q", heads * dim), (k, "k", heads * dim), (v, "v", heads * vdim)):
        if t.device.type != "cuda" or t.dim() != 2 or t.shape != (n, width) or t.stride(1) != 1 or t.dtype != q.dtype:
            raise KernelError(f"{name} must be CUDA rows [{n}, {width}] of one type with unit column stride")
    require(state, "state", dtype=torch.float32, dims=4)
    require(norm_state, "norm_state", dtype=torch.float32, dims=3)
    if tuple(state.shape[1:]) != (heads, dim, vdim) or tuple(norm_state.shape[1:]) != (heads, dim) or norm_state.shape[0] != state.shape[0]:
        raise KernelError(f"states have shapes {tuple(state.shape)} and {tuple(norm_state.shape)}, expected [slots, {heads}, {dim}, {vdim}] "
                          f"and [slots, {heads}, {dim}]")
    require(decay, "decay", dtype=torch.float32, shape=(n, heads))
    require(gain, "gain", dtype=torch.float32, shape=(n, heads))
    require(q_start, "q_start", dtype=torch.int32, dims=1)
    entries = q_start.shape[0] - 1
    require(slots, "slots", dtype=torch.int32, shape=(entries,))
    lens = _lengths(lens, n, entries)
    out = torch.empty((n, heads * vdim), dtype=torch.float32, device=q.device)
    norm_out = torch.empty((n, heads), dtype=torch.float32, device=q.device)
    plan = [("chain", 0, entries)]
    if q.dtype == torch.bfloat16:
        plan = _scan_plan(lens, n, entries, heads, dim, vdim, vdim + 1, False, fixed_order)      # the normaliser is a column of the state
    for kind, first, last, rows, chunks in _parts(plan, lens, n):
        starts, at = (q_start, slots) if last - first == entries else (q_start[first : last + 1], slots[first:last])
        shared = dict(heads=heads, qk_heads=heads, dim=dim, vdim=vdim, state=state, q_start=starts, slots=at, out=out, row_decay=decay,
                      row_gain=gain, norm_state=norm_state, norm_out=norm_out, q_scale=q_scale)
        if kind == "single" and state.data_ptr() % 16 == 0:
            _scan_single(q, k, v, **shared)
        elif kind == "chunks":
            _scan_chunks(q, k, v, chunks=chunks, lens=lens[first:last] if lens else None, **shared)
        else:
            call("b200_linear_scan_row_gates", ptr(q), ptr(k), ptr(v), q.stride(0), k.stride(0), v.stride(0), ptr(decay), ptr(gain), ptr(state),
                 ptr(norm_state), ptr(out), ptr(norm_out), ptr(starts), ptr(at), last - first, rows, heads, dim, vdim, float(q_scale),
                 1 if fixed_order else 0, tag(q.dtype), stream_ptr())
    return out, norm_out


def memory_gates(
    proj: torch.Tensor, *, heads: int, i_offset: int, f_offset: int, i_bias: torch.Tensor, f_bias: torch.Tensor, cap: float,
    m_state: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor,
) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """Exponential gates kept in range by a running maximum.  With ``i = cap tanh((zi + i_bias) / cap)`` and
    ``f = ln sigmoid(cap tanh((zf + f_bias) / cap))`` (logits: columns ``i_offset + h`` and ``f_offset + h`` of ``proj``), token after
    token: ``m_t = max(f + m_(t-1), i)`` from the slot's ``m`` (``m_state`` float32 ``[slots, heads]``, updated in place).  Returns
    float32 ``[N, heads]`` each: ``exp(f + m_(t-1) - m_t)``, ``exp(i - m_t)`` and ``exp(-m_t)``."""

    require(proj, "proj", dims=2)
    n, ld = proj.shape
    require(i_bias, "i_bias", dtype=torch.float32, shape=(heads,))
    require(f_bias, "f_bias", dtype=torch.float32, shape=(heads,))
    require(m_state, "m_state", dtype=torch.float32, dims=2)
    if m_state.shape[1] != heads or max(i_offset, f_offset) + heads > ld:
        raise KernelError("memory_gates: the logits lie outside the rows, or the state has another number of heads")
    require(q_start, "q_start", dtype=torch.int32, dims=1)
    entries = q_start.shape[0] - 1
    require(slots, "slots", dtype=torch.int32, shape=(entries,))
    decay, gain, floor = torch.empty((3, n, heads), dtype=torch.float32, device=proj.device)
    call("b200_memory_gates", ptr(proj), ld, i_offset, f_offset, ptr(i_bias), ptr(f_bias), float(cap), ptr(m_state), ptr(decay), ptr(gain),
         ptr(floor), ptr(q_start), ptr(slots), entries, heads, tag(proj.dtype), stream_ptr())
    return decay, gain, floor


def channel_decay(proj: torch.Tensor, up: torch.Tensor, bias: torch.Tensor, *, offset: int, tau: float) -> torch.Tensor:
    """Decays per key channel from a low-rank map: ``sigmoid(proj[:, offset : offset + rank] @ up + bias)^(1 / tau)``, float32
    ``[N, width]``; ``up`` is ``[rank, width]`` (the map's weight transposed) in the type of ``proj``."""

    require(proj, "proj", dims=2)
    n, ld = proj.shape
    require(up, "up", dtype=proj.dtype, dims=2)
    rank, width = up.shape
    require(bias, "bias", dtype=torch.float32, shape=(width,))
    if offset + rank > ld:
        raise KernelError("channel_decay: the low-rank columns lie outside the rows")
    alpha = torch.empty((n, width), dtype=torch.float32, device=proj.device)
    call("b200_channel_decay", ptr(proj), ld, offset, rank, ptr(up), ptr(bias), float(tau), ptr(alpha), n, width, tag(proj.dtype),
         stream_ptr())
    return alpha


def delta_prepare(
    proj: torch.Tensor, *, heads: int, qk_heads: int, dim: int, vdim: int, beta_offset: int, low_offset: int, rank: int,
    taps: torch.Tensor, conv_state: torch.Tensor, a_log: torch.Tensor, dt_bias: torch.Tensor, a_up: torch.Tensor | None,
    q_start: torch.Tensor, slots: torch.Tensor, token_entry: torch.Tensor, unit_eps: float, q_scale: float,
):
    """From one stacked projection ``[N, q | k | v | ...]``: the short convolution over time and SiLU of every q, k
    and v channel (inputs before the step come from ``conv_state`` ``[slots, taps-1, channels]``), each q and k head
    divided by ``sqrt(sum of squares + unit_eps)`` (q times ``q_scale``), ``beta = sigmoid(proj[:, beta_offset + h])``
    and the decay factors ``exp(-exp(a_log[h]) * softplus(proj[:, low_offset : low_offset + rank] @ a_up + dt_bias))``
    (``a_up`` is ``[rank, heads * dim]``: the map's weight transposed, so that neighbouring threads read neighbouring outputs).
    ``rank`` 0 (``a_up`` ``None``): one decay per head, ``exp(-exp(a_log[h]) * softplus(proj[:, low_offset + h] + dt_bias[h]))``, and ``g``
    is ``[N, heads]``.
    Returns float32 ``(q, k, v, g, beta)``."""

    require(proj, "proj", dims=2)
    n, ld = proj.shape
    channels = 2 * qk_heads * dim + heads * vdim
    require(taps, "taps", dtype=torch.float32, dims=2)
    ntaps = taps.shape[1]
    if taps.shape[0] != channels:
        raise KernelError(f"taps has {taps.shape[0]} channels, expected {channels}")
    require(conv_state, "conv_state", dtype=torch.float32, dims=3)
    if tuple(conv_state.shape[1:]) != (ntaps - 1, channels):
        raise KernelError(f"conv_state has shape {tuple(conv_state.shape)}, expected [slots, {ntaps - 1}, {channels}]")
    require(a_log, "a_log", dtype=torch.float32, shape=(heads,))
    decays = heads * dim if rank else heads
    require(dt_bias, "dt_bias", dtype=torch.float32, shape=(decays,))
    if rank:
        require(a_up, "a_up", dtype=proj.dtype, shape=(rank, heads * dim))
    if max(beta_offset + heads, low_offset + (rank or heads), channels) > ld:
        raise KernelError("delta_prepare: a column block lies outside the projection")
    dev = proj.device
    q = torch.empty((n, qk_heads * dim), dtype=torch.float32, device=dev)
    k = torch.empty_like(q)
    v = torch.empty((n, heads * vdim), dtype=torch.float32, device=dev)
    g = torch.empty((n, decays), dtype=torch.float32, device=dev)
    beta = torch.empty((n, heads), dtype=torch.float32, device=dev)
    call("b200_delta_prepare", ptr(proj), ld, beta_offset, low_offset, rank, ptr(taps), ntaps, ptr(conv_state), ptr(a_log),
         ptr(dt_bias), ptr(a_up), ptr(q), ptr(k), ptr(v), ptr(g), ptr(beta), ptr(q_start), ptr(slots), ptr(token_entry),
         n, heads, qk_heads, dim, vdim, float(unit_eps), float(q_scale), tag(proj.dtype), stream_ptr())
    return q, k, v, g, beta


def conv_state_update(proj: torch.Tensor, conv_state: torch.Tensor, q_start: torch.Tensor, slots: torch.Tensor) -> None:
    """After a step: every entry's slot keeps the last ``taps - 1`` inputs of its sequence (columns ``0 .. channels-1``
    of ``proj``), oldest first; a step shorter than that keeps the tail of what the slot held."""

    require(proj, "proj", dims=2)
    require(conv_state, "conv_state", dtype=torch.float32, dims=3)
    entries = q_start.shape[0] - 1
    call("b200_conv_state_update", ptr(proj), proj.shape[1], ptr(conv_state), conv_state.shape[2], conv_state.shape[1] + 1,
         ptr(q_start), ptr(slots), entries, tag(proj.dtype), stream_ptr())


def group_norm_gate(x: torch.Tensor, weight: torch.Tensor | None, eps: float, gate_in: torch.Tensor, *, gate_offset: int = 0,
                    gate_up: torch.Tensor | None = None, out_dtype: torch.dtype, group: int | None = None, act: str = "sigmoid",
                    divisor: "tuple[torch.Tensor, torch.Tensor, float] | None" = None) -> torch.Tensor:
    """``x`` float32 ``[N, width]`` in groups of ``group`` columns (default ``len(weight)``): each group divided by its root mean
    square, times ``weight`` (one group's, or ``[width]``; ``None``: no weight, ``group`` is given), times ``sigmoid(logit)`` or ``silu(logit)`` (``act``).  ``divisor =
    (den, floor, e)``: before that, each group divided by ``max(|den|, floor) + e`` with its own numbers (float32 ``[N, width /
    group]`` each).  The logits are columns ``gate_offset ..`` of ``gate_in`` (``width`` of
    them), or, with ``gate_up`` ``[rank, width]`` (a low-rank map's weight transposed),
    ``gate_in[:, gate_offset : gate_offset + rank] @ gate_up``."""

    require(x, "x", dtype=torch.float32, dims=2)
    n, width = x.shape
    if weight is not None:
        require(weight, "weight", dtype=torch.float32, dims=1)
        group = weight.shape[0] if group is None else group
    if not group or group < 0 or width % group or (weight is not None and weight.shape[0] not in (group, width)):
        raise KernelError(f"width {width} is not a multiple of the group size {group}, or the weight has another number of entries")
    if act not in ("sigmoid", "silu"):
        raise KernelError(f"unknown gate {act!r}")
    den = floor = None
    den_eps = 0.0
    if divisor is not None:
        den, floor, den_eps = divisor
        require(den, "divisor", dtype=torch.float32, shape=(n, width // group))
        require(floor, "divisor floor", dtype=torch.float32, shape=(n, width // group))
    require(gate_in, "gate_in", dtype=out_dtype, dims=2)
    rank = 0
    if gate_up is not None:
        require(gate_up, "gate_up", dtype=out_dtype, dims=2)
        rank = gate_up.shape[0]
        if gate_up.shape[1] != width:
            raise KernelError(f"gate_up has {gate_up.shape[1]} columns, expected {width}")
    if gate_offset + (rank or width) > gate_in.shape[1]:
        raise KernelError("group_norm_gate: the gate's columns lie outside gate_in")
    out = torch.empty((n, width), dtype=out_dtype, device=x.device)
    gate_ptr = gate_in.data_ptr() + gate_offset * gate_in.element_size()
    call("b200_group_norm_gate", ptr(x), n, width, group, ptr(weight), weight.shape[0] if weight is not None else 0, float(eps), ptr(den), ptr(floor), float(den_eps),
         gate_ptr, gate_in.shape[1], rank, ptr(gate_up), 1 if act == "silu" else 0, ptr(out), tag(out_dtype), stream_ptr())
    return out
