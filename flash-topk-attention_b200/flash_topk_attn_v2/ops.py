"""Operators of the flash_topk_attn_v2 path on top of the C ABI.

Same names, arguments, checks and exceptions as the reference's operator layer
(flash_topk_attn_v2/block_score.py, topk_select.py, qblock_merge.py,
sparse_attn.py, build_reverse_indices_cuda.py, sort_by_count_cuda.py); the
work itself is done by libftk_sm100.so.  The operators of the hot path
(scoring, merge, attention and its backward) reach it through the native host
layer _native.so, which allocates, launches and holds the autograd node; the
others through ctypes.  PyTorch is used for device memory and streams only.
"""

from __future__ import annotations

import math
import os

import torch

from . import _lib
from ._lib import check, lib, native, ptr, stream_ptr

_SCORE_SCRATCH_BYTES = int(os.environ.get("FTK_SCORE_SCRATCH_BYTES", 4 << 30))
_DEBUG = os.environ.get("FTK_DEBUG", "0") not in ("", "0")
native.set_debug(_DEBUG)


def launch_count() -> int:
    """Kernels of libftk_sm100.so enqueued by this process so far."""
    return lib.ftk_launch_count()


# Optional per-call CUDA-event timing (off by default; bench.py switches it on
# around its timed loop).  Every entry point is bracketed by two events on the
# stream it launches on; `event_times()` returns milliseconds per entry point.
_events = None


def enable_event_timing(on: bool) -> None:
    global _events
    _events = [] if on else None
    native.set_timing(on)


def _call(name, fn, *args):
    """Run one entry point (C ABI: map its return code; native: hand back what it
    returns), timed when asked."""
    if _events is None:
        out = fn(*args)
    else:
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        out = fn(*args)
        e1.record()
        _events.append((name, e0, e1))
    if out.__class__ is int:
        check(out, name)
    return out


def _plain(fn, *args):
    """What a native entry point returns for an ordinary call: one whose arguments it
    finds in order and that wants neither timing nor synchronous checks.  None:
    go through the checks, which raise or handle the special cases."""
    if _events is not None or _DEBUG:
        return None
    try:
        return fn(*args)
    except TypeError:          # an argument that is not of the declared kind
        return None


def event_times() -> dict:
    """Sum of device milliseconds and call count per entry point since
    enable_event_timing(True); synchronises."""
    out = {}
    if _events is not None:
        torch.cuda.synchronize()
        times = [(name, e0.elapsed_time(e1)) for name, e0, e1 in _events] + native.take_times()
        for name, t in times:
            ms, n = out.get(name, (0.0, 0))
            out[name] = (ms + t, n + 1)
    return out


def _device_index(device) -> int:
    index = torch.device(device).index
    return torch.cuda.current_device() if index is None else index


# A device-side failure (a bounded wait that ran out, a block id out of range)
# only sets a sticky status word, one per device, in pinned host memory.  So that
# a caller who never calls check_errors() still hears of it, every operator
# begins by looking at the word: the failure raises at the first call that finds
# it.  FTK_DEBUG=1 checks synchronously after every operator instead.
def status_word(device) -> torch.Tensor:
    """Sticky per-device status word handed to every launch (pinned host memory)."""
    return native.status_word(_device_index(device))


def check_errors(device=None) -> None:
    """Synchronise the current stream and raise if any launch since the last
    check reported a device-side failure."""
    if device is None or torch.device(device).index is None:
        indices = range(torch.cuda.device_count()) if device is None else [_device_index(device)]
    else:
        indices = [torch.device(device).index]
    for index in indices:
        torch.cuda.current_stream(index).synchronize()
        code = native.take_status(index)
        if code != 0:
            raise RuntimeError(
                f"flash_topk_attn_v2 device error: {_lib.error_text(code)} (status {code})"
            )


def deferred_checks(on: bool) -> None:
    """Switch the operators' look at the status word on or off (on by default).
    Off, a device-side failure is only reported by check_errors()."""
    native.set_deferred(bool(on))


def _before(device) -> None:
    native.look(_device_index(device))


def _after(device) -> None:
    if _DEBUG and not torch.cuda.is_current_stream_capturing():   # a capture cannot synchronise
        check_errors(device)


def _next_pow2(x: int) -> int:
    return 1 if x <= 1 else 1 << (x - 1).bit_length()


# --------------------------------------------------------------------------
# layout helpers
# --------------------------------------------------------------------------
def _kernel_head_dim(d: int) -> int:
    if d <= 64:
        return 64
    if d <= 128:
        return 128
    if d <= 256:      # 160 and 256 of the reference's list (block_score_cuda.py:16) share one kernel
        return 256
    raise NotImplementedError(f"head dim {d} > 256 is not supported")


def _as_bnhd(x: torch.Tensor, input_4d: bool, H: int, D: int):
    """Return (tensor, sb, sn, sh) addressing x as [b][n][h][d] with d-stride 1,
    16-byte aligned base, strides that are multiples of 8 elements and no
    repeated (expanded) dimension.  Copies only when the layout cannot be
    addressed in place."""
    if any(n > 1 and s <= 0 for n, s in zip(x.shape[:-1], x.stride())):
        x = x.contiguous()
    if input_4d:                       # [B, H, N, D]
        if x.stride(3) != 1:
            x = x.contiguous()
        sb, sh, sn = x.stride(0), x.stride(1), x.stride(2)
    else:                              # [B, N, H*D]
        if x.stride(2) != 1:
            x = x.contiguous()
        sb, sn, sh = x.stride(0), x.stride(1), D
    if x.data_ptr() % 16 or sb % 8 or sn % 8 or sh % 8:
        x = x.contiguous()
        if input_4d:
            sb, sh, sn = x.stride(0), x.stride(1), x.stride(2)
        else:
            sb, sn, sh = x.stride(0), x.stride(1), D
        if x.data_ptr() % 16 or sb % 8 or sn % 8 or sh % 8:
            raise ValueError("tensor cannot be aligned to 16 bytes (head dim must be a multiple of 8)")
    return x, sb, sn, sh


def _pad_head_dim(x: torch.Tensor, input_4d: bool, H: int, D: int, Dk: int) -> torch.Tensor:
    """Zero-pad the head dim to the kernel's, as the reference does
    (block_score_cuda.py:130-132, sparse_attn.py:358-373)."""
    if Dk == D:
        return x
    if input_4d:
        return torch.nn.functional.pad(x, (0, Dk - D))
    B, N, _ = x.shape
    return torch.nn.functional.pad(x.reshape(B, N, H, D), (0, Dk - D)).reshape(B, N, H * Dk)


def _check_device(what: str, x: torch.Tensor, device: torch.device) -> None:
    """Kernels take raw pointers: a tensor that lives elsewhere must not get that far."""
    if x.device != device:
        raise ValueError(f"{what} must be on {device}, got {x.device}")


# --------------------------------------------------------------------------
# scoring
# --------------------------------------------------------------------------
def _parse_block_score_args(q, k, num_heads, score_block_size, padding):
    """Argument checks of the reference (block_score.py:369-414)."""
    if q.device.type != "cuda":
        raise ValueError("flash_block_score requires CUDA tensors")
    input_4d = q.ndim == 4
    if input_4d:
        B, H, N, D = q.shape
        if num_heads != H:
            raise ValueError(f"num_heads ({num_heads}) != q.shape[1] ({H})")
        C = H * D
    else:
        if q.ndim != 3:
            raise ValueError("q must be 3D [B, N, C] or 4D [B, H, N, D]")
        B, N, C = q.shape
    H = num_heads
    D = C // H
    pad_head, pad_tail = padding
    if pad_head < 0 or pad_tail < 0:
        raise ValueError("padding must be non-negative (pad_head, pad_tail)")
    if pad_head >= score_block_size or pad_tail >= score_block_size:
        raise ValueError(
            f"padding ({pad_head}, {pad_tail}) must each be < score_block_size "
            f"({score_block_size})"
        )
    n_padded = pad_head + N + pad_tail
    if n_padded % score_block_size != 0:
        need = score_block_size - (n_padded % score_block_size)
        raise ValueError(
            f"pad_head + N + pad_tail = {n_padded} must be divisible by "
            f"score_block_size ({score_block_size}). Try padding=(0, {pad_tail + need})."
        )
    if input_4d:
        if k.shape != (B, H, N, D):
            raise ValueError(f"k shape {k.shape} != {(B, H, N, D)}")
    else:
        if k.shape != (B, N, C):
            raise ValueError(f"k shape {k.shape} != {(B, N, C)}")
    if C % H != 0:
        raise ValueError(f"C={C} not divisible by num_heads={H}")
    if q.dtype != k.dtype:
        raise ValueError(f"q.dtype ({q.dtype}) != k.dtype ({k.dtype})")
    if q.dtype not in (torch.float16, torch.bfloat16, torch.float32):
        raise ValueError("q must be float16, bfloat16, or float32")
    _check_device("k", k, q.device)
    return input_4d, B, H, N, D, n_padded // score_block_size, pad_head, pad_tail


def _prep_qk(q, k, input_4d, H, D):
    if q.dtype == torch.float32:       # block_score_cuda.py:115-118
        q, k = q.bfloat16(), k.bfloat16()
    Dk = _kernel_head_dim(D)
    q = _pad_head_dim(q, input_4d, H, D, Dk)
    k = _pad_head_dim(k, input_4d, H, D, Dk)
    q, *sq = _as_bnhd(q, input_4d, H, Dk)
    k, *sk = _as_bnhd(k, input_4d, H, Dk)
    return q, sq, k, sk, Dk


def flash_block_score(q, k, num_heads, score_block_size, padding=(0, 0)):
    """Softmax mass per (query, score block): [B, H, N, M] float32.

    Mirrors flash_block_score (flash_topk_attn_v2/block_score.py:417-452)."""
    input_4d, B, H, N, D, M, ph, pt = _parse_block_score_args(
        q, k, num_heads, score_block_size, padding)
    _before(q.device)
    qq, sq, kk, sk, Dk = _prep_qk(q, k, input_4d, H, D)
    out = torch.empty(B, H, N, M, dtype=torch.float32, device=q.device)
    status = status_word(q.device)
    # slices are independent; chunk so that launches stay below the grid limit
    step = min(B * H, 32768)
    ws = torch.empty(lib.ftk_block_score_workspace(step, N), dtype=torch.uint8, device=q.device)
    flat = out.view(B * H, N, M)
    for b0 in range(0, B * H, step):
        cnt = min(step, B * H - b0)
        _call("ftk_block_score", lib.ftk_block_score, 
            ptr(qq), ptr(kk), _lib.dtype_code(qq), B, H, N, Dk, *sq, *sk, b0, cnt,
            score_block_size, ph, pt, float(D) ** -0.5, ptr(flat[b0]), ptr(ws), ws.numel(),
            ptr(status), stream_ptr(q.device))
    _after(q.device)
    return out


def flash_topk_select(block_scores, threshold, max_topk, score_block_size, padding=(0, 0),
                      backend="auto"):
    """Top-k blocks per query with cumulative-threshold cut.

    Mirrors flash_topk_select (flash_topk_attn_v2/topk_select.py:185-311); the
    `backend` argument is accepted for compatibility and ignored (one native
    path, ties keep the lower block id)."""
    if block_scores.ndim != 4:
        raise ValueError("block_scores must be [B, H, N, M]")
    if block_scores.device.type != "cuda":
        raise ValueError("flash_topk_select requires CUDA tensor")
    if block_scores.dtype not in (torch.float16, torch.bfloat16, torch.float32):
        raise ValueError("block_scores must be float16/bfloat16/float32")
    B, H, N, M = block_scores.shape
    if M <= 0:
        raise ValueError("M must be positive")
    if score_block_size <= 0:
        raise ValueError("score_block_size must be positive")
    pad_head, pad_tail = padding
    if pad_head < 0 or pad_tail < 0:
        raise ValueError("padding must be non-negative (pad_head, pad_tail)")
    if pad_head >= score_block_size or pad_tail >= score_block_size:
        raise ValueError(
            f"padding ({pad_head}, {pad_tail}) must each be < score_block_size "
            f"({score_block_size})"
        )
    if max_topk < 0:
        raise ValueError("max_topk must be >= 0")
    if backend not in ("auto", "triton", "cuda"):
        raise ValueError(f"backend must be 'auto', 'triton', or 'cuda', got '{backend}'")
    if M > 4096:
        raise NotImplementedError(f"select requires M <= 4096, got M={M}")
    m_out = min(max_topk, M) if max_topk > 0 else M
    scores = block_scores.float().contiguous()
    dev = scores.device
    _before(dev)
    idx = torch.empty(B, H, N, m_out, dtype=torch.int32, device=dev)
    raw = torch.empty(B, H, N, m_out, dtype=torch.float32, device=dev)
    avg = torch.empty(B, H, N, m_out, dtype=torch.float32, device=dev)
    _call("ftk_topk_select", lib.ftk_topk_select, 
        ptr(scores), 0, B * H * N, M, max_topk, score_block_size, pad_head, pad_tail,
        float(threshold), ptr(idx), ptr(raw), ptr(avg), ptr(status_word(dev)), stream_ptr(dev))
    _after(dev)
    return idx, raw, avg


def flash_topk_score_fused(q, k, num_heads, score_block_size, topk, padding, threshold):
    """block score + select without materialising [B,H,N,M] for the caller."""
    plain = _plain(native.plain_score, q, k, num_heads, score_block_size, topk, padding, threshold,
                   _SCORE_SCRATCH_BYTES)
    if plain is not None:
        idx, raw, avg, M = plain
        idx._ftk_num_score_blocks = M
        return idx, raw, avg
    input_4d, B, H, N, D, M, ph, pt = _parse_block_score_args(
        q, k, num_heads, score_block_size, padding)
    if topk < 0:
        raise ValueError("max_topk must be >= 0")
    if M > 4096:
        raise NotImplementedError(f"select requires M <= 4096, got M={M}")
    if D % 8 or D > 256:   # head dims that a tensor map cannot read in place
        Dk = _kernel_head_dim(D)
        q = _pad_head_dim(q, input_4d, H, D, Dk)
        k = _pad_head_dim(k, input_4d, H, D, Dk)
    slices = B * H
    step = min(slices, 32768,
               max(1, _SCORE_SCRATCH_BYTES // native.score_topk_workspace(1, N, M)))
    if step < slices and q.dtype == torch.float32:
        q, k = q.bfloat16(), k.bfloat16()
    outs = []
    for b0 in range(0, slices, step):
        outs = _call("ftk_score_topk", native.score_topk, q, k, input_4d, H, score_block_size, topk,
                     ph, pt, threshold, float(D) ** -0.5, b0, min(step, slices - b0), outs)
    if _DEBUG:
        _after(q.device)
    idx, raw, avg = outs
    # lets build_qblock_topk_indices size its table without a device round trip
    idx._ftk_num_score_blocks = M
    return idx, raw, avg


# --------------------------------------------------------------------------
# merge
# --------------------------------------------------------------------------
def num_score_blocks_of(topk_indices) -> int:
    """max(valid id) + 1 (at least 1) of an index tensor: one device reduction
    (ftk_max_index_plus1) and one four-byte read-back, where the reference
    masks, gathers and reduces with PyTorch (__init__.py:101-105)."""
    idx = topk_indices.to(torch.int32).contiguous()
    dev = idx.device
    out = torch.empty(1, dtype=torch.int32, device=dev)
    _call("ftk_max_index_plus1", lib.ftk_max_index_plus1, ptr(idx), idx.numel(), ptr(out),
          stream_ptr(dev))
    return int(out.item())


def flash_qblock_merge(topk_indices, topk_scores, q_block_size, qblock_topk, num_score_blocks,
                       q_padding=(0, 0), return_counts=False, want_scores=True):
    """Per-q-block aggregation + ranking of (block, score) pairs.

    Mirrors flash_qblock_merge (flash_topk_attn_v2/qblock_merge.py:85-156).
    `q_padding` is an extension: the reference pads the index tensor on the
    host first (__init__.py:90-96); here the kernel skips the virtual rows.
    `want_scores=False` leaves the aggregated scores out (None in their place)."""
    if topk_indices.ndim != 4:
        raise ValueError("topk_indices must be [B, H, N, M_out]")
    if topk_scores is not None and topk_scores.ndim != 4:
        raise ValueError("topk_scores must be [B, H, N, M_out]")
    if topk_indices.device.type != "cuda":
        raise ValueError("flash_qblock_merge requires CUDA tensors")
    N = topk_indices.shape[2]
    qh, qt = q_padding
    if (qh + N + qt) % q_block_size != 0:
        raise ValueError(f"N ({qh + N + qt}) must be divisible by q_block_size ({q_block_size})")
    if num_score_blocks <= 0:
        raise ValueError("num_score_blocks must be positive")
    if num_score_blocks > 4096:
        raise NotImplementedError(
            f"num_score_blocks={num_score_blocks} exceeds CUDA block sort limit 4096")
    if qblock_topk <= 0:
        raise ValueError("qblock_topk must be positive")
    if topk_scores is not None:
        if topk_scores.shape != topk_indices.shape:
            raise ValueError(f"topk_scores {tuple(topk_scores.shape)} must have the shape of "
                             f"topk_indices {tuple(topk_indices.shape)}")
        _check_device("topk_scores", topk_scores, topk_indices.device)
    merged, mscores, counts = _call(
        "ftk_qblock_merge", native.qblock_merge, topk_indices, topk_scores, q_block_size, qh, qt,
        num_score_blocks, qblock_topk, want_scores)
    if _DEBUG:
        _after(merged.device)
    if return_counts:
        return merged, mscores, counts
    return merged, mscores


def flash_qblock_union(topk_indices, q_block_size, q_padding=(0, 0), num_score_blocks=None,
                       width=None):
    """Distinct block ids picked inside each q-block, ascending, -1 padded:
    (merged [B, H, QM, width] int32, counts [B, H, QM] int32).

    The exact-union merge of the first-generation operators
    (flash_topk_attn/attention.py:70-138).  `width` defaults to the
    reference's next_pow2(q_block_size * K); `num_score_blocks` bounds the ids
    (default: read back from the indices, one host round trip)."""
    if topk_indices.ndim != 4:
        raise ValueError("topk_indices must be [B, H, N, K]")
    if topk_indices.device.type != "cuda":
        raise ValueError("flash_qblock_union requires CUDA tensors")
    B, H, N, K = topk_indices.shape
    qh, qt = q_padding
    QM = (qh + N + qt) // q_block_size
    dev = topk_indices.device
    _before(dev)
    idx = topk_indices.to(torch.int32).contiguous()
    if num_score_blocks is None:
        num_score_blocks = max(int(idx.max().item()) + 1, 1)
    if num_score_blocks > 65536:
        raise NotImplementedError(f"num_score_blocks={num_score_blocks} exceeds 65536")
    if width is None:
        width = _next_pow2(q_block_size * K)
    merged = torch.empty(B, H, QM, width, dtype=torch.int32, device=dev)
    counts = torch.empty(B, H, QM, dtype=torch.int32, device=dev)
    _call("ftk_qblock_union", lib.ftk_qblock_union,
          ptr(idx), B * H, N, K, q_block_size, qh, qt, num_score_blocks, width, ptr(merged),
          ptr(counts), ptr(status_word(dev)), stream_ptr(dev))
    _after(dev)
    return merged, counts


# --------------------------------------------------------------------------
# reverse index / count sort
# --------------------------------------------------------------------------
def flash_build_reverse_indices_cuda(merged_indices, counts, num_kv_blocks):
    """(reverse_indices [B,H,M,QM], reverse_counts [B,H,M], sorted_kv [B,H,M]).

    Mirrors flash_build_reverse_indices_cuda
    (flash_topk_attn_v2/build_reverse_indices_cuda.py:32-78)."""
    B, H, QM, W = merged_indices.shape
    M = num_kv_blocks
    dev = merged_indices.device
    if counts is not None:
        if counts.numel() != B * H * QM:
            raise ValueError(f"counts must be [B, H, QM] = {(B, H, QM)}, got {tuple(counts.shape)}")
        _check_device("counts", counts, dev)
    _before(dev)
    merged = merged_indices.contiguous()
    cnt = None if counts is None else counts.to(torch.int32).contiguous()
    rev = torch.empty(B, H, M, QM, dtype=torch.int32, device=dev)
    rc = torch.empty(B, H, M, dtype=torch.int32, device=dev)
    skv = torch.empty(B, H, M, dtype=torch.int32, device=dev)
    ws = torch.empty(lib.ftk_build_reverse_workspace(B * H, QM, M), dtype=torch.uint8, device=dev)
    _call("ftk_build_reverse", lib.ftk_build_reverse, 
        ptr(merged), ptr(cnt), B * H, QM, W, M, ptr(rev), ptr(rc), ptr(skv), ptr(ws), ws.numel(),
        ptr(status_word(dev)), stream_ptr(dev))
    _after(dev)
    return rev, rc, skv


def flash_sort_by_count_cuda(reverse_counts, num_heads, num_kv_blocks):
    """Global descending sort of the reverse counts with flat ids.

    Mirrors flash_sort_by_count_cuda (flash_topk_attn_v2/sort_by_count_cuda.py:33-67),
    including its host read of the maximum count."""
    flat = reverse_counts.reshape(-1).to(torch.int32).contiguous()
    total = flat.numel()
    dev = flat.device
    max_val = int(flat.max().item()) if total else 0
    sc = torch.empty_like(flat)
    ids = torch.empty(total, dtype=torch.int32, device=dev)
    ws = torch.empty(lib.ftk_sort_by_count_workspace(total, max_val), dtype=torch.uint8, device=dev)
    _call("ftk_sort_by_count", lib.ftk_sort_by_count, ptr(flat), total, max_val, ptr(sc), ptr(ids), ptr(ws), ws.numel(),
                                stream_ptr(dev))
    return sc, ids


# --------------------------------------------------------------------------
# sparse attention
# --------------------------------------------------------------------------
def _check_backward_blocks(D, g, kvb):
    """Block sizes the gradient kernels take (the reference's take any q block of
    1..64 rows and any kv block): multiples of 16 rows, and at head dims above 128
    sizes that halve down to 16 or 32 rows."""
    if g % 16 != 0:
        raise NotImplementedError(
            f"the backward needs a q_block_size that is a multiple of 16, got {g}")
    if D > 128:
        for name, blk in (("q_block_size", g), ("kv_block_size", kvb)):
            part = blk
            while part > 32 and part % 2 == 0:
                part //= 2
            if part > 32 or part % 16 != 0:
                raise NotImplementedError(
                    f"backward at head dim > 128 needs a {name} that halves down to 16 or "
                    f"32 rows (16, 32, 64, 128), got {blk}")


def flash_sparse_attn(q, k, v, merged_indices, num_heads, q_block_size, kv_block_size,
                      scale=None, q_padding=(0, 0), kv_padding=(0, 0), num_kv_heads=None):
    """Block-sparse attention, differentiable in q, k, v: (O [B,N,C], lse [B,H,N]).

    Mirrors flash_sparse_attn (flash_topk_attn_v2/sparse_attn.py:227-392)
    including its argument checks, with one extension: q and kv blocks of up to
    128 rows (multiples of 32 above 64) are accepted for forward and backward;
    the reference rejects q blocks above 64 (sparse_attn.py:279) and its
    dK/dV kernel is only correct up to 64-row kv blocks.  `num_kv_heads`
    (grouped-query attention, also beyond the reference): k and v are
    [B, N, num_kv_heads * D] and query head h reads kv head
    h // (num_heads // num_kv_heads)."""
    plain = _plain(native.plain_attn, q, k, v, merged_indices, num_heads, q_block_size,
                   kv_block_size, scale, q_padding, kv_padding, num_kv_heads)
    if plain is not None:
        return plain
    if q.ndim != 3:
        raise ValueError("q must be [B, N, C]")
    if q.device.type != "cuda":
        raise ValueError("flash_sparse_attn requires CUDA tensors")
    if q.dtype not in (torch.float16, torch.bfloat16, torch.float32):
        raise ValueError("q must be float16, bfloat16, or float32")
    mixed = q.dtype == torch.float32 and not (k.dtype == v.dtype == torch.float32)
    if mixed:
        q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    B, N, C = q.shape
    H = num_heads
    D = C // H
    if C != H * D:
        raise ValueError(f"C ({C}) must be divisible by num_heads ({H})")
    Hkv = H if num_kv_heads is None else int(num_kv_heads)
    if Hkv <= 0 or H % Hkv != 0:
        raise ValueError(f"num_heads ({H}) must be a multiple of num_kv_heads ({Hkv})")
    if k.shape != (B, N, Hkv * D) or v.shape != (B, N, Hkv * D):
        raise ValueError(f"k and v must be [B, N, num_kv_heads * D] = {(B, N, Hkv * D)}")
    if q_block_size <= 0 or q_block_size > 128:
        raise ValueError(f"q_block_size must be in (0, 128], got {q_block_size}")
    if kv_block_size <= 0:
        raise ValueError(f"kv_block_size must be positive, got {kv_block_size}")
    if kv_block_size > 128:
        raise NotImplementedError(f"kv_block_size must be <= 128, got {kv_block_size}")
    for name, blk in (("q_block_size", q_block_size), ("kv_block_size", kv_block_size)):
        if blk > 64 and blk % 32 != 0:
            raise NotImplementedError(f"{name} above 64 must be a multiple of 32, got {blk}")
    if merged_indices.ndim != 4:
        raise ValueError("merged_indices must be [B, H, QM, qblock_topk]")
    if merged_indices.dtype != torch.int32:
        raise ValueError("merged_indices must be int32")
    q_pad_head, q_pad_tail = q_padding
    kv_pad_head, kv_pad_tail = kv_padding
    if q_pad_head < 0 or q_pad_tail < 0:
        raise ValueError("q_padding values must be non-negative")
    if kv_pad_head < 0 or kv_pad_tail < 0:
        raise ValueError("kv_padding values must be non-negative")
    if q_pad_head >= q_block_size:
        raise ValueError(f"q_pad_head={q_pad_head} must be < q_block_size={q_block_size}")
    if q_pad_tail >= q_block_size:
        raise ValueError(f"q_pad_tail={q_pad_tail} must be < q_block_size={q_block_size}")
    if kv_pad_head >= kv_block_size:
        raise ValueError(f"kv_pad_head={kv_pad_head} must be < kv_block_size={kv_block_size}")
    if kv_pad_tail >= kv_block_size:
        raise ValueError(f"kv_pad_tail={kv_pad_tail} must be < kv_block_size={kv_block_size}")
    n_q = q_pad_head + N + q_pad_tail
    n_kv = kv_pad_head + N + kv_pad_tail
    if n_q % q_block_size != 0:
        raise ValueError(
            f"q_pad_head + N + q_pad_tail = {n_q} must be divisible by q_block_size={q_block_size}")
    if n_kv % kv_block_size != 0:
        raise ValueError(
            f"kv_pad_head + N + kv_pad_tail = {n_kv} must be divisible by "
            f"kv_block_size={kv_block_size}")
    QM = n_q // q_block_size
    if merged_indices.shape[2] != QM:
        raise ValueError(
            f"merged_indices dim 2 ({merged_indices.shape[2]}) must match "
            f"QM = (q_pad_head + N + q_pad_tail) // q_block_size = {QM}")
    if merged_indices.shape[:2] != (B, H):
        raise ValueError(
            f"merged_indices {tuple(merged_indices.shape)} must begin with [B, H] = {(B, H)}")
    if D <= 0 or D % 16 != 0:
        raise ValueError(f"D ({D}) must be a positive multiple of 16")
    if D > 256:
        raise ValueError(f"D ({D}) must be <= 256")
    if not (k.dtype == v.dtype == q.dtype):
        raise ValueError(f"k ({k.dtype}) and v ({v.dtype}) must have the type of q ({q.dtype})")
    for name, x in (("k", k), ("v", v), ("merged_indices", merged_indices)):
        _check_device(name, x, q.device)
    if scale is None:
        scale = 1.0 / math.sqrt(D)
    if torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad):
        # say so now rather than inside backward()
        _check_backward_blocks(D, q_block_size, kv_block_size)
    o, lse = native.sparse_attn(q, k, v, merged_indices, H, Hkv, q_block_size, kv_block_size,
                                q_pad_head, kv_pad_head, scale)
    if _DEBUG:
        _after(o.device)
    return (o.float() if mixed else o), lse
