"""Low-level Python entry points of the sm_100a attention kernels (one ring step each).

``flash_fwd`` runs ``attn_fwd_sm100.cu``: local queries against one KV block with optional carry-in
``(o_prev, lse_prev)``, masks driven by global positions, and an optional in-kernel copy job that
pulls the *next* ring step's KV block from a peer GPU. ``flash_bwd`` runs ``attn_bwd_sm100.cu``.
Both take ``(B, S, H, D)`` bf16 views with a contiguous last dim (``D`` in {64, 128}).
"""
from __future__ import annotations

import math
import struct
from dataclasses import dataclass
from typing import Optional

import torch

from . import _lib


@dataclass
class Positions:
    """Global positions of a shard: one run ``[off0, off0+n)`` or two runs of ``half`` tokens."""

    off0: int
    off1: int = 0
    half: int = 1 << 30

    @classmethod
    def from_segments(cls, segs) -> "Positions":
        if len(segs) == 1:
            return cls(segs[0][1], 0, 1 << 30)
        (_, g0, n0), (l1, g1, _) = segs
        assert l1 == n0
        return cls(g0, g1, n0)

    def tensor(self, n: int, device) -> torch.Tensor:
        i = torch.arange(n, device=device)
        return torch.where(i < self.half, self.off0 + i, self.off1 + (i - self.half))


@dataclass
class MaskSpec:
    """Everything the kernels need to know about masking for one (q shard, kv block) pair."""

    causal_block_size: int = 0            # 0 = not causal
    q_pos: Positions = None               # type: ignore[assignment]
    k_pos: Positions = None               # type: ignore[assignment]
    seg_q: Optional[torch.Tensor] = None  # (B, Sq) int32, ids of the local queries
    seg_k: Optional[torch.Tensor] = None  # (B, Sk) int32, ids of this KV block
    seg_q_mm: Optional[torch.Tensor] = None
    seg_k_mm: Optional[torch.Tensor] = None
    bias: Optional[torch.Tensor] = None   # (B, 1|H, Sk) fp32 key bias for this KV block
    seed: int = 0
    pdrop: float = 0.0
    keep_q: Optional[torch.Tensor] = None  # (B, 1|H, Sq, 4*ceil(Sk/128)) int32 bitmap by query row (forward)
    keep_k: Optional[torch.Tensor] = None  # (B, 1|H, Sk, 4*ceil(Sq/128)) int32 bitmap by kv row (backward)
    keep_tiles: Optional[torch.Tensor] = None  # (B, 1|H, ceil(Sq/128), ceil(Sk/128)) uint8 of the bitmap's tiles: 0 empty, 1 full, 2 mixed


def seg_tile_minmax(seg: torch.Tensor) -> torch.Tensor:
    """Per-128-token-tile ``{min, max}`` of segment ids: ``(B, ceil(S/128), 2)`` int32."""
    B, S = seg.shape
    nt = (S + 127) // 128
    pad = nt * 128 - S
    if pad:
        seg = torch.cat([seg, seg[:, -1:].expand(B, pad)], dim=1)
    t = seg.view(B, nt, 128)
    return torch.stack([t.amin(dim=2), t.amax(dim=2)], dim=2).to(torch.int32).contiguous()


def _check_runs(pos: Positions, n: int, total: int) -> None:
    runs = [(pos.off0, min(n, pos.half))] + ([(pos.off1, n - pos.half)] if n > pos.half else [])
    if any(off < 0 or off + m > total for off, m in runs):
        raise IndexError(f"positions {runs} reach past the {total} given ones")


def take_positions(x: torch.Tensor, dim: int, pos: Positions, n: int) -> torch.Tensor:
    """The ``n`` positions of a shard along ``dim`` of a global tensor, as a contiguous copy."""
    _check_runs(pos, n, x.shape[dim])
    if n <= pos.half:
        return x.narrow(dim, pos.off0, n).clone(memory_format=torch.contiguous_format)
    return torch.cat([x.narrow(dim, pos.off0, pos.half), x.narrow(dim, pos.off1, n - pos.half)], dim=dim).contiguous()


def segment_shard(seg: torch.Tensor, pos: Positions, n: int):
    """``(ids, minmax)`` of a shard's ``n`` positions out of the global int32 ids ``(B, S_total)``: a contiguous copy and
    what :func:`seg_tile_minmax` gives for it, in one launch (any device but CUDA, and batches past a grid's limit: PyTorch)."""
    B = seg.shape[0]
    if not seg.is_cuda or B > 65535:
        ids = take_positions(seg, 1, pos, n)
        return ids, seg_tile_minmax(ids)
    _check_runs(pos, n, seg.shape[1])
    if seg.stride(1) != 1:
        seg = seg.contiguous()
    ids = torch.empty(B, n, device=seg.device, dtype=torch.int32)
    mm = torch.empty(B, (n + 127) // 128, 2, device=seg.device, dtype=torch.int32)
    _lib.call("ra_segment_tiles", seg.data_ptr(), seg.stride(0), pos.off0, pos.off1, min(pos.half, 1 << 30), B, n,
              ids.data_ptr(), mm.data_ptr(), _lib.stream_handle())
    return ids, mm


# ``RaAttnFwdArgs`` (attn_fwd_sm100.cu), packed as the C compiler lays it out: q k v, their strides, out and its strides, out_fp32, lse_out,
# o_prev lse_prev, B H Sq Sk D, softmax_scale, the mask's fields (:func:`_mask_fields`), the copy job, status, stream, splits, ws. (A
# ctypes structure of these fields takes 11 us to fill, this 3.)
_FWD_ARGS = struct.Struct("@3P9q P3qi P 2P 5i f 7i4P P2q QI P3q P2q 2Pqi 2P iP")


def tma_ready(t: torch.Tensor) -> bool:
    """Whether the kernels take a ``(B, S, H, D)`` view as it is: contiguous ``D``, strides and base of whole 16 bytes."""
    sb, ss, sh, sd = t.stride()
    return sd == 1 and not (sb | ss | sh) & 7 and not t.data_ptr() & 15


def _check_bshd(t: torch.Tensor, name: str) -> None:
    if t.dim() != 4 or t.dtype != torch.bfloat16 or not t.is_cuda or t.stride(3) != 1:
        raise ValueError(f"{name} must be a CUDA bf16 (B, S, H, D) view with contiguous D")
    if not tma_ready(t):
        raise ValueError(f"{name}: strides must be multiples of 8 elements and base 16-byte aligned")


def _ptr(t):
    return 0 if t is None else t.data_ptr()


def mask_bitmaps(mask: torch.Tensor, want_q: bool = True, want_k: bool = True):
    """Pack a boolean ``(B, 1|H, 1|Sq, Sk)`` mask (True = attend) into what the kernels read: the bitmaps by query row
    for the forward and by kv row for the backward (``MaskSpec.keep_q`` / ``keep_k``), and the kind of every tile
    (``keep_tiles``). A mask without query rows (a key-padding mask) must be expanded by the caller to the query length first."""
    assert mask.dim() == 4 and mask.is_cuda
    m = mask.view(torch.uint8) if mask.dtype == torch.bool else mask.to(torch.uint8)  # a bool is a byte of 0 or 1
    if m.stride(3) != 1:
        m = m.contiguous()
    B, Hm, Sq, Sk = m.shape
    nq, nk = (Sq + 127) // 128, (Sk + 127) // 128
    by_q = torch.empty(B, Hm, Sq, 4 * nk, device=m.device, dtype=torch.int32) if want_q else None
    by_k = torch.empty(B, Hm, Sk, 4 * nq, device=m.device, dtype=torch.int32) if want_k else None
    tiles = torch.empty(B, Hm, nq, nk, device=m.device, dtype=torch.uint8)
    _lib.call("ra_pack_mask", m.data_ptr(), m.stride(0), m.stride(1), m.stride(2), _ptr(by_q), _ptr(by_k), tiles.data_ptr(),
              B, Hm, Sq, Sk, _lib.stream_handle())
    return by_q, by_k, tiles


def pack_mask(mask: torch.Tensor, want_q: bool = True, want_k: bool = True):
    """The two bitmaps of :func:`mask_bitmaps`."""
    return mask_bitmaps(mask, want_q, want_k)[:2]


def _mask_fields(mask: MaskSpec, H: int, by_k: bool = False) -> tuple:
    """The mask's fields of the launch arguments, in their order from ``causal_block_size`` to ``keep_tiles_sh``."""
    keep = mask.keep_k if by_k else mask.keep_q
    if (mask.keep_q is not None or mask.keep_k is not None) and keep is None:
        raise ValueError("the mask bitmap for this pass is missing (pack_mask builds both)")
    kp = (0, 0, 0, 0, 0, 0, 0)
    if keep is not None:
        assert keep.dtype == torch.int32 and keep.dim() == 4 and keep.is_contiguous()
        per_head = keep.shape[1] == H
        kp = (keep.data_ptr(), keep.stride(0), keep.stride(1) if per_head else 0, keep.stride(2), 0, 0, 0)
        tiles = mask.keep_tiles
        if tiles is not None:
            assert tiles.dtype == torch.uint8 and tiles.is_contiguous() and tiles.shape[:2] == keep.shape[:2]
            kp = kp[:4] + (tiles.data_ptr(), tiles.stride(0), tiles.stride(1) if per_head else 0)
    bias = (0, 0, 0)
    if mask.bias is not None:
        bm = mask.bias
        assert bm.dtype == torch.float32 and bm.dim() == 3 and bm.stride(2) == 1
        bias = (bm.data_ptr(), bm.stride(0), bm.stride(1) if bm.shape[1] == H else 0)
    drop = max(1, min(int(mask.pdrop * 4294967296.0), 0xFFFFFFFF)) if mask.pdrop > 0.0 else 0
    qp, kv = mask.q_pos, mask.k_pos
    return (int(mask.causal_block_size or 0), qp.off0, qp.off1, qp.half, kv.off0, kv.off1, kv.half,
            _ptr(mask.seg_q), _ptr(mask.seg_k), _ptr(mask.seg_q_mm), _ptr(mask.seg_k_mm), *bias,
            int(mask.seed) & (2**64 - 1), drop, *kp)


def flash_fwd(q, k, v, mask: MaskSpec, *, o_prev=None, lse_prev=None, out_fp32=False,
              out=None, lse_out=None, copy_src: int = 0, copy_dst: int = 0, copy_bytes: int = 0,
              copy_ctas: int = 8):
    """One ring step of the forward. Returns ``(out, lse)``; ``out`` is ``(B,Sq,H,D)`` fp32 or
    bf16, ``lse`` is ``(B,H,Sq)`` fp32 (natural log). ``o_prev`` must be fp32 contiguous."""
    _check_bshd(q, "q"); _check_bshd(k, "k"); _check_bshd(v, "v")
    B, Sq, H, D = q.shape
    Sk = k.shape[1]
    dev = q.device
    if out is None:
        out = torch.empty(B, Sq, H, D, device=dev, dtype=torch.float32 if out_fp32 else torch.bfloat16)
    if lse_out is None:
        lse_out = torch.empty(B, H, Sq, device=dev, dtype=torch.float32)
    if o_prev is not None:
        assert o_prev.dtype == torch.float32 and o_prev.is_contiguous() and lse_prev is not None
    fields = (q.data_ptr(), k.data_ptr(), v.data_ptr(), *q.stride()[:3], *k.stride()[:3], *v.stride()[:3],
              out.data_ptr(), *out.stride()[:3], int(out.dtype == torch.float32), lse_out.data_ptr(),
              _ptr(o_prev), _ptr(lse_prev), B, H, Sq, Sk, D, 1.0 / math.sqrt(D), *_mask_fields(mask, H),
              copy_src, copy_dst, copy_bytes, copy_ctas, _lib.status_tensor(dev).data_ptr(), _lib.stream_handle())
    args = _FWD_ARGS.pack(*fields, 0, 0)
    splits = _lib.lib().ra_attn_fwd_splits(args)
    if splits > 1:  # few query tiles: the keys are split over several CTAs, partial results meet in a second launch
        ws = torch.empty(splits * B * Sq * H * (D + 1), device=dev, dtype=torch.float32)
        args = _FWD_ARGS.pack(*fields, splits, ws.data_ptr())
    _lib.call("ra_attn_fwd", args, n_kernels=2 if splits > 1 else 1)
    return out, lse_out


# ``RaAttnBwdArgs`` (attn_api.h): q k v dO, their strides, lse2 delta Sq_pad, dq_acc, dk dv and their strides and mode, B H Sq Sk D,
# softmax_scale, the mask's fields, the copy job, status, stream, trace
_BWD_FORMAT = "@4P12q 2Pi P 2P3qi 5i f 7i4P P2q QI P3q P2q 2Pqi 3P"
_BWD_ARGS = struct.Struct(_BWD_FORMAT)
# ``RaAttnBwdRun`` (backward_runs.cu): the same, then out and its strides, lse, dq and the distance of its rows
_BWD_RUN_ARGS = struct.Struct(_BWD_FORMAT + "P3q 2Pq")


# Phase-timestamp buffers by device index: a backward launch on that device records into its buffer
# (utils.tracing.BackwardPhaseTrace installs and removes them); launches on other devices are not traced.
BWD_TRACE_BUFFERS: dict = {}

DKV_STORE_BF16 = 0
DKV_STORE_FP32 = 1
DKV_REDUCE_FP32 = 2


def flash_bwd_prep(out, dout, lse, dq_acc=None):
    """``delta = rowsum(dO*O)`` and ``lse*log2(e)`` in ``(B, H, Sq_pad)`` fp32 buffers (padded to a
    multiple of 128 queries; padding and fully masked rows get ``+inf`` / 0). ``dq_acc`` (fp32, contiguous, ``out``'s
    shape), when given, is zeroed in the same launch."""
    _check_bshd(out, "out"); _check_bshd(dout, "dout")
    B, Sq, H, D = out.shape
    sq_pad = (Sq + 127) // 128 * 128
    lse2 = torch.empty(B, H, sq_pad, device=out.device, dtype=torch.float32)
    delta = torch.empty(B, H, sq_pad, device=out.device, dtype=torch.float32)
    assert lse.dtype == torch.float32 and lse.is_contiguous() and lse.shape == (B, H, Sq)
    assert dq_acc is None or (dq_acc.dtype == torch.float32 and dq_acc.is_contiguous() and dq_acc.shape == out.shape)
    _lib.call("ra_attn_bwd_prep", out.data_ptr(), *out.stride()[:3], dout.data_ptr(), *dout.stride()[:3], lse.data_ptr(),
              lse2.data_ptr(), delta.data_ptr(), _ptr(dq_acc), B, H, Sq, sq_pad, D, _lib.stream_handle())
    return lse2, delta


def flash_bwd(q, k, v, dout, lse2, delta, mask: MaskSpec, dq_acc, dk, dv, dkv_mode=DKV_STORE_BF16,
              *, copy_src: int = 0, copy_dst: int = 0, copy_bytes: int = 0, copy_ctas: int = 8):
    """One ring step of the backward. ``dq_acc`` (fp32, contiguous, pre-zeroed by the caller before
    the first step) receives ``dQ`` by reduction; ``dk``/``dv`` are written according to
    ``dkv_mode`` (store bf16, store fp32, or fp32 reduction into possibly remote memory)."""
    assert dq_acc.dtype == torch.float32 and dq_acc.is_contiguous() and dq_acc.shape == q.shape
    fields = _bwd_fields(q, k, v, dout, lse2.data_ptr(), delta.data_ptr(), lse2.shape[2], mask, dq_acc.data_ptr(), dk, dv, dkv_mode,
                         copy_src, copy_dst, copy_bytes, copy_ctas)
    _lib.call("ra_attn_bwd", _BWD_ARGS.pack(*fields))


def flash_bwd_run(q, k, v, out, lse, dout, mask: MaskSpec, dq, dk, dv) -> None:
    """The whole backward on one device in one call: :func:`flash_bwd_prep`, :func:`flash_bwd` and ``dq`` in bf16. ``dq``, ``dk`` and ``dv``
    are bf16 views; those of ``dq`` whose batch and sequence form rows of ``H * D`` values a fixed distance apart."""
    _check_bshd(out, "out")
    B, Sq, H, D = q.shape
    assert out.shape == q.shape and lse.dtype == torch.float32 and lse.is_contiguous() and lse.shape == (B, H, Sq)
    assert dq.shape == q.shape and dq.dtype == torch.bfloat16 and dq_rows(dq) is not None
    sq_pad = (Sq + 127) // 128 * 128
    n, rows = B * Sq * H * D, B * H * sq_pad
    scratch = torch.empty(n + 2 * rows, device=q.device, dtype=torch.float32)  # dq_acc, lse2, delta
    at = scratch.data_ptr()
    fields = _bwd_fields(q, k, v, dout, at + 4 * n, at + 4 * (n + rows), sq_pad, mask, at, dk, dv, DKV_STORE_BF16, 0, 0, 0, 0)
    _lib.call("ra_attn_bwd_run", _BWD_RUN_ARGS.pack(*fields, out.data_ptr(), *out.stride()[:3], lse.data_ptr(), dq.data_ptr(), dq_rows(dq)),
              n_kernels=3)


def dq_rows(dq: torch.Tensor) -> Optional[int]:
    """Distance in elements of the rows of ``H * D`` values that batch and sequence of ``dq (B, S, H, D)`` form, or None."""
    B, S, H, D = dq.shape
    sb, ss, sh, sd = dq.stride()
    return ss if sd == 1 and sh == D and sb == S * ss else None


def _bwd_fields(q, k, v, dout, lse2: int, delta: int, sq_pad: int, mask: MaskSpec, dq_acc: int, dk, dv, dkv_mode, copy_src, copy_dst,
                copy_bytes, copy_ctas) -> tuple:
    """The fields of ``RaAttnBwdArgs``."""
    _check_bshd(q, "q"); _check_bshd(k, "k"); _check_bshd(v, "v"); _check_bshd(dout, "dout")
    B, Sq, H, D = q.shape
    Sk = k.shape[1]
    dev = q.device
    assert dk.shape == k.shape and dv.shape == k.shape and dk.stride() == dv.stride()
    want = torch.bfloat16 if dkv_mode == DKV_STORE_BF16 else torch.float32
    assert dk.dtype == want and dv.dtype == want and dk.stride(3) == 1
    tb = BWD_TRACE_BUFFERS.get(dev.index if dev.index is not None else torch.cuda.current_device())
    return (q.data_ptr(), k.data_ptr(), v.data_ptr(), dout.data_ptr(), *q.stride()[:3], *k.stride()[:3], *v.stride()[:3],
            *dout.stride()[:3], lse2, delta, sq_pad, dq_acc, dk.data_ptr(), dv.data_ptr(), *dk.stride()[:3], dkv_mode, B, H, Sq, Sk, D,
            1.0 / math.sqrt(D), *_mask_fields(mask, H, by_k=True), copy_src, copy_dst, copy_bytes, copy_ctas,
            _lib.status_tensor(dev).data_ptr(), _lib.stream_handle(), 0 if tb is None else tb.data_ptr())
