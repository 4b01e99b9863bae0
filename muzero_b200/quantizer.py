"""Quantizer front end: alpha selection and flat-row quantize / dequantize.

Mirrors the public functions of the reference's ``muzero/quantizer.py``
(``select_alpha`` :29-83, ``quantize_rows`` :119-158, ``dequantize_rows``
:205-226, ``roundtrip`` :273-323).  The row kernels are the CUDA library's; there
is no torch or Triton backend behind them, so CPU tensors raise.
Alpha selection is a one-time statistic per layer, taken on the device (``mz_alpha_stats``) for 16-bit CUDA blocks and in
torch otherwise; code widths with one alpha take none.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch
import torch.nn.functional as F

from .kernels._cabi import check, dtype_code, on_device, stream_ptr
from .kernels.loader import (MuZeroKernelError, ensure_expand_table, load_mu_zero_cuda_extension, mu_zero_dequantize_cuda,
                             mu_zero_quantize_cuda)

_TINY = 1e-8


def alpha_from_stats(*, bits: int, kind: str, tail_ratio: float, concentration_ratio: float,
                     anchor_offset: float) -> float:
    """Decision table of the reference (muzero/quantizer.py:65-83)."""
    if kind == "key":
        if bits == 1:
            if tail_ratio > 3.0 or concentration_ratio > 12.0 or anchor_offset > 0.22:
                return 16.0
            if tail_ratio > 2.0 or concentration_ratio > 8.0 or anchor_offset > 0.16:
                return 4.0
            return 2.0
        if bits == 8 and (tail_ratio > 2.6 or concentration_ratio > 10.0):
            return 4.0
        return 2.0
    if bits >= 8:
        if tail_ratio > 2.0 or concentration_ratio > 6.0 or anchor_offset > 0.14:
            return 4.0
        return 2.0
    if bits == 3 and tail_ratio > 2.3 and anchor_offset > 0.12:
        return 4.0
    return 2.0


def _statistics_needed(bits: int, kind: str) -> int:
    """Which statistics the decision table reads for (bits, kind): 1 = magnitude ratios, 2 = anchor offset.  Most
    code widths have one alpha whatever the data is."""
    if kind == "key":
        return {1: 3, 8: 1}.get(bits, 0)
    return 3 if bits >= 8 else 1 if bits == 3 else 0


def _anchor_decides(bits: int, kind: str, tail: float, conc: float) -> bool:
    """Whether the anchor offset can still change the choice once the magnitude ratios are known."""
    if not _statistics_needed(bits, kind):
        return False
    a, b = (alpha_from_stats(bits=bits, kind=kind, tail_ratio=tail, concentration_ratio=conc, anchor_offset=off)
            for off in (0.0, 0.5))
    return a != b


_stat_workspaces: dict = {}


def _stat_workspace(device: torch.device) -> torch.Tensor:
    key = (device.index, torch.cuda.current_stream(device).cuda_stream)
    ws = _stat_workspaces.get(key)
    if ws is None:
        if len(_stat_workspaces) >= 64:      # streams come and go; the oldest buffer's stream orders what is still in flight
            _stat_workspaces.pop(next(iter(_stat_workspaces)), None)
        ws = torch.zeros(load_mu_zero_cuda_extension().mz_alpha_stats_workspace_bytes(), dtype=torch.uint8, device=device)
        _stat_workspaces[key] = ws
    return ws


def device_alphas(requests: list, *, bits: int, q_group_size: int, max_points: int) -> list:
    """Alphas of 16-bit CUDA blocks [B,H,S,D] (innermost contiguous): ``requests`` holds (block, kind, sample order)
    with the orders of ``mz_alpha_stats``.  The statistics of all requests are read back with one copy."""
    lib = load_mu_zero_cuda_extension()
    out: list = [None] * len(requests)
    stats: list = [None] * len(requests)

    def launch(todo: list) -> None:
        dev = requests[todo[0][0]][0].device
        buf = torch.empty((len(todo), 4), dtype=torch.float32, device=dev)
        ws, st = _stat_workspace(dev), stream_ptr(dev)
        with torch.cuda.device(dev):
            for row, (i, want) in enumerate(todo):
                block, kind, order = requests[i]
                check(lib.mz_alpha_stats(block.data_ptr(), dtype_code(block.dtype), (ctypes.c_int * 4)(*block.shape),
                                         (ctypes.c_longlong * 3)(*block.stride()[:3]), q_group_size, int(kind == "key"), order,
                                         max_points, want, ws.data_ptr(), buf.data_ptr() + 16 * row, st), "mz_alpha_stats")
        for (i, want), got in zip(todo, buf.tolist()):
            stats[i] = (got[:3] if want & 1 else stats[i][:3]) + [got[3] if want & 2 else None]

    todo = []
    for i, (_, kind, _) in enumerate(requests):
        want = _statistics_needed(bits, kind)
        if want:
            todo.append((i, want))
        else:
            out[i] = alpha_from_stats(bits=bits, kind=kind, tail_ratio=0.0, concentration_ratio=0.0, anchor_offset=0.0)
    while todo:
        launch(todo)
        again = []
        for i, _ in todo:
            kind = requests[i][1]
            p50, p95, p99, off = stats[i]
            tail, conc = p99 / max(p95, _TINY), p95 / max(p50, _TINY)
            if off is None and _anchor_decides(bits, kind, tail, conc):
                again.append((i, 2))
            else:
                out[i] = alpha_from_stats(bits=bits, kind=kind, tail_ratio=tail, concentration_ratio=conc, anchor_offset=off or 0.0)
        todo = again
    return out


def _on_device(block: torch.Tensor) -> bool:
    return block.is_cuda and block.dtype in (torch.bfloat16, torch.float16) and block.dim() == 4 and block.stride(-1) == 1


def _magnitude_ratios(sample: torch.Tensor) -> tuple[float, float]:
    """(p99/p95, p95/p50) of |sample| by order statistics at k = max(1, floor(p*n))."""
    mag = sample.float().abs().reshape(-1)
    n = mag.numel()
    ks = [max(1, int(p * n)) for p in (0.50, 0.95, 0.99)]
    ordered, _ = torch.sort(mag)
    p50, p95, p99 = (float(v) for v in ordered[torch.tensor(ks, device=mag.device) - 1].tolist())
    return p99 / max(p95, _TINY), p95 / max(p50, _TINY)


def _strided_sample(flat: torch.Tensor, max_points: int) -> torch.Tensor:
    if flat.numel() <= max_points:
        return flat
    step = max(1, flat.numel() // max_points)
    return flat[::step][:max_points]


def _anchor_offset(groups: torch.Tensor) -> float:
    """mean |zero_anchor - 0.5| over groups laid out on the last axis."""
    lo = groups.amin(dim=-1)
    hi = groups.amax(dim=-1)
    anchor = ((0.0 - lo) / (hi - lo).clamp_min(_TINY)).clamp(0.0, 1.0)
    return float((anchor - 0.5).abs().mean())


def select_alpha(tensor: torch.Tensor, *, bits: int, q_group_size: int, kind: str,
                 max_points: int = 65536) -> float:
    """Log-compander alpha for ``tensor`` ([N,G] rows or [B,H,S,D]); always 2.0 where the decision table has one value."""
    if not _statistics_needed(bits, kind):
        return 2.0
    if _on_device(tensor) and (kind == "key" or tensor.shape[3] % q_group_size == 0):
        return device_alphas([(tensor, kind, -1)], bits=bits, q_group_size=q_group_size, max_points=max_points)[0]
    work = tensor.float()
    tail, conc = _magnitude_ratios(_strided_sample(work.reshape(-1), max_points))
    if not _anchor_decides(bits, kind, tail, conc):
        return alpha_from_stats(bits=bits, kind=kind, tail_ratio=tail, concentration_ratio=conc, anchor_offset=0.0)
    if work.dim() == 2:
        rows, width = work.shape
        if width != q_group_size:
            ng = max(1, width // q_group_size)
            work = work[:, : ng * q_group_size].reshape(rows, ng, q_group_size)
    else:
        if kind == "key":
            work = work.transpose(2, 3).contiguous()
        b, h, s, d = work.shape
        d_pad = -(-d // q_group_size) * q_group_size
        if d_pad != d:
            work = F.pad(work, (0, d_pad - d))
        work = work.reshape(b, h, s, d_pad // q_group_size, q_group_size)
    return alpha_from_stats(bits=bits, kind=kind, tail_ratio=tail, concentration_ratio=conc,
                            anchor_offset=_anchor_offset(work))


def select_alpha_key_block(block: torch.Tensor, *, bits: int, q_group_size: int, max_points: int = 65536) -> float:
    """``select_alpha(rows, kind="key")`` for the rows [B*KVH*nsg*D, G] of a key block
    [B,KVH,nsg*G,D], without materialising the transposed rows: the strided sample is
    gathered through the row index arithmetic and the group min/max reduce over the token axis.
    """
    if not _statistics_needed(bits, "key"):
        return 2.0
    if _on_device(block):
        return device_alphas([(block, "key", 1)], bits=bits, q_group_size=q_group_size, max_points=max_points)[0]
    b, h, s, d = block.shape
    g = q_group_size
    nsg = s // g
    total = b * h * nsg * d * g
    step = max(1, total // max_points) if total > max_points else 1
    idx = torch.arange(0, total, step, device=block.device)[:max_points] if total > max_points \
        else torch.arange(0, total, device=block.device)
    t = idx % g
    rest = idx // g
    ch = rest % d
    rest = rest // d
    grp = rest % nsg
    rest = rest // nsg
    hh = rest % h
    bb = rest // h
    sample = block[bb, hh, grp * g + t, ch]
    tail, conc = _magnitude_ratios(sample)
    grouped = block[:, :, : nsg * g].float().reshape(b, h, nsg, g, d).transpose(3, 4)
    return alpha_from_stats(bits=bits, kind="key", tail_ratio=tail, concentration_ratio=conc,
                            anchor_offset=_anchor_offset(grouped))


def quantize_rows(flat_grouped: torch.Tensor, bits: int, alpha: float, amax_eps: float,
                  amax_dtype: torch.dtype, *, backend: str = "auto", _cuda_ok: bool = True,
                  _triton_ok: bool = True):
    """[N,G] -> (packed uint8 [N,QB], mn [N,1], scale [N,1]).  ``backend`` is ignored."""
    if not flat_grouped.is_cuda:
        raise MuZeroKernelError("quantize_rows needs a CUDA tensor; this package has no CPU path")
    n, g = flat_grouped.shape
    qb = (g * bits + 7) // 8
    dev = flat_grouped.device
    packed = torch.empty((n, qb), dtype=torch.uint8, device=dev)
    mn = torch.empty((n, 1), dtype=amax_dtype, device=dev)
    scale = torch.empty((n, 1), dtype=amax_dtype, device=dev)
    mu_zero_quantize_cuda(flat_grouped.contiguous(), packed, mn, scale, bits, float(alpha), amax_eps)
    return packed, mn, scale


def dequantize_rows(packed_q: torch.Tensor, mn: torch.Tensor, scale: torch.Tensor, bits: int, alpha: float,
                    q_group_size: int, out_dtype: torch.dtype, *, amax_eps: float = 1e-8,
                    _cuda_ok: bool = True) -> torch.Tensor:
    """Inverse of ``quantize_rows``: [N,QB] -> [N,G] in ``out_dtype``."""
    if not packed_q.is_cuda:
        raise MuZeroKernelError("dequantize_rows needs CUDA tensors; this package has no CPU path")
    out = torch.empty((packed_q.shape[0], q_group_size), dtype=out_dtype, device=packed_q.device)
    mu_zero_dequantize_cuda(packed_q.contiguous(), mn.contiguous(), scale.contiguous(), out, bits, float(alpha), amax_eps)
    return out


def _fused_roundtrip_serves(t: torch.Tensor, g: int, kind: str) -> bool:
    """The shapes of ``mz_roundtrip_kv``; others go through rows."""
    b, h, s, d = t.shape
    unit = 1 if kind == "key" else 7
    return (_on_device(t) and t.numel() > 0 and d in (64, 128) and g in (32, 64, 128) and d % g == 0 and s < 1 << 27
            and (kind == "value" or s % g == 0) and not any(x & unit for x in t.stride()[:3])
            and t.data_ptr() % (4 if kind == "key" else 16) == 0)


def _fused_roundtrip(key: torch.Tensor, value: torch.Tensor, bits: int, g: int, alpha_key: float, alpha_value: float,
                     amax_dtype: torch.dtype, amax_eps: float):
    outs, args = [], []
    for t, alpha in ((key, alpha_key), (value, alpha_value)):
        ensure_expand_table(bits, alpha, t.device)
        outs.append(t.new_empty(t.shape))
        args += [t.data_ptr(), (ctypes.c_int * 4)(*t.shape), (ctypes.c_longlong * 3)(*t.stride()[:3]), float(alpha), outs[-1].data_ptr()]
    check(on_device(key.device, load_mu_zero_cuda_extension().mz_roundtrip_kv, *args, dtype_code(key.dtype), g, bits, float(amax_eps),
                    dtype_code(amax_dtype), stream_ptr(key.device)), "mz_roundtrip_kv")
    return tuple(outs)


def roundtrip(key: torch.Tensor, value: torch.Tensor, *, bits: int = 4, q_group_size: int = 64,
              alpha_key: Optional[float] = None, alpha_value: Optional[float] = None,
              amax_dtype: torch.dtype = torch.float16, amax_eps: float = 1e-8):
    """Quantize then dequantize K ([B,H,S,D], grouped over tokens) and V (grouped over channels)."""
    g = q_group_size
    if alpha_key is None:
        alpha_key = select_alpha(key, bits=bits, q_group_size=g, kind="key")
    if alpha_value is None:
        alpha_value = select_alpha(value, bits=bits, q_group_size=g, kind="value")

    if (key.dtype == value.dtype and key.device == value.device and _fused_roundtrip_serves(key, g, "key")
            and _fused_roundtrip_serves(value, g, "value")):
        return _fused_roundtrip(key, value, bits, g, alpha_key, alpha_value, amax_dtype, amax_eps)
    b, h, s, d = key.shape
    nsg = s // g
    rows = key.reshape(b, h, nsg, g, d).transpose(3, 4).contiguous().reshape(-1, g).float()
    back = dequantize_rows(*quantize_rows(rows, bits, alpha_key, amax_eps, amax_dtype), bits, alpha_key, g,
                           key.dtype, amax_eps=amax_eps)
    key_out = back.reshape(b, h, nsg, d, g).transpose(3, 4).reshape(b, h, s, d).contiguous()

    b, h, s, d = value.shape
    d_pad = -(-d // g) * g
    padded = F.pad(value, (0, d_pad - d)) if d_pad != d else value
    rows = padded.reshape(-1, g).float()
    back = dequantize_rows(*quantize_rows(rows, bits, alpha_value, amax_eps, amax_dtype), bits, alpha_value, g,
                           value.dtype, amax_eps=amax_eps)
    value_out = back.reshape(b, h, s, d_pad)[..., :d].contiguous()
    return key_out, value_out
