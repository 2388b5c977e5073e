"""Primitive-major record grouping, same surface as scannet/primitive_csr.py:14-29.

`group_records` returns the same `PrimitiveCSR` fields; the stable grouping runs as a device-wide
radix sort inside libmlpsp_b200.so instead of torch.argsort/bincount/cumsum.
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass

import torch

from . import _lib as L
from .engine import _on, _stream_ptr


@dataclass
class PrimitiveCSR:
    offsets: torch.Tensor
    record_indices: torch.Tensor
    x6: torch.Tensor
    grad4: torch.Tensor
    relu_masks: torch.Tensor | None = None


def _group(primitive_ids, num_primitives, x6=None, grad4=None, relu_masks=None):
    lib = L.load()
    if not primitive_ids.is_cuda:
        raise RuntimeError("group_records runs on a CUDA device; there is no CPU path")
    ids = primitive_ids.to(torch.int32).contiguous()
    dev = ids.device
    R, n = int(ids.numel()), int(num_primitives)
    offsets = torch.empty(n + 1, device=dev, dtype=torch.int64)
    order = torch.empty(R, device=dev, dtype=torch.int64)
    outs = [None if t is None else torch.empty_like(t) for t in (x6, grad4, relu_masks)]
    nbytes = int(lib.mlpsp_group_records_scratch_bytes(R, n))
    scratch = torch.empty(nbytes, device=dev, dtype=torch.uint8)
    with _on(dev):
        st = _stream_ptr(dev)
        L.check(lib.mlpsp_group_rows(L.ptr(ids), R, n, L.ptr(x6), L.ptr(grad4), L.ptr(relu_masks), L.ptr(offsets), L.ptr(order),
                                     *(L.ptr(t) for t in outs), L.ptr(scratch), nbytes, st), "mlpsp_group_rows")
    return offsets, order, outs


def group_order(primitive_ids: torch.Tensor, num_primitives: int):
    """(offsets int64 [N+1], order int64 [R]): records grouped by primitive, record order kept inside a group."""
    return _group(primitive_ids, num_primitives)[:2]


def group_records(primitive_ids, x6, grad4, num_primitives: int, relu_masks=None) -> PrimitiveCSR:
    """Group records by primitive, preserving pixel order inside each group."""
    rows = [t for t in (x6, grad4, relu_masks) if t is not None]
    R = int(primitive_ids.numel())
    if (primitive_ids.is_cuda and all(t.is_contiguous() and t.device == primitive_ids.device for t in rows)
            and x6.dtype == torch.float32 and tuple(x6.shape) == (R, 6) and x6.data_ptr() % 8 == 0
            and grad4.dtype == torch.float32 and tuple(grad4.shape) == (R, 4) and grad4.data_ptr() % 16 == 0
            and (relu_masks is None or (relu_masks.dtype == torch.int32 and tuple(relu_masks.shape) == (R, 2)
                                        and relu_masks.data_ptr() % 8 == 0))
            and not any(t.requires_grad for t in rows)):
        # the record layout of the path: the sort's last kernel moves the rows as well
        offsets, order, outs = _group(primitive_ids, num_primitives, x6, grad4, relu_masks)
        return PrimitiveCSR(offsets, order, *outs)
    offsets, order = group_order(primitive_ids, num_primitives)
    return PrimitiveCSR(offsets, order, x6[order], grad4[order],
                        None if relu_masks is None else relu_masks[order])


@torch.no_grad()
def primitive_records_reverse(ids, offsets, x6, raw, log_scales, quats, grad_rgb, grad_t):
    """Reverse compositing over saved records, the extension entry of the same name in the reference
    (scannet/cuda/primitive_records.cuh:51-74): returns [d4 (R,4), grad_positions (N,3), grad_log_scales (N,3),
    grad_quats (N,4)].  ids int32 [R]; offsets int64 [pixels+1]; x6 [R,6]; raw [R,8]; float32 CUDA tensors."""
    for t in (ids, offsets, x6, raw, log_scales, quats, grad_rgb, grad_t):
        if not (t.is_cuda and t.is_contiguous() and t.device == ids.device):
            raise ValueError("all inputs must be contiguous tensors on one CUDA device")
    if ids.dtype != torch.int32 or offsets.dtype != torch.int64:
        raise ValueError("ids must be int32 and offsets int64")
    if any(t.dtype != torch.float32 for t in (x6, raw, log_scales, quats, grad_rgb, grad_t)):
        raise ValueError("records, geometry and adjoints must be FP32")
    total, pixels, n = int(ids.numel()), int(grad_rgb.shape[0]), int(log_scales.shape[0])
    if offsets.ndim != 1 or offsets.numel() != pixels + 1 or x6.shape != (total, 6) or raw.shape != (total, 8):
        raise ValueError("record tensors do not match the pixel offsets")
    if quats.shape != (n, 4) or log_scales.shape != (n, 3) or grad_rgb.shape != (pixels, 3) or grad_t.numel() != pixels:
        raise ValueError("geometry or adjoint shapes do not match")
    lib = L.load()
    dev = ids.device
    d4 = torch.empty((total, 4), device=dev, dtype=torch.float32)
    gp = torch.empty((n, 3), device=dev, dtype=torch.float32)
    gs = torch.empty((n, 3), device=dev, dtype=torch.float32)
    gq = torch.empty((n, 4), device=dev, dtype=torch.float32)
    nbytes = int(lib.mlpsp_records_reverse_scratch_bytes(total, n))
    scratch = torch.empty(nbytes, device=dev, dtype=torch.uint8)
    found = C.c_int32(0)
    with _on(dev):
        st = _stream_ptr(dev)
        L.check(lib.mlpsp_records_reverse_checked(
            L.ptr(ids), L.ptr(offsets), L.ptr(x6), L.ptr(raw), L.ptr(log_scales), L.ptr(quats), L.ptr(grad_rgb), L.ptr(grad_t),
            pixels, total, n, L.ptr(d4), L.ptr(gp), L.ptr(gs), L.ptr(gq), L.ptr(scratch), nbytes, C.byref(found), st),
            "mlpsp_records_reverse")
    if found.value & L.REVERSE_BAD_OFFSETS:
        raise ValueError("pixel offsets must start at zero, end at the record count and be monotone")
    if found.value & L.REVERSE_BAD_IDS:
        raise ValueError("record primitive ids out of range")
    return [d4, gp, gs, gq]
