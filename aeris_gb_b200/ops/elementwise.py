"""Python front ends of the memory-bound kernels in ``csrc/elementwise.cu``."""
from __future__ import annotations

import ctypes

import torch

from . import lib as _l
from .build import CHECKED as _CHECKED

MODE_MOD_THEN_NORM = 0   # h = RMSNorm(x * (1 + scale) + shift) * w      (layerwise_t_emb_after_mod_norm)
MODE_NORM_THEN_MOD = 1   # h = (RMSNorm(x) * w) * (1 + scale) + shift    (DiT ordering)


def _peer_array(ptrs: list[int]):
    arr = (ctypes.c_void_p * len(ptrs))(*ptrs)
    return arr


def _pitch(v: torch.Tensor, batch: int, D: int) -> int | None:
    """Elements between the rows of ``v`` [batch, D], or None where the kernels cannot read it in place."""
    if v.is_contiguous() and v.numel() == batch * D:
        return D
    return v.stride(0) if v.shape == (batch, D) and v.stride(1) == 1 and v.stride(0) % 4 == 0 else None


def modnorm_fwd(x: torch.Tensor, scale: torch.Tensor | None, shift: torch.Tensor | None, w: torch.Tensor, *,
                mode: int, eps: float, out: torch.Tensor | None = None, gather_idx: torch.Tensor | None = None,
                peer_ptrs: list[int] | None = None, x_out: torch.Tensor | None = None,
                rows: int | None = None, out_lo: torch.Tensor | None = None,
                src_rows: int | None = None, batch: int = 1) -> torch.Tensor:
    """``w`` bf16, or fp32 (the output head's norm); ``out_lo`` optionally receives ``h - bf16(h)``. ``src_rows``: rows of
    every peer buffer the gather table points into (used by the checking build only). ``batch`` > 1: the rows are that
    many samples of equal length, ``scale`` and ``shift`` are [batch, D], without gaps inside a row."""
    D = w.numel()
    rows = rows if rows is not None else (gather_idx.numel() if gather_idx is not None else x.shape[0])
    if _CHECKED and gather_idx is not None:
        set_gather_bounds(src_rows or 0)
    if out is None:
        out = torch.empty((rows, D), dtype=torch.bfloat16, device=w.device)
    peers = _peer_array(peer_ptrs) if gather_idx is not None else None
    w32, w = (w, None) if w.dtype == torch.float32 else (None, w)
    stride = D
    if batch > 1:
        pitches = {_pitch(v, batch, D) for v in (scale, shift) if v is not None} or {D}
        stride = pitches.pop()
        assert rows % batch == 0 and stride is not None and not pitches
    head = (_l.ptr(x), _l.ptr(gather_idx), peers, len(peer_ptrs) if peer_ptrs else 0, _l.ptr(x_out), _l.ptr(scale),
            _l.ptr(shift))
    tail = (D, mode, _l._c_float(eps), _l.ptr(w32), _l.ptr(out_lo), _l.stream_ptr())
    rc = (_l.lib().aeris_modnorm_fwd(*head, _l.ptr(w), _l.ptr(out), rows, *tail) if batch == 1 else
          _l.lib().aeris_modnorm_fwd_batch(*head, stride, _l.ptr(w), _l.ptr(out), batch, rows // batch, *tail))
    _l.check(rc, "aeris_modnorm_fwd")
    return out


def modnorm_bwd(x: torch.Tensor, dh: torch.Tensor, dres: torch.Tensor | None, scale: torch.Tensor | None,
                shift: torch.Tensor | None, w: torch.Tensor, *, mode: int, eps: float, dx: torch.Tensor,
                dscale: torch.Tensor | None, dshift: torch.Tensor | None, dw: torch.Tensor | None) -> torch.Tensor:
    rows, D = x.shape
    w32, w = (w, None) if w.dtype == torch.float32 else (None, w)
    rc = _l.lib().aeris_modnorm_bwd(_l.ptr(x), _l.ptr(dh), _l.ptr(dres), _l.ptr(scale), _l.ptr(shift), _l.ptr(w),
                                    _l.ptr(dx), _l.ptr(dscale), _l.ptr(dshift), _l.ptr(dw), rows, D, mode,
                                    _l._c_float(eps), _l.ptr(w32), _l.stream_ptr())
    _l.check(rc, "aeris_modnorm_bwd")
    return dx


def modnorm_fwd_f32(x: torch.Tensor, scale: torch.Tensor, shift: torch.Tensor, w: torch.Tensor, *, mode: int, eps: float,
                    out: torch.Tensor) -> torch.Tensor:
    """:func:`modnorm_fwd` with an fp32 result ``out`` [rows, D]; ``w`` fp32, ``scale`` and ``shift`` [batch, D]."""
    B, D = scale.shape
    rc = _l.lib().aeris_modnorm_fwd_f32(_l.ptr(x), _l.ptr(scale), _l.ptr(shift), _l.ptr(w), _l.ptr(out), B,
                                        x.shape[0] // B, D, mode, _l._c_float(eps), _l.stream_ptr())
    _l.check(rc, "aeris_modnorm_fwd_f32")
    return out


def modnorm_bwd_f32(x: torch.Tensor, dh: torch.Tensor, scale: torch.Tensor, shift: torch.Tensor, w: torch.Tensor, *,
                    mode: int, eps: float, dx: torch.Tensor, dscale: torch.Tensor, dshift: torch.Tensor,
                    dw: torch.Tensor) -> None:
    """Backward of :func:`modnorm_fwd_f32` for one sample, ``dh`` fp32; ``dscale``, ``dshift`` and ``dw`` are added to."""
    rows, D = x.shape
    ctas = torch.cuda.get_device_properties(x.device).multi_processor_count      # one per SM at most, one row of sums each
    sums = torch.empty((ctas, 3, D), dtype=torch.float32, device=x.device)
    rc = _l.lib().aeris_modnorm_bwd_f32(_l.ptr(x), _l.ptr(dh), _l.ptr(scale), _l.ptr(shift), _l.ptr(w), _l.ptr(dx),
                                        _l.ptr(dscale), _l.ptr(dshift), _l.ptr(dw), _l.ptr(sums), sums.shape[0], rows, D,
                                        mode, _l._c_float(eps), _l.stream_ptr())
    _l.check(rc, "aeris_modnorm_bwd_f32")


def set_gather_bounds(src_rows: int) -> bool:
    """Checking build (AERIS_BOUNDS_CHECK=1) only: rows of the source buffers of the gathers launched next, so that
    every table entry is validated on the device. Returns whether the loaded library checks at all."""
    return bool(_l.lib().aeris_debug_set_gather_bounds(_l.ptr(_l.status_word()), int(src_rows)))


def gather_rows(gather_idx: torch.Tensor, peer_ptrs: list[int], out: torch.Tensor,
                src_rows: int | None = None) -> torch.Tensor:
    rows, D = out.shape
    if _CHECKED:
        set_gather_bounds(src_rows or 0)
    rc = _l.lib().aeris_gather_rows(_l.ptr(gather_idx), _peer_array(peer_ptrs), len(peer_ptrs), _l.ptr(out),
                                    _l._c_ll(rows), D, _l.stream_ptr())
    _l.check(rc, "aeris_gather_rows")
    return out


def swiglu_fwd(u: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    rows, F2 = u.shape
    F = F2 // 2
    if out is None:
        out = torch.empty((rows, F), dtype=u.dtype, device=u.device)
    _l.check(_l.lib().aeris_swiglu_fwd(_l.ptr(u), _l.ptr(out), _l._c_ll(rows), F, _l.stream_ptr()), "swiglu_fwd")
    return out


def swiglu_bwd(u: torch.Tensor, dact: torch.Tensor, du: torch.Tensor | None = None) -> torch.Tensor:
    rows, F2 = u.shape
    if du is None:
        du = torch.empty_like(u)
    _l.check(_l.lib().aeris_swiglu_bwd(_l.ptr(u), _l.ptr(dact), _l.ptr(du), _l._c_ll(rows), F2 // 2,
                                       _l.stream_ptr()), "swiglu_bwd")
    return du


def scale_rows(W: torch.Tensor, g: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    R, C = W.shape
    if out is None:
        out = torch.empty_like(W)
    _l.check(_l.lib().aeris_scale_rows(_l.ptr(W), _l.ptr(g), _l.ptr(out), R, C, _l.stream_ptr()), "scale_rows")
    return out


def rope_qk_(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, L: int, heads: int, head_dim: int,
             inverse: bool = False) -> torch.Tensor:
    """Rotates the q and k sections of ``qkv`` [rows, 3 * heads * head_dim] (bf16, contiguous) in place by the 2-D rotary
    angles ``cos`` / ``sin`` [L, head_dim / 2] (fp32); row r belongs to token r mod L of its window."""
    assert qkv.is_contiguous() and qkv.shape[1] == 3 * heads * head_dim and cos.shape == (L, head_dim // 2)
    _l.check(_l.lib().aeris_rope_qk(_l.ptr(qkv), _l.ptr(cos), _l.ptr(sin), _l._c_ll(qkv.shape[0]), L, heads, head_dim,
                                    int(inverse), _l.stream_ptr()), "rope_qk")
    return qkv


def gate_grad_finalize(G: torch.Tensor, W: torch.Tensor, g: torch.Tensor, dW: torch.Tensor, dg: torch.Tensor) -> None:
    R, C = W.shape
    _l.check(_l.lib().aeris_gate_grad_finalize(_l.ptr(G), _l.ptr(W), _l.ptr(g), _l.ptr(dW), _l.ptr(dg), R, C,
                                               _l.stream_ptr()), "gate_grad_finalize")


def sumsq(x: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    _l.check(_l.lib().aeris_sumsq(_l.ptr(x), _l._c_ll(x.numel()), _l.ptr(out), _l.stream_ptr()), "sumsq")
    return out


def adamw(master: torch.Tensor, grad: torch.Tensor, m: torch.Tensor, v: torch.Tensor, wbf16: torch.Tensor | None,
          ema: torch.Tensor | None, norm_sq: torch.Tensor | None, *, lr: float, betas: tuple[float, float],
          eps: float, weight_decay: float, step: int, grad_scale: float, max_norm: float, ema_beta: float) -> None:
    f = _l._c_float
    _l.check(_l.lib().aeris_adamw(_l.ptr(master), _l.ptr(grad), _l.ptr(m), _l.ptr(v), _l.ptr(wbf16), _l.ptr(ema),
                                  _l.ptr(norm_sq), _l._c_ll(master.numel()), f(lr), f(betas[0]), f(betas[1]),
                                  f(eps), f(weight_decay), step, f(grad_scale), f(max_norm), f(ema_beta),
                                  _l.stream_ptr()), "adamw")
