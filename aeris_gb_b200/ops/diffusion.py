"""Python front ends of ``csrc/diffusion.cu``: noising + embedding pack, TrigFlow loss, sampler updates, channel
affine maps and the small-batch GEMV of the modulation MLPs."""
from __future__ import annotations

import ctypes

import torch

from . import lib as _l


class TokGeom(ctypes.Structure):
    """Mirror of the C struct: this rank's token stream / image block inside the global image."""
    _fields_ = [("B", ctypes.c_int), ("nwy_loc", ctypes.c_int), ("nwx_loc", ctypes.c_int), ("ws_y", ctypes.c_int),
                ("ws_x", ctypes.c_int), ("n_local", ctypes.c_int), ("sp_rank", ctypes.c_int), ("y0", ctypes.c_int),
                ("x0", ctypes.c_int), ("H", ctypes.c_int), ("W", ctypes.c_int), ("sample0", ctypes.c_longlong)]

    @property
    def rows(self) -> int:
        return self.B * self.nwy_loc * self.nwx_loc * self.n_local

    @property
    def block_shape(self) -> tuple[int, int, int]:
        return self.B, self.nwy_loc * self.ws_y, self.nwx_loc * self.ws_x


def make_geom(grid, batch: int, rank: int = 0, sample0: int = 0) -> TokGeom:
    """Geometry of ``rank`` (= wp_rank * sp + sp_rank) of a :class:`aeris_gb_b200.models.layout.Grid`."""
    ry, rx = grid.rank_coords(rank)
    return TokGeom(batch, grid.nwy_loc, grid.nwx_loc, grid.ws_y, grid.ws_x, grid.n_local, rank % grid.sp,
                   ry * grid.nwy_loc * grid.ws_y, rx * grid.nwx_loc * grid.ws_x, grid.H, grid.W, sample0)


def _u64(v: int) -> ctypes.c_ulonglong:
    return ctypes.c_ulonglong(v & 0xFFFFFFFFFFFFFFFF)


def embed_pack(x_img: torch.Tensor, c_img: torch.Tensor | None, cs: torch.Tensor, g: TokGeom,
               ape_y: torch.Tensor | None, ape_x: torch.Tensor | None, seed: int, sigma_data: float, noise: bool,
               out: torch.Tensor, row0: int = 0) -> torch.Tensor:
    """Rows ``[row0, row0 + out.shape[0])`` of the packed model input ``[hi | lo | hi | 1 | 1 | 0..]`` (bf16)."""
    Cx = x_img.shape[-1]
    Cc = c_img.shape[-1] if c_img is not None else 0
    rc = _l.lib().aeris_embed_pack(_l.ptr(x_img), _l.ptr(c_img), _l.ptr(cs), ctypes.byref(g), Cx, Cc, _l.ptr(ape_y),
                                   _l.ptr(ape_x), ape_y.shape[1] if ape_y is not None else 0, _u64(seed),
                                   _l._c_float(sigma_data), int(noise), _l.ptr(out), out.stride(0),
                                   _l._c_ll(row0), _l._c_ll(out.shape[0]), _l.stream_ptr())
    _l.check(rc, "aeris_embed_pack")
    return out


def trigflow_loss(pred: torch.Tensor, x_img: torch.Tensor, cs: torch.Tensor, g: TokGeom, seed: int,
                  sigma_data: float, w_var: torch.Tensor | None, w_lat: torch.Tensor | None, inv_rows: float,
                  loss: torch.Tensor, dpred: torch.Tensor | None = None, gscale: float = 1.0, row0: int = 0) -> None:
    """Adds the loss of ``pred.shape[0]`` rows starting at ``row0`` to ``loss`` (float64 [1]); writes d loss / d pred."""
    rc = _l.lib().aeris_trigflow_loss(_l.ptr(pred), pred.stride(0), _l.ptr(x_img), _l.ptr(cs), ctypes.byref(g),
                                      x_img.shape[-1], _u64(seed), _l._c_float(sigma_data), _l.ptr(w_var),
                                      _l.ptr(w_lat), _l._c_float(inv_rows), _l._c_float(gscale), _l.ptr(dpred),
                                      dpred.stride(0) if dpred is not None else 4, _l.ptr(loss), _l._c_ll(row0),
                                      _l._c_ll(pred.shape[0]), _l.stream_ptr())
    _l.check(rc, "aeris_trigflow_loss")


def sampler_update(x_out: torch.Tensor, x_base: torch.Tensor, pa: torch.Tensor, pb: torch.Tensor | None, ca: float,
                   cb: float, g: TokGeom) -> torch.Tensor:
    """``x_out = x_base + ca * pa + cb * pb`` with ``pa, pb`` [rows, ld] fp32 in token order, x in image order."""
    rc = _l.lib().aeris_sampler_update(_l.ptr(x_out), _l.ptr(x_base), _l.ptr(pa), _l.ptr(pb), pa.stride(0),
                                       _l._c_float(ca), _l._c_float(cb), ctypes.byref(g), x_out.shape[-1],
                                       _l.stream_ptr())
    _l.check(rc, "aeris_sampler_update")
    return x_out


def noise_mix(x: torch.Tensor, a: float, b: float, seed: int, g: TokGeom) -> torch.Tensor:
    """In place ``x = a * x + b * z`` with z ~ N(0, 1) from the counter-based generator (x: [B, hb, wb, C] fp32)."""
    rc = _l.lib().aeris_noise_mix(_l.ptr(x), _l._c_float(a), _l._c_float(b), _u64(seed), ctypes.byref(g),
                                  x.shape[-1], _l.stream_ptr())
    _l.check(rc, "aeris_noise_mix")
    return x


def affine_channels(inp: torch.Tensor, a: torch.Tensor, b: torch.Tensor, add: torch.Tensor | None = None,
                    out: torch.Tensor | None = None) -> torch.Tensor:
    """``out = inp * a[c] + b[c] (+ add)`` over the last (channel) axis, fp32."""
    if out is None:
        out = torch.empty_like(inp)
    rc = _l.lib().aeris_affine_channels(_l.ptr(out), _l.ptr(inp), _l.ptr(a), _l.ptr(b), _l.ptr(add),
                                        _l._c_ll(inp.numel()), inp.shape[-1], _l.stream_ptr())
    _l.check(rc, "aeris_affine_channels")
    return out


def _gemv_flags(W: torch.Tensor, bias: torch.Tensor | None, x: torch.Tensor) -> int:
    return (int(W.dtype == torch.float32) | 2 * int(bias is not None and bias.dtype == torch.bfloat16)
            | 4 * int(x.dtype == torch.bfloat16))


def _f32_or_bf16(t: torch.Tensor | None) -> torch.Tensor | None:
    return t if t is None or t.dtype in (torch.float32, torch.bfloat16) else t.float()


def gemv_ok(B: int, K: int) -> bool:
    """Whether :func:`gemv_bias_act` takes ``B`` rows of ``K`` columns: at most 8, and what the kernel pads them to (1, 2, 4
    or 8 rows of whole vectors, fp32) in 200 KB of shared memory."""
    return B <= 8 and 4 * (1 << (B - 1).bit_length()) * ((K + 3) // 4 * 4) <= 200 * 1024


def gemv_bias_act(W: torch.Tensor, bias: torch.Tensor | None, x: torch.Tensor, act: int = 0,
                  silu_in: bool = False) -> torch.Tensor:
    """``act(silu?(x) @ W^T + bias)`` for the few rows of ``x`` that :func:`gemv_ok` accepts; W [N, K], bias and x bf16 or
    fp32; fp32 result."""
    N, K = W.shape
    x, bias = _f32_or_bf16(x).contiguous(), _f32_or_bf16(bias)
    B = x.shape[0]
    y = torch.empty((B, N), dtype=torch.float32, device=x.device)
    rc = _l.lib().aeris_gemv_bias_act(_l.ptr(W), _gemv_flags(W, bias, x), _l.ptr(bias), _l.ptr(x), _l.ptr(y), N,
                                      K, B, act, int(silu_in), _l.stream_ptr())
    _l.check(rc, "aeris_gemv_bias_act")
    return y


def modulation_mlp(W1: torch.Tensor, b1: torch.Tensor, x: torch.Tensor, W2: torch.Tensor,
                   b2: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """``y1 = x @ W1^T + b1`` and ``silu(y1) @ W2^T + b2``, fp32: two :func:`gemv_bias_act` in one call."""
    (N1, K), N2 = W1.shape, W2.shape[0]
    assert W2.shape[1] == N1
    x, b1, b2 = _f32_or_bf16(x).contiguous(), _f32_or_bf16(b1), _f32_or_bf16(b2)
    B = x.shape[0]
    y1 = torch.empty((B, N1), dtype=torch.float32, device=x.device)
    y2 = torch.empty((B, N2), dtype=torch.float32, device=x.device)
    rc = _l.lib().aeris_modulation_mlp(_l.ptr(W1), _gemv_flags(W1, b1, x), _l.ptr(b1), _l.ptr(x), _l.ptr(y1), N1, K,
                                       _l.ptr(W2), _gemv_flags(W2, b2, y1), _l.ptr(b2), _l.ptr(y2), N2, B, _l.stream_ptr())
    _l.check(rc, "aeris_modulation_mlp", kernels=2)
    return y1, y2


def gemv_bwd(W: torch.Tensor, x: torch.Tensor, dy: torch.Tensor, dW: torch.Tensor, db: torch.Tensor | None,
             dx: torch.Tensor | None, silu_in: bool = False) -> None:
    """Adds the gradients of ``silu?(x) @ W^T + b`` (at most 8 rows) to fp32 ``dW``, ``db`` and ``dx``."""
    N, K = W.shape
    x, dy = _f32_or_bf16(x).contiguous(), dy.float().contiguous()
    rc = _l.lib().aeris_gemv_bwd(_l.ptr(W), _gemv_flags(W, None, x), _l.ptr(x), _l.ptr(dy), _l.ptr(dW), _l.ptr(db),
                                 _l.ptr(dx), N, K, x.shape[0], int(silu_in), _l.stream_ptr())
    _l.check(rc, "aeris_gemv_bwd")


def modulation_mlp_bwd(W1: torch.Tensor, x: torch.Tensor, W2: torch.Tensor, y1: torch.Tensor, dy: torch.Tensor,
                       dW1: torch.Tensor, db1: torch.Tensor, dW2: torch.Tensor, db2: torch.Tensor,
                       need_dx: bool) -> torch.Tensor | None:
    """Adds the gradients of :func:`modulation_mlp` to fp32 ``dW1 .. db2``; returns that of ``x`` (fp32) if asked for. ``x``
    and ``y1`` may have any strides: they are what autograd saved."""
    (N1, K), N2 = W1.shape, W2.shape[0]
    x, y1, dy = _f32_or_bf16(x).contiguous(), _f32_or_bf16(y1).contiguous(), dy.float().contiguous()
    B = x.shape[0]
    assert y1.shape == (B, N1) and dy.shape == (B, N2)
    dy1 = torch.empty((B, N1), dtype=torch.float32, device=x.device)
    dx = torch.empty((B, K), dtype=torch.float32, device=x.device) if need_dx else None
    rc = _l.lib().aeris_modulation_mlp_bwd(_l.ptr(W1), _gemv_flags(W1, None, x), _l.ptr(x), _l.ptr(dW1), _l.ptr(db1),
                                           _l.ptr(dx), N1, K, _l.ptr(W2), _gemv_flags(W2, None, y1), _l.ptr(y1), _l.ptr(dy),
                                           _l.ptr(dW2), _l.ptr(db2), _l.ptr(dy1), N2, B, _l.stream_ptr())
    _l.check(rc, "aeris_modulation_mlp_bwd", kernels=2)
    return dx


def gemv_bwd_ok(W: torch.Tensor, dW: torch.Tensor) -> bool:
    """Whether :func:`gemv_bwd` takes these operands: whole vectors of four along K, an fp32 gradient, and no more rows of
    W than the grid covers in its second dimension."""
    return (W.shape[1] % 4 == 0 and W.is_contiguous() and dW.is_contiguous() and dW.data_ptr() % 16 == 0
            and dW.dtype == torch.float32 and W.shape[0] <= 65535 * 16 and W.data_ptr() % (4 * W.element_size()) == 0
            and W.dtype in (torch.bfloat16, torch.float32))


def noise_embedding(t: torch.Tensor, dim: int, max_period: float, dtype: torch.dtype) -> torch.Tensor:
    """``[sin | cos]`` embedding [B, dim] of the noise levels ``t`` (fp32 [B]) in ``dtype`` (bf16 or fp32)."""
    out = torch.empty((t.shape[0], dim), dtype=dtype, device=t.device)
    rc = _l.lib().aeris_noise_embedding(_l.ptr(t), _l.ptr(out), int(dtype == torch.bfloat16), t.shape[0], dim,
                                        ctypes.c_double(max_period), _l.stream_ptr())
    _l.check(rc, "aeris_noise_embedding")
    return out


MAX_LEVELS = 64


def noise_embedding_of(levels: list[float], dim: int, max_period: float, dtype: torch.dtype, device) -> torch.Tensor:
    """:func:`noise_embedding` of levels that the host knows, without a copy to the device (which would wait)."""
    out = torch.empty((len(levels), dim), dtype=dtype, device=device)
    for i in range(0, len(levels), MAX_LEVELS):
        part = levels[i:i + MAX_LEVELS]
        rc = _l.lib().aeris_noise_embedding_of((ctypes.c_float * len(part))(*part), _l.ptr(out[i:]),
                                               int(dtype == torch.bfloat16), len(part), dim, ctypes.c_double(max_period),
                                               _l.stream_ptr())
        _l.check(rc, "aeris_noise_embedding_of")
    return out


def pack_embed_weights(W: torch.Tensor, b: torch.Tensor, KP: int) -> torch.Tensor:
    """``[hi(W) | hi(W) | lo(W) | hi(b) | lo(b) | 0..]`` (bf16 [D, KP]) of an fp32 weight [D, Cin] and bias."""
    D, Cin = W.shape
    out = torch.empty((D, KP), dtype=torch.bfloat16, device=W.device)
    rc = _l.lib().aeris_pack_embed_weights(_l.ptr(W), _l.ptr(b), _l.ptr(out), D, Cin, KP, _l.stream_ptr())
    _l.check(rc, "aeris_pack_embed_weights")
    return out


def fold_embed_grad(G: torch.Tensor, dW: torch.Tensor, db: torch.Tensor) -> None:
    """Adds the gradient ``G`` (fp32 [D, KP]) of the packed operand to ``dW`` [D, Cin] and ``db`` [D]."""
    D, Cin = dW.shape
    rc = _l.lib().aeris_fold_embed_grad(_l.ptr(G), _l.ptr(dW), _l.ptr(db), D, Cin, G.shape[1], _l.stream_ptr())
    _l.check(rc, "aeris_fold_embed_grad")


def pack_head_weights(W: torch.Tensor, rows: int) -> torch.Tensor:
    """``[hi | lo | hi]`` (bf16 [rows, 3 D]) of an fp32 weight [C, D], padded with zero rows."""
    C, D = W.shape
    out = torch.empty((rows, 3 * D), dtype=torch.bfloat16, device=W.device)
    rc = _l.lib().aeris_pack_head_weights(_l.ptr(W), _l.ptr(out), C, rows, D, _l.stream_ptr())
    _l.check(rc, "aeris_pack_head_weights")
    return out


def head_gemm(y: torch.Tensor, n: int, w: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """``out[:n]`` (fp32 [*, 128]) = the product of the values whose bf16 parts are ``y[0, :n]`` and ``y[1, :n]`` (``y``
    [2, rows, D]) with the weight packed by :func:`pack_head_weights`, up to the dropped lo x lo term."""
    assert y.is_contiguous() and y.dim() == 3 and w.shape == (128, 3 * y.shape[2])
    rc = _l.lib().aeris_gemm_split(_l.ptr(y), _l.ptr(w), _l.ptr(out), n, y.shape[2], y.shape[1], out.stride(0),
                                   _l.ptr(_l.status_word()), _l.stream_ptr())
    _l.check(rc, "aeris_gemm_split")
    return out
