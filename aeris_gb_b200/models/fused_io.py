"""CUDA execution of the two ends of the network: noising + position encoding + input projection, and the fp32 output
head with the TrigFlow loss.

Both ends are fp32 in the reference (src/aeris/models/parallel_swin.py:383-386 and :519-529, the loss at
src/aeris/parallelism/parallel_engine.py:990-997). Here their contractions run on the bf16 tensor cores at fp32-level
accuracy by splitting each fp32 operand into a bf16 value and a bf16 remainder and summing the three significant
products (hi*hi + lo*hi + hi*lo); the rest (noise, mixing, position encoding, window partition, norm, modulation,
loss and its gradient) lives in the element-wise kernels around them, so the fp32 model input, the noise and the
prediction error never exist in memory as full-size tensors.
"""
from __future__ import annotations

from dataclasses import dataclass

import torch

from ..ops import diffusion as DF
from ..ops import elementwise as E
from ..ops import gemm as G
from . import oracle as O
from .fused import workspace

PAD_N = 128          # output channels are padded to one GEMM tile
CHUNK_ROWS = 1 << 16


@dataclass
class IoPlan:
    """What the fused input/output ends need to know about one training or sampling call."""
    geom: DF.TokGeom
    sigma_data: float
    seed: int = 0
    noise: bool = True
    ape_y: torch.Tensor | None = None     # [H (+offset applied), ch] fp32
    ape_x: torch.Tensor | None = None     # [W, ch] fp32
    w_var: torch.Tensor | None = None     # [C_out] fp32
    w_lat: torch.Tensor | None = None     # [H] fp32 (global image rows)
    eps: float = 1.1920929e-07


def ape_tables(cfg, device) -> tuple[torch.Tensor, torch.Tensor]:
    off = cfg.ape_row_offset if cfg.ape_row_offset is not None else (1 if cfg.img[0] == 720 else 0)
    ty, tx = O.positional_tables(cfg.in_channels, cfg.img[0] + off, cfg.img[1])
    return ty[off:].contiguous().to(device), tx.contiguous().to(device)


def _grad_slot(p: torch.Tensor):
    """fp32 accumulation target of a parameter: the engine's ``main_grad`` view, or a fresh buffer handed back to
    autograd."""
    mg = getattr(p, "main_grad", None)
    if mg is not None:
        return (mg.view(p.shape) if mg.shape != p.shape else mg), None
    z = torch.zeros(p.shape, dtype=torch.float32, device=p.device)
    return z, z


def _kernel_target(slot: torch.Tensor) -> torch.Tensor:
    """Where a kernel may add fp32 gradients by address: the slot itself, or zeros for :func:`_settle` to add to it when
    somebody's ``main_grad`` has another type or layout."""
    if slot.dtype == torch.float32 and slot.is_contiguous():
        return slot
    return torch.zeros(slot.shape, dtype=torch.float32, device=slot.device)


def _settle(slot: torch.Tensor, target: torch.Tensor) -> None:
    if target is not slot:
        slot += target


def _pack_dim(c_in: int) -> int:
    return (3 * c_in + 2 + 127) // 128 * 128


def embed_workspace(c_in: int, T: int, dev) -> torch.Tensor:
    return workspace().get("embed_a", (min(CHUNK_ROWS, T), _pack_dim(c_in)), torch.bfloat16, dev)


def head_workspace(T: int, B: int, D: int, dev) -> torch.Tensor:
    """The bf16 value and remainder of the normalised rows of one pass over the head."""
    rows = max(n for *_, n in _sample_chunks(B, T // B))
    return workspace().get("head_y", (2, rows, D), torch.bfloat16, dev)


def embed(x_img, c_img, cs, W, b, plan: IoPlan, packed: torch.Tensor | None = None,
          out: torch.Tensor | None = None) -> torch.Tensor:
    """``(cat[(cos t x + sin t z) / sigma_d, cond] + ape) W^T + b`` -> bf16 token stream in the unshifted window layout.
    ``packed``: :func:`.diffusion.pack_embed_weights` of W and b, from callers with several evaluations to run."""
    D, Cin = W.shape
    KP = _pack_dim(Cin)
    dev = x_img.device
    Wp = packed if packed is not None else \
        DF.pack_embed_weights(W.detach().float().contiguous(), b.detach().float().contiguous(), KP)
    T = plan.geom.rows
    out = out if out is not None else torch.empty((T, D), dtype=torch.bfloat16, device=dev)
    A = embed_workspace(Cin, T, dev)
    for r0 in range(0, T, CHUNK_ROWS):
        n = min(CHUNK_ROWS, T - r0)
        DF.embed_pack(x_img, c_img, cs, plan.geom, plan.ape_y, plan.ape_x, plan.seed, plan.sigma_data,
                      plan.noise, A[:n], row0=r0)
        G.gemm(A[:n], Wp, out=out[r0:r0 + n])
    return out


class EmbedFn(torch.autograd.Function):
    """:func:`embed` with the gradients of the weight and the bias."""

    @staticmethod
    def forward(ctx, x_img, c_img, cs, W, b, plan: IoPlan):
        ctx.plan = plan
        ctx.save_for_backward(x_img, c_img, cs, W, b)
        return embed(x_img, c_img, cs, W, b, plan)

    @staticmethod
    def backward(ctx, dout):
        x_img, c_img, cs, W, b = ctx.saved_tensors
        plan = ctx.plan
        D, Cin = W.shape
        KP = _pack_dim(Cin)
        dev = dout.device
        dout = dout.contiguous()
        T = plan.geom.rows
        A = workspace().get("embed_a", (min(CHUNK_ROWS, T), KP), torch.bfloat16, dev)
        Gw = workspace().get("embed_g", (D, KP), torch.float32, dev, zero=True)
        for r0 in range(0, T, CHUNK_ROWS):
            n = min(CHUNK_ROWS, T - r0)
            DF.embed_pack(x_img, c_img, cs, plan.geom, plan.ape_y, plan.ape_x, plan.seed, plan.sigma_data,
                          plan.noise, A[:n], row0=r0)
            G.gemm(dout[r0:r0 + n], A[:n], a_t=True, b_t=True, out=Gw, epi=G.EPI_ACC_F32, k_splits=8)
        sW, rW = _grad_slot(W)
        sb, rb = _grad_slot(b)
        tW, tb = _kernel_target(sW), _kernel_target(sb)
        DF.fold_embed_grad(Gw, tW, tb)
        _settle(sW, tW)
        _settle(sb, tb)
        return (None, None, None, rW.to(W.dtype) if rW is not None else None,
                rb.to(b.dtype) if rb is not None else None, None)


def _head_weights(head_w: torch.Tensor):
    return DF.pack_head_weights(head_w.detach().float().contiguous(), PAD_N)


def _head_rows(x, scale, shift, norm_w, w3, eps, pred, y, table=None):
    """pred[n, 128] (fp32) = (RMSNorm(x) * w * (1 + scale) + shift) @ head^T for ``n`` rows of ``scale.shape[0]`` samples;
    ``y`` [2, rows, D]: workspace for the bf16 value and remainder of the normalised rows. ``table`` (``n`` codes): where
    in ``x`` those rows are."""
    n, D = x.shape[0] if table is None else table.shape[0], x.shape[1]
    where = {} if table is None else dict(gather_idx=table, peer_ptrs=[x.data_ptr()], src_rows=x.shape[0])
    E.modnorm_fwd(x if table is None else None, scale, shift, norm_w, mode=E.MODE_NORM_THEN_MOD, eps=eps, out=y[0, :n],
                  out_lo=y[1, :n], batch=scale.shape[0], **where)
    if D % 64 == 0:
        DF.head_gemm(y, n, w3, pred)
    else:                                  # the packed product's three sections consist of whole k-blocks
        w_hi, w_lo = w3[:, :D], w3[:, D:2 * D]
        G.gemm(y[1, :n], w_hi, out=pred[:n], epi=G.EPI_STORE_F32)
        G.gemm(y[0, :n], w_lo, out=pred[:n], epi=G.EPI_ACC_F32)
        G.gemm(y[0, :n], w_hi, out=pred[:n], epi=G.EPI_ACC_F32)
    return pred[:n]


def _mod_rows(shift: torch.Tensor, scale: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """fp32 ``shift`` and ``scale`` [B, D] as the kernels read them: where they are (halves of one tensor) if their rows are
    whole 16-byte vectors at the same pitch."""
    shift, scale = shift.float(), scale.float()
    if (shift.stride() == scale.stride() and shift.stride(1) == 1 and shift.stride(0) % 4 == 0
            and shift.data_ptr() % 16 == 0 and scale.data_ptr() % 16 == 0):
        return shift, scale
    return shift.contiguous(), scale.contiguous()


def _sample_chunks(B: int, rows_per_sample: int) -> list[tuple[int, int, int, int]]:
    """(first sample, samples, first row, rows) of every pass over the head: all samples at once where they fit one
    chunk, else chunks of one sample."""
    if B * rows_per_sample <= CHUNK_ROWS:
        return [(0, B, 0, B * rows_per_sample)]
    return [(b, 1, b * rows_per_sample + r, min(CHUNK_ROWS, rows_per_sample - r))
            for b in range(B) for r in range(0, rows_per_sample, CHUNK_ROWS)]


def head_forward(x: torch.Tensor, shift: torch.Tensor, scale: torch.Tensor, norm_w: torch.Tensor,
                 head_w: torch.Tensor, eps: float, packed: torch.Tensor | None = None,
                 pred: torch.Tensor | None = None, table: torch.Tensor | None = None) -> torch.Tensor:
    """Network output ``F`` in token order, fp32 ``[T, 128]`` (columns past the channel count are zero). ``packed``:
    :func:`_head_weights` of ``head_w``. ``table``: the gather codes of a stream in a shifted window layout, whose rows the
    norm then reads from where they are (1,036,800 rows of 1536: no pass of 6.4 GB before it, 1.1 ms)."""
    T, D = x.shape
    B = shift.shape[0]
    dev = x.device
    w3 = packed if packed is not None else _head_weights(head_w)
    spans = _sample_chunks(B, T // B)
    y = head_workspace(T, B, D, dev)
    pred = pred if pred is not None else torch.empty((T, PAD_N), dtype=torch.float32, device=dev)
    shift, scale = _mod_rows(shift, scale)
    for b, nb, r0, n in spans:
        rows, codes = (x[r0:r0 + n], None) if table is None else (x, table[r0:r0 + n])
        _head_rows(rows, scale[b:b + nb], shift[b:b + nb], norm_w, w3, eps, pred[r0:r0 + n], y, codes)
    return pred


class HeadLossFn(torch.autograd.Function):
    """Output head + TrigFlow loss: returns ``sum_b mean_rows sum_c w_lat w_var (sigma_d F - v_t)^2`` as a scalar.
    Forward keeps the stream input and d loss / d F (bf16, 128 columns per row); backward recomputes the normalised
    rows chunk by chunk."""

    @staticmethod
    def forward(ctx, x, shift, scale, norm_w, head_w, x_img, cs, plan: IoPlan):
        T, D = x.shape
        B = shift.shape[0]
        dev = x.device
        w3 = _head_weights(head_w)
        ws = workspace()
        spans = _sample_chunks(B, T // B)
        cm = max(n for *_, n in spans)
        y = ws.get("head_y", (2, cm, D), torch.bfloat16, dev)
        pred = ws.get("head_pred", (cm, PAD_N), torch.float32, dev)
        dpred = torch.empty((T, PAD_N), dtype=torch.bfloat16, device=dev)
        loss = torch.zeros(1, dtype=torch.float64, device=dev)
        shift32, scale32 = _mod_rows(shift, scale)
        inv_rows = 1.0 / (T // B)
        for b, nb, r0, n in spans:
            _head_rows(x[r0:r0 + n], scale32[b:b + nb], shift32[b:b + nb], norm_w, w3, plan.eps, pred, y)
            DF.trigflow_loss(pred[:n], x_img, cs, plan.geom, plan.seed, plan.sigma_data, plan.w_var, plan.w_lat,
                             inv_rows, loss, dpred=dpred[r0:r0 + n], row0=r0)
        ctx.plan = plan
        ctx.save_for_backward(x, shift, scale, norm_w, head_w, dpred)
        return loss.float().squeeze(0)

    @staticmethod
    def backward(ctx, g):
        x, shift, scale, norm_w, head_w, dpred = ctx.saved_tensors
        plan = ctx.plan
        T, D = x.shape
        B = shift.shape[0]
        C = head_w.shape[0]
        dev = x.device
        w_hi = _head_weights(head_w)[:, :D]
        ws = workspace()
        spans = _sample_chunks(B, T // B)
        cm = max(n for *_, n in spans)
        y_hi, dy = ws.get("head_y", (2, cm, D), torch.bfloat16, dev).unbind(0)
        Gh = ws.get("head_g", (PAD_N, D), torch.float32, dev, zero=True)
        shift32, scale32 = _mod_rows(shift, scale)
        dshift, dscale = torch.zeros((2, *shift32.shape), dtype=torch.float32, device=dev).unbind(0)
        s_nw, r_nw = _grad_slot(norm_w)
        t_nw = _kernel_target(s_nw)
        dx = torch.empty_like(x)
        dpred = dpred * g.to(dpred.dtype)
        for b, nb, r0, n in spans:
            E.modnorm_fwd(x[r0:r0 + n], scale32[b:b + nb], shift32[b:b + nb], norm_w, mode=E.MODE_NORM_THEN_MOD,
                          eps=plan.eps, out=y_hi[:n], batch=nb)
            dp = dpred[r0:r0 + n]
            G.gemm(dp, y_hi[:n], a_t=True, b_t=True, out=Gh, epi=G.EPI_ACC_F32, k_splits=16 * nb, two_cta=False)
            G.gemm(dp, w_hi, b_t=True, out=dy[:n])
            m = n // nb
            for i in range(nb):        # column sums per sample
                sl = slice(r0 + i * m, r0 + (i + 1) * m)
                E.modnorm_bwd(x[sl], dy[i * m:(i + 1) * m], None, scale32[b + i], shift32[b + i], norm_w,
                              mode=E.MODE_NORM_THEN_MOD, eps=plan.eps, dx=dx[sl], dscale=dscale[b + i],
                              dshift=dshift[b + i], dw=t_nw)
        _settle(s_nw, t_nw)
        s_hw, r_hw = _grad_slot(head_w)
        s_hw += Gh[:C]
        return (dx, dshift.to(shift.dtype), dscale.to(scale.dtype), r_nw.to(norm_w.dtype) if r_nw is not None else None,
                r_hw.to(head_w.dtype) if r_hw is not None else None, None, None, None)
