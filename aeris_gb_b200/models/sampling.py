"""The network evaluations of one sampler run on one GPU, laid out together.

A sampler run evaluates the same weights a dozen times at noise levels that are known before the first one. Issued one by
one (:meth:`.aeris.AerisModel.predict_images`) an evaluation of a small model costs the host 460 us for 28 launches, more
than the GPU takes for them: the modulation vectors of every block, the packed weights of both ends, a dozen allocations,
views, checks and argument objects. None of it depends on the state, so :class:`Evaluations` does it once per run: all
levels' modulation vectors in one pass over the modulation weights, one argument record per block over three streams that
take turns, and per evaluation one native call for all blocks. Seven evaluations of two blocks of width 256 on 14,400
tokens: 3.29 -> 2.24 ms, issued in 1.5, where the GPU is the bound; wide models are bound by the GPU either way.
"""
from __future__ import annotations

import ctypes

import torch
from torch.nn.modules import module as _module

from ..ops import diffusion as DF
from ..ops import elementwise as E
from ..ops import lib as _l
from . import block as NB
from . import fused, fused_io


class _Refused(Exception):
    """A block that the native call does not take."""


def _hooked(modules) -> bool:
    """Whether a forward hook would miss a call of one of ``modules`` (where PyTorch does not say: yes)."""
    return bool(getattr(_module, "_global_forward_hooks", True) or getattr(_module, "_global_forward_pre_hooks", True)
                or any(m._forward_hooks or m._forward_pre_hooks for m in modules))


class Evaluations:
    """``run(e, x_img)`` is what ``predict_images(x_img, c_img, levels[e], ...)`` returns with every member at that noise
    level, bit for bit: the same kernels on the same values. A result is valid until the next evaluation in its ``slot``."""

    @classmethod
    def prepare(cls, model, c_img, levels: list[float], ctx, plan, slots: int, x_img) -> "Evaluations | None":
        """None where the evaluations have to go one by one: parallel ranks, objectives without a noise level or with a
        shared embedding, what the native call does not take, anything that watches or replaces a part of the model, and
        where all buffers at once do not fit."""
        from . import aeris as A
        cfg, grid, M, D = model.cfg, ctx.grid, plan.geom.B, model.cfg.dim
        if (not levels or not len(model.layers) or A.replaced(model, A.AerisModel)
                or A.replaced(model.input_stage, A.InputStage) or A.replaced(model.output_stage, A.OutputStage)
                or any(A.replaced(l, A.SwinLayer) for l in model.layers) or A.replaced(ctx, A.StreamContext)
                or _hooked(model.layers)
                or grid.n_ranks != 1 or ctx.peer_fn is not None or cfg.tp != 1 or ctx.batch != M
                or not (cfg.diffusion and cfg.conditioned and cfg.layerwise_t_emb) or cfg.model_dtype != torch.bfloat16
                or cfg.data_dtype != torch.float32 or D % 8 or not DF.gemv_ok(M, D) or fused.recorded()
                or not A.use_fused(x_img)):
            return None
        try:
            return cls(model, c_img, levels, ctx, plan, slots, x_img.device)
        except (torch.OutOfMemoryError, _Refused):
            return None

    def __init__(self, model, c_img, levels, ctx, plan, slots, dev):
        cfg, M, D, T = model.cfg, plan.geom.B, model.cfg.dim, plan.geom.rows
        self.model, self.c_img, self.plan, self.cfg = model, c_img, plan, cfg
        emb = DF.noise_embedding_of(levels, D, cfg.max_period, torch.bfloat16, dev)
        group = next(g for g in (8, 4, 2, 1) if DF.gemv_ok(g, D))
        groups = [emb[i:i + group] for i in range(0, len(levels), group)]

        def vectors(seq):
            parts = [fused.modulation(seq, g) for g in groups]
            return parts[0] if len(parts) == 1 else torch.cat(parts)

        self.head_mod = vectors(model.output_stage.modulation)
        proj, out = model.input_stage.proj, model.output_stage
        self.embed_w = DF.pack_embed_weights(proj.weight.float().contiguous(), proj.bias.float().contiguous(),
                                             fused_io._pack_dim(cfg.in_channels))
        self.head_w = fused_io._head_weights(out.head.weight)
        self.cs = torch.zeros((M, 2), device=dev)
        self.cs[:, 0] = 1.0
        # what an evaluation would otherwise ask for first when all else is already there
        fused_io.embed_workspace(cfg.in_channels, T, dev), fused_io.head_workspace(T, M, D, dev)
        self.pred = [torch.empty((T, fused_io.PAD_N), dtype=torch.float32, device=dev) for _ in range(slots)]
        self._lay_out_blocks(model, ctx, M, T, vectors, dev)

    def _lay_out_blocks(self, model, ctx, M, T, vectors, dev):
        """One argument record per block. ``self._alive``: every tensor that a record holds the address of."""
        cfg, D = self.cfg, self.cfg.dim
        HD = cfg.heads * cfg.head_dim
        after_mod_norm = cfg.after_mod_norm
        meta = fused.BlockMeta(ctx.grid.windows_per_rank, ctx.grid.n_local, cfg.heads, cfg.head_dim,
                               E.MODE_MOD_THEN_NORM if after_mod_norm else E.MODE_NORM_THEN_MOD, cfg.eps(torch.bfloat16),
                               cfg.chunk_windows, rope=ctx.rope(dev), min_chunk_bytes=cfg.min_chunk_bytes)
        step = fused.chunk_step(meta, D, cfg.mlp_dim)
        spans = fused._forward_spans(meta, M, step, D, cfg.mlp_dim, False)
        rows = max(nw for _, _, nw, _ in spans) * meta.L
        ws = fused.workspace()
        bufs = {k: ws.whole(k, *sh, dev) for k, sh in fused._chunk_shapes(rows, D, HD, cfg.heads, cfg.mlp_dim).items()
                if k != "h2"}
        bufs["h1"] = bufs["h2"] = bufs.pop("h")
        addr = {k: t.data_ptr() for k, t in bufs.items()}
        shifts = [cfg.layer_shift(i) for i in range(len(model.layers))] + [(0, 0)]
        moves = any(a != b for a, b in zip([(0, 0)] + shifts, shifts))
        self.streams = [torch.empty((T, D), dtype=torch.bfloat16, device=dev) for _ in range(3 if moves else 2)]
        self._alive = [bufs]
        records, cur, layout = [], 0, (0, 0)
        for layer, shift in zip(model.layers, shifts):
            for j, (n1, attn, n2, ff, mod) in enumerate(layer.blocks()):
                weights = (n1, attn.to_qkv.weight, attn.wo.weight, n2, ff.w1.weight, ff.w2.weight)
                m = vectors(mod.modulation)
                gather = j == 0 and shift != layout
                src, table = cur, ctx.table(layout, shift, dev) if gather else None
                if gather:
                    cur = (src + 1) % 3
                y = next(i for i in range(len(self.streams)) if i not in (src, cur))
                x, row = self.streams[cur], m[:1].expand(M, 6 * D)
                if not (NB.takes(meta, x, row, weights) and NB.fits(meta, x, row, weights, table=table)):
                    raise _Refused
                a, alive = NB._args(meta, x, m, M, D, cfg.mlp_dim, step, weights, addr, False, 0)
                a.merged, a.mod_sample, a.y = spans[0][3] > 1, 0, self.streams[y].data_ptr()
                if gather:
                    peers = E._peer_array([self.streams[src].data_ptr()])
                    a.table, a.peers, a.n_peers = table.data_ptr(), ctypes.addressof(peers), 1
                    alive = (*alive, table, peers)
                self._alive.append((weights, m, alive))
                records.append(a)
                cur = y
            layout = shift
        self.records = (NB.BlockArgs * len(records))(*records)
        self.last = self.streams[cur]
        self.back = ctx.table(layout, (0, 0), dev) if layout != (0, 0) else None

    def run(self, e: int, x_img: torch.Tensor, slot: int) -> torch.Tensor:
        proj, out, cfg = self.model.input_stage.proj, self.model.output_stage, self.cfg
        M, D = self.plan.geom.B, cfg.dim
        fused_io.embed(x_img, self.c_img, self.cs, proj.weight, proj.bias, self.plan, packed=self.embed_w,
                       out=self.streams[0])
        if E._CHECKED:
            E.set_gather_bounds(self.last.shape[0])
        NB.issue_forward(self.records, e * 6 * D)
        shift, scale = self.head_mod[e].view(2, 1, D).expand(2, M, D).unbind(0)
        return fused_io.head_forward(self.last, shift, scale, out.norm.weight, out.head.weight, cfg.eps(cfg.data_dtype),
                                     packed=self.head_w, pred=self.pred[slot], table=self.back)
