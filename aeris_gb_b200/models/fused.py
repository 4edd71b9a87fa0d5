"""CUDA execution of one Swin-TrigFlow block (forward and hand-derived backward) on the sm_100a kernels.

The block is processed in *chunks of whole windows* of one sample: inside a block every token only interacts with its
own window, so a chunk runs modulate+RMSNorm -> QKV GEMM -> window attention -> (wo GEMM + gated residual) ->
modulate+RMSNorm -> (w1 GEMM + SwiGLU) -> (w2 GEMM + gated residual) with a working set of a few GB no matter how
large the image is. Training keeps a block's internals where memory allows (:func:`plan_kept_blocks`) and only the block
input elsewhere (activation checkpointing, absent from the reference and mandatory for one million tokens per sample);
the backward pass then recomputes a chunk's internals and immediately back-propagates through them, accumulating weight
gradients in fp32 directly from the GEMM epilogue.

Math restated from src/aeris/models/parallel_swin.py:453-472 (block), :82-104 (SwiGLU), :261-308 (attention).
"""
from __future__ import annotations

import math
from dataclasses import dataclass
from types import SimpleNamespace

import torch
from torch.autograd import forward_ad

from ..ops import attention as A
from ..ops import elementwise as E
from ..ops import gemm as G
from . import block as NB


@dataclass
class BlockMeta:
    n_win_per_sample: int      # windows of one sample held by this rank
    L: int                     # tokens per window
    heads: int
    head_dim: int
    mode: int                  # E.MODE_MOD_THEN_NORM or E.MODE_NORM_THEN_MOD
    eps: float
    chunk_windows: int = 64
    sp: "SPExchange | None" = None     # Ulysses sequence parallelism: L is then the LOCAL token count of a window
    rope: tuple | None = None          # (cos, sin) [L, head_dim / 2]: optional 2-D rotary embedding of q and k
    tp: object | None = None           # parallel.tensor.TPExchange: w1 / w2 are this rank's shards of the MLP weights
    keep: bool = False                 # forward keeps its internals for the backward pass (see plan_kept_blocks)
    min_chunk_bytes: int | None = None  # chunks with fewer bytes of internals are merged; None: MIN_CHUNK_BYTES

    @property
    def chunk_floor(self) -> int:
        return MIN_CHUNK_BYTES if self.min_chunk_bytes is None else self.min_chunk_bytes


class Workspace:
    """Named scratch tensors, allocated once at the largest size asked for and reused by every block."""

    def __init__(self):
        self._buf: dict[str, torch.Tensor] = {}

    def whole(self, name: str, shape: tuple[int, ...], dtype: torch.dtype, device) -> torch.Tensor:
        """The buffer behind :meth:`get`, without the view of ``shape``: for callers that only pass its address on.
        0.6 us of host time against 3.8, and a block asks for seven buffers forward and ten backward."""
        n = math.prod(shape)
        b = self._buf.get(name)
        if b is None or b.numel() < n or b.dtype != dtype or b.device != torch.device(device):
            b = torch.empty(n, dtype=dtype, device=device)
            self._buf[name] = b
        return b

    def get(self, name: str, shape: tuple[int, ...], dtype: torch.dtype, device, zero: bool = False) -> torch.Tensor:
        v = self.whole(name, shape, dtype, device)[:math.prod(shape)].view(*shape)
        if zero:
            v.zero_()
        return v

    def missing(self, shapes: dict[str, tuple[tuple[int, ...], torch.dtype]], device) -> int:
        """Bytes of the buffers that asking for ``shapes`` would allocate."""
        total = 0
        for name, (shape, dtype) in shapes.items():
            b, n = self._buf.get(name), math.prod(shape)
            if b is None or b.numel() < n or b.dtype != dtype or b.device != torch.device(device):
                total += n * dtype.itemsize
        return total

    def clear(self):
        self._buf.clear()


_WS = Workspace()


def workspace() -> Workspace:
    return _WS


class SPExchange:
    """Symmetric buffers and rank barrier of one Ulysses sequence-parallel group.

    The exchanges of src/aeris/parallelism/sequence_parallel.py:40-86 (three all-to-alls before and one after every
    attention, and their mirrors in backward) do not exist as separate operations here: the QKV GEMM's epilogue stores
    each head's tile into the buffer of the rank that owns the head, and the attention kernels store their output
    (forward) and dQ/dK/dV (backward) into the buffers of the ranks that own the tokens. What is left of the
    collective is a flag barrier between producer and consumer kernels.
    """

    def __init__(self, group, device, timeout_s: float = 20.0):
        import torch.distributed as dist
        from ..engine.fused_dp import RankBarrier
        self.group, self.device = group, torch.device(device)
        self.sp, self.rank = dist.get_world_size(group), dist.get_rank(group)
        self.barrier = RankBarrier(group, self.device, timeout_s)
        self._bufs: dict[str, tuple] = {}

    def buffer(self, name: str, shape: tuple[int, int]) -> tuple[torch.Tensor, list[int]]:
        """Symmetric bf16 buffer of at least ``shape`` (every rank must ask for the same sizes in the same order)."""
        import torch.distributed._symmetric_memory as symm_mem
        n = shape[0] * shape[1]
        ent = self._bufs.get(name)
        if ent is None or ent[0].numel() < n:
            t = symm_mem.empty(n, dtype=torch.bfloat16, device=self.device)
            hdl = symm_mem.rendezvous(t, self.group)
            ent = (t, [int(x) for x in hdl.buffer_ptrs], hdl)
            self._bufs[name] = ent
        return ent[0][:n].view(*shape), ent[1]


def _scatter_heads(a: torch.Tensor, w: torch.Tensor, sp: "SPExchange", peers: list[int], n_local: int, L: int,
                   sec_w: int, b_t: bool = False):
    """``a @ w^T`` (or ``a @ w`` with ``b_t``) whose head tiles go to their owner ranks (GEMM-epilogue Ulysses)."""
    import ctypes
    from ..ops import lib as _l
    M, K = a.shape
    N = w.shape[1] if b_t else w.shape[0]
    arr = (ctypes.c_void_p * len(peers))(*peers)
    rc = _l.lib().aeris_gemm_scatter_heads(_l.ptr(a), _l.ptr(w), M, N, K, a.stride(0), w.stride(0), int(b_t), arr,
                                           sp.sp, sp.rank, n_local, L, sec_w, _l.ptr(_l.status_word()),
                                           _l.stream_ptr())
    _l.check(rc, "aeris_gemm_scatter_heads")


def _rope_qk_(qkv: torch.Tensor, meta: BlockMeta, nw: int, inverse: bool = False) -> None:
    """Rotates the q and k sections of a chunk's fused qkv tensor in place (``rope_qk_kernel``; ``inverse`` turns
    gradients with respect to the rotated q, k into gradients with respect to the projections)."""
    assert meta.sp is None, "the rotary embedding is not combined with sequence parallelism"
    cos, sin = meta.rope
    E.rope_qk_(qkv, cos.float().contiguous(), sin.float().contiguous(), meta.L, meta.heads, meta.head_dim, inverse)


KEPT = ("h1", "qkv", "o", "lse", "x1", "h2", "act", "u")


def _kept_shapes(T: int, D: int, HD: int, heads: int, F: int) -> dict[str, tuple[tuple[int, ...], torch.dtype]]:
    """What a block keeps for its backward pass: every internal the recompute would produce again."""
    bf = torch.bfloat16
    return {"h1": ((T, D), bf), "qkv": ((T, 3 * HD), bf), "o": ((T, HD), bf), "lse": ((T * heads,), torch.float32),
            "x1": ((T, D), bf), "h2": ((T, D), bf), "act": ((T, F), bf), "u": ((T, 2 * F), bf)}


class FreshKept(dict):
    """Internals' buffers as :class:`FusedBlock` allocates them for one forward pass: nothing about them needs a check."""


def _all_whole(kept: dict[str, torch.Tensor], T: int, D: int, HD: int, heads: int, F: int, device: int) -> bool:
    """Whether kernels may take all of ``kept`` (:func:`_kept_shapes`) by address. Every backward pass asks."""
    td, th, tf = T * D, T * HD, T * F
    for k, n in (("h1", td), ("qkv", 3 * th), ("o", th), ("x1", td), ("h2", td), ("act", tf), ("u", 2 * tf),
                 ("lse", T * heads)):
        t = kept[k]
        if not (t.is_contiguous() and t.numel() == n and t.dtype is (torch.float32 if k == "lse" else torch.bfloat16)
                and t.get_device() == device and t.data_ptr() % 16 == 0):
            return False
    return True


def _whole_kept(kept: dict[str, torch.Tensor], shapes, device) -> dict[str, torch.Tensor]:
    """``kept`` for kernels where :func:`_all_whole` says no: a saved-tensor hook may have handed back other strides or an
    odd start (copied) or something else altogether (refused). ``shapes``: see :func:`_kept_shapes`."""
    out = {}
    for k, (shape, dt) in shapes.items():
        t = kept[k]
        if t.shape != shape or t.dtype != dt or t.device != device:
            raise ValueError(f"kept {k}: {tuple(t.shape)} {t.dtype} on {t.device}, not {shape} {dt} on {device}")
        whole = t.is_contiguous() and t.data_ptr() % 16 == 0
        out[k] = t if whole else t.clone(memory_format=torch.contiguous_format)
    return out


def kept_bytes(T: int, D: int, HD: int, heads: int, F: int) -> int:
    """Bytes of :func:`_kept_shapes`, in closed form: every pass over a block asks for them."""
    return T * (2 * (3 * D + 4 * HD + 3 * F) + 4 * heads)


def _chunk_shapes(rows: int, D: int, HD: int, heads: int, F: int, tpn: int = 1):
    """Chunk workspaces of a forward pass that keeps nothing, and of the recompute (``h2`` in the forward pass is ``h``).
    ``tpn``: ranks whose rows a tensor-parallel MLP gathers."""
    bf = torch.bfloat16
    return {"h": ((rows, D), bf), "qkv": ((rows, 3 * HD), bf), "o": ((rows, HD), bf),
            "lse": ((rows * heads,), torch.float32), "x1": ((rows, D), bf), "h2": ((rows, D), bf),
            "act": ((rows * tpn, F), bf)}


def _grad_shapes(rows: int, D: int, HD: int, heads: int, F: int, tpn: int = 1):
    """Workspaces of every backward pass: a chunk's gradients, the gated weights, one sample's ungated weight gradients."""
    bf, f32 = torch.bfloat16, torch.float32
    return {"u": ((rows * tpn, 2 * F), bf), "dh": ((rows, D), bf), "dx1": ((rows, D), bf), "d_o": ((rows, HD), bf),
            "dqkv": ((rows, 3 * HD), bf), "delta": ((rows * heads,), f32), "w2g": ((D, F), bf), "wog": ((D, HD), bf),
            "G2": ((D, F), f32), "Go": ((D, HD), f32)}


def n_kept(n_blocks: int, per_block: int, base: int, free: int) -> int:
    """How many of ``n_blocks`` blocks may keep their internals: these take at most half of what is left of ``free``
    after the ``base`` bytes that the step needs in any case."""
    return max(0, min(n_blocks, (free - base) // 2 // per_block))


def plan_kept_blocks(meta: BlockMeta, batch: int, D: int, F: int, n_blocks: int, device) -> int:
    """How many blocks of a training forward keep their internals instead of recomputing them in the backward pass.

    The recompute is a quarter of a step's tensor-core work (one more QKV, wo and w1 product and attention forward per
    block) and under the power cap time follows work, so it is only worth its price where memory is short: a full-size
    image (1 M tokens x 40 blocks) needs it, one with a few GB of internals on a 180 GB GPU does not. The kept internals
    take at most half of the memory that is free now (the allocator's unused cache included) and not needed by the step
    in any case: block inputs, stream gradients, and the workspaces that are not there yet.

    One exception saves a question to the driver (0.1 to 2 ms each, measured; a fifth of a small step): where the allocator's
    cache by itself covers the internals of all blocks and the rest of the step, as it does from the second step on, all
    blocks keep theirs. Fragments (unused parts of blocks in use) count there, because an earlier step's tensors lie in
    them; where they turn out too small for a block's internals, :class:`FusedBlock` lets that block recompute. Elsewhere
    they do not count as free."""
    HD = meta.heads * meta.head_dim
    T = batch * meta.n_win_per_sample * meta.L
    per_block = kept_bytes(T, D, HD, meta.heads, F)
    step = chunk_step(meta, D, F)
    rows = step * meta.L
    fwd_rows = max(nw for _, _, nw, _ in _forward_spans(meta, batch, step, D, F, False)) * meta.L
    # at the peak: every block's input, the gradient of the last one's output, and what a shifted layer hands back
    stream = T * D * 2
    grads = _WS.missing(_grad_shapes(rows, D, HD, meta.heads, F), device)
    stats = torch.cuda.memory_stats_as_nested_dict(device)
    reserved, allocated, fragments = (stats.get(k, {}).get("all", {}).get("current", 0)
                                      for k in ("reserved_bytes", "allocated_bytes", "inactive_split_bytes"))
    if n_blocks * per_block + (n_blocks + 2) * stream + grads <= reserved - allocated:
        return n_blocks
    # a margin of two streams, and the workspaces of the blocks that recompute
    base = (n_blocks + 4) * stream + grads + _WS.missing(_chunk_shapes(fwd_rows, D, HD, meta.heads, F), device)
    free = max(0, reserved - allocated - fragments) + torch.cuda.mem_get_info(device)[0]
    return n_kept(n_blocks, per_block, base, free)


MIN_CHUNK_BYTES = 512 << 20
MAX_CHUNK_WINDOWS = 65535      # the attention kernels' grid has one layer per window


def chunk_step(meta: BlockMeta, D: int, F: int) -> int:
    """Windows per chunk: ``meta.chunk_windows`` bounds the working set, but a chunk whose internals take less than half a
    gigabyte saves no memory worth having and costs launches that the GPU finishes faster than they are issued (32
    windows of 64 tokens at dim 128 in chunks of 8: 1,582 launches per step for 7 ms of device time). With
    ``min_chunk_bytes = 0`` the bound is ``chunk_windows`` itself."""
    floor = meta.chunk_floor // (kept_bytes(1, D, meta.heads * meta.head_dim, meta.heads, F) * meta.L)
    step = min(max(meta.chunk_windows, floor), meta.n_win_per_sample, MAX_CHUNK_WINDOWS)
    if step < 1:
        raise ValueError(f"chunks of {step} windows: chunk_windows {meta.chunk_windows} with min_chunk_bytes "
                         f"{meta.chunk_floor}, {meta.n_win_per_sample} windows per sample")
    return step


def wanted_slices(meta: BlockMeta, nw: int) -> int:
    """Slices that the weight gradients of a chunk of ``nw`` windows should keep of the shorter sums: four per chunk of
    ``chunk_windows``, which may be 0 where the floor of :func:`chunk_step` alone sets the chunk."""
    return 4 * -(-nw // max(1, min(meta.chunk_windows, meta.n_win_per_sample)))


def _forward_spans(meta: BlockMeta, B: int, step: int, D: int, F: int, kept: bool) -> list[tuple[int, int, int, int]]:
    """What one pass over the forward kernels covers: (first sample, first window, windows, samples). Samples that are one
    chunk each run in one launch per kernel (their modulation vectors are picked by row), when their internals are kept
    anyway or take less than the smallest chunk; the exchanges of the parallel paths work on one sample at a time."""
    if (B > 1 and step == meta.n_win_per_sample and meta.sp is None and meta.tp is None
            and (kept or kept_bytes(B * step * meta.L, D, meta.heads * meta.head_dim, meta.heads, F) <= meta.chunk_floor)
            and B * step <= MAX_CHUNK_WINDOWS):
        return [(0, 0, B * step, B)]
    return [(b, w0, nw, 1) for b in range(B) for w0, nw in _chunks(meta, step)]


def _chunks(meta: BlockMeta, step: int):
    for w0 in range(0, meta.n_win_per_sample, step):
        yield w0, min(step, meta.n_win_per_sample - w0)


def _sp_attention_fwd(meta: BlockMeta, h: torch.Tensor, wqkv: torch.Tensor, nw: int, keep_local: bool):
    """Sequence-parallel attention of one chunk. ``h`` [nw * n_local, D] -> o [nw * n_local, heads * d] (tokens of this
    rank, all heads). Returns (o, state for the backward pass)."""
    import ctypes
    from ..ops import lib as _l
    sp = meta.sp
    n_local, L = meta.L, meta.L * sp.sp
    hl, d = meta.heads // sp.sp, meta.head_dim
    HD = meta.heads * d
    n, nf = nw * n_local, nw * L
    qkv_full, qkv_peers = sp.buffer("qkv_full", (nf, 3 * hl * d))
    o_loc, o_peers = sp.buffer("o_loc", (n, HD))
    _scatter_heads(h, wqkv, sp, qkv_peers, n_local, L, HD)
    sp.barrier()                                  # every rank's q/k/v tiles for my heads have landed
    o_full = _WS.get("sp_o_full", (nf, hl * d), torch.bfloat16, h.device) if keep_local else None
    lse = _WS.get("sp_lse", (nw, hl, L), torch.float32, h.device)
    arr = (ctypes.c_void_p * sp.sp)(*o_peers)
    rc = _l.lib().aeris_attn_fwd_push(_l.ptr(qkv_full), qkv_full.stride(0), hl, _l.ptr(o_full),
                                      o_full.stride(0) if o_full is not None else 0, _l.ptr(lse), nw, L, d,
                                      _l._c_float(1.0 / d ** 0.5), arr, sp.sp, n_local, HD, sp.rank * hl * d,
                                      _l.ptr(_l.status_word()), _l.stream_ptr())
    _l.check(rc, "aeris_attn_fwd_push")
    sp.barrier()                                  # every rank's output rows for my tokens have landed
    return o_loc, (qkv_full, o_full, lse)


def _sp_attention_bwd(meta: BlockMeta, dx1: torch.Tensor, wog: torch.Tensor, nw: int, state):
    """Backward of :func:`_sp_attention_fwd` up to d(qkv) for this rank's tokens [nw * n_local, 3 * heads * d]."""
    import ctypes
    from ..ops import lib as _l
    sp = meta.sp
    qkv_full, o_full, lse = state
    n_local, L = meta.L, meta.L * sp.sp
    hl, d = meta.heads // sp.sp, meta.head_dim
    HD = meta.heads * d
    n, nf = nw * n_local, nw * L
    do_full, do_peers = sp.buffer("do_full", (nf, hl * d))
    dqkv_loc, dq_peers = sp.buffer("dqkv_loc", (n, 3 * HD))
    _scatter_heads(dx1, wog, sp, do_peers, n_local, L, HD, b_t=True)     # d(o) = (dx1 * g1) @ wo, pushed by head
    sp.barrier()
    delta = _WS.get("sp_delta", (nw, hl, L), torch.float32, dx1.device)
    arr = (ctypes.c_void_p * sp.sp)(*dq_peers)
    rc = _l.lib().aeris_attn_bwd_push(_l.ptr(qkv_full), qkv_full.stride(0), hl, _l.ptr(o_full), _l.ptr(do_full),
                                      o_full.stride(0), _l.ptr(lse), _l.ptr(delta), nw, L, d,
                                      _l._c_float(1.0 / d ** 0.5), arr, sp.sp, n_local, 3 * HD, HD, sp.rank * hl * d,
                                      _l.ptr(_l.status_word()), _l.stream_ptr())
    _l.check(rc, "aeris_attn_bwd_push", kernels=2)
    sp.barrier()
    return dqkv_loc


def _tp_mlp_fwd(tp, x1, sc2, sh2, wn2, meta: BlockMeta, w1, w2, g2, act, y_out):
    """Tensor-parallel MLP half of a chunk: ``y = x1 + g2 * reduce_scatter(swiglu(all_gather(h2) @ w1_r^T) @ w2_r^T)``
    with both collectives inside the GEMM kernels (parallel/tensor.py). The modulate+norm kernel writes this rank's
    rows of h2 straight into the all-gather buffer; the barrier inside the reduce-scatter orders a chunk's reads
    before the next chunk's pushes."""
    from ..parallel import tensor as TP
    n, D = x1.shape
    M = tp.tp * n
    a_buf, peers = tp.buffer("ag_x", (M, D))
    E.modnorm_fwd(x1, sc2, sh2, wn2, mode=meta.mode, eps=meta.eps, out=a_buf[tp.rank * n:(tp.rank + 1) * n])
    tp.barrier()
    TP.gemm_allgather_a(tp, a_buf, peers, w1, out=act[:M], epi=G.EPI_SWIGLU)
    TP.gemm_reduce_scatter(tp, act[:M], w2, resid=x1, gate=g2, out=y_out)


def _chunk_views(bufs: dict[str, torch.Tensor], r0: int, n: int, heads: int):
    """Rows ``[r0, r0 + n)`` of h1, qkv, o, x1, h2, act and the matching slice of lse (whole windows: rows x heads)."""
    return (*(bufs[k][r0:r0 + n] for k in ("h1", "qkv", "o", "x1", "h2", "act")), bufs["lse"][r0 * heads:(r0 + n) * heads])


def block_forward(x: torch.Tensor, mod: torch.Tensor, meta: BlockMeta, wn1, wqkv, wo, wn2, w1, w2,
                  out: torch.Tensor | None = None, gather=None,
                  kept: dict[str, torch.Tensor] | None = None) -> torch.Tensor:
    """x: [B * n_win * L, D] bf16 window-major; mod: [B, 6D] fp32 (shift1, scale1, gate1, shift2, scale2, gate2).

    ``gather = (table, peer_ptrs, src)``: ``x`` is then an EMPTY buffer in this block's window layout; the first
    modulate+norm kernel of every chunk pulls its rows through the table from ``src`` on this or a peer GPU (the
    re-partition / halo exchange of a shifted layer) and writes them into ``x`` on the way.

    ``kept``: full-size buffers (:func:`_kept_shapes`) that receive the block's internals; without it they live in chunk
    workspaces and are gone afterwards."""
    T, D = x.shape
    B = mod.shape[0]
    F = w2.shape[1]
    HD = meta.heads * meta.head_dim
    rows_per_sample = meta.n_win_per_sample * meta.L
    assert T == B * rows_per_sample
    y = out if out is not None else torch.empty_like(x)
    ws, dev = _WS, x.device
    step = chunk_step(meta, D, F)
    spans = _forward_spans(meta, B, step, D, F, kept is not None)
    weights = (wn1, wqkv, wo, wn2, w1, w2)
    table = gather[0] if gather is not None else None
    rows = () if out is None else (out,)
    native = (NB.takes(meta, x, mod, (*weights, *rows)) and NB.fits(meta, x, mod, weights, rows, table=table)
              and (kept is None or type(kept) is FreshKept or _all_whole(kept, T, D, HD, meta.heads, F, x.get_device())))
    if not native:
        NB.refuse_misfits(meta, x, mod, weights, table=table)
    if kept is None:
        cmax = max(nw for _, _, nw, _ in spans) * meta.L
        tpn = meta.tp.tp if meta.tp is not None else 1   # gathered rows x local features: the same element count
        shapes = _chunk_shapes(cmax, D, HD, meta.heads, F, tpn)
        get = ws.whole if native else ws.get
        chunk_bufs = {k: get(k, *sh, dev) for k, sh in shapes.items() if k != "h2"}
        chunk_bufs["h1"] = chunk_bufs["h2"] = chunk_bufs.pop("h")
    if native:
        NB.forward(meta, x, mod, weights, y, step, spans[0][3] > 1,
                   {k: t.data_ptr() for k, t in (kept or chunk_bufs).items()}, kept is not None, gather)
        return y
    mods = mod.reshape(B, 6, D).transpose(0, 1).contiguous()           # [6, B, D]: every vector of all samples in a row
    for b, w0, nw, nb in spans:
        sh1, sc1, g1, sh2, sc2, g2 = (mods[:, b] if nb == 1 else mods[:, b:b + nb]).unbind(0)
        r0 = b * rows_per_sample + w0 * meta.L
        n = nw * meta.L
        xc = x[r0:r0 + n]
        h1, qkv, o, x1, h2, act, lse = _chunk_views(kept, r0, n, meta.heads) if kept is not None else \
            _chunk_views(chunk_bufs, 0, n, meta.heads)
        if gather is not None:
            table, peers, src = gather
            E.modnorm_fwd(None, sc1, sh1, wn1, mode=meta.mode, eps=meta.eps, batch=nb, out=h1,
                          gather_idx=table[r0:r0 + n], peer_ptrs=peers, x_out=xc, rows=n,
                          src_rows=src.shape[0])
        else:
            E.modnorm_fwd(xc, sc1, sh1, wn1, mode=meta.mode, eps=meta.eps, batch=nb, out=h1)
        if meta.sp is None:
            G.gemm(h1, wqkv, out=qkv)
            if meta.rope is not None:
                _rope_qk_(qkv, meta, nw)
            A.attn_fwd(qkv, nw, meta.L, meta.heads, meta.head_dim, out=o, lse=lse.view(nw, meta.heads, meta.L))
            oc = o
        else:
            oc = _sp_attention_fwd(meta, h1, wqkv, nw, keep_local=False)[0]
        G.gemm(oc, wo, out=x1, epi=G.EPI_GATE_RESID, resid=xc, gate=g1, rows_per_gate=n // nb)
        if meta.tp is not None:
            _tp_mlp_fwd(meta.tp, x1, sc2, sh2, wn2, meta, w1, w2, g2, chunk_bufs["act"], y[r0:r0 + n])
            continue
        E.modnorm_fwd(x1, sc2, sh2, wn2, mode=meta.mode, eps=meta.eps, batch=nb, out=h2)
        if kept is not None:
            G.gemm(h2, w1, out=act, epi=G.EPI_SWIGLU_BOTH, aux=kept["u"][r0:r0 + n])
        else:
            G.gemm(h2, w1, out=act, epi=G.EPI_SWIGLU)
        G.gemm(act, w2, out=y[r0:r0 + n], epi=G.EPI_GATE_RESID, resid=x1, gate=g2, rows_per_gate=n // nb)
    return y


def block_backward(x: torch.Tensor, mod: torch.Tensor, dy: torch.Tensor, meta: BlockMeta, wn1, wqkv, wo, wn2, w1, w2,
                   grads: dict[str, torch.Tensor], dx: torch.Tensor | None = None,
                   kept: dict[str, torch.Tensor] | None = None):
    """Recompute-and-backpropagate; with ``kept`` (what :func:`block_forward` stored) nothing is recomputed and ``kept`` is
    only read. ``grads`` maps n1, to_qkv, wo, n2, w1, w2 to fp32 accumulators (+=).
    Returns (dx bf16, dmod [B, 6D] fp32). ``dx`` may alias ``dy``."""
    T, D = x.shape
    B = mod.shape[0]
    F = w2.shape[1]
    HD = meta.heads * meta.head_dim
    rows_per_sample = meta.n_win_per_sample * meta.L
    ws, dev, f32 = _WS, x.device, torch.float32
    step = chunk_step(meta, D, F)
    cmax = step * meta.L
    tp = meta.tp
    tpn = tp.tp if tp is not None else 1
    weights = (wn1, wqkv, wo, wn2, w1, w2)
    rows = (dy,) if dx is None else (dy, dx)
    native = NB.takes(meta, x, mod, (*weights, *rows), grads.values()) and NB.fits(meta, x, mod, weights, rows, grads)
    if not native:
        NB.refuse_misfits(meta, x, mod, weights, dx, grads)
    get = ws.whole if native else ws.get
    if kept is not None:
        if not _all_whole(kept, T, D, HD, meta.heads, F, x.get_device()):
            kept = _whole_kept(kept, _kept_shapes(T, D, HD, meta.heads, F), dev)
    else:
        chunk_bufs = {k: get(k, *sh, dev) for k, sh in _chunk_shapes(cmax, D, HD, meta.heads, F, tpn).items()}
        chunk_bufs["h1"], act_b = chunk_bufs.pop("h"), chunk_bufs["act"]
    work = {k: get(k, *sh, dev) for k, sh in _grad_shapes(cmax, D, HD, meta.heads, F, tpn).items()}
    if native:
        dx = torch.empty_like(x) if dx is None else dx
        dmod = torch.empty((B, 6 * D), dtype=f32, device=dev)
        addr = {"du" if k == "u" else k: t.data_ptr() for k, t in work.items()}
        NB.backward(meta, x, mod, dy, weights, step, {k: t.data_ptr() for k, t in (kept or chunk_bufs).items()},
                    kept is not None, addr, dx, dmod, grads)
        return dx, dmod
    du_b, dh, dx1, d_o, dqkv, delta, w2g, wog, G2, Go = work.values()
    G2.zero_()          # dy^T act (ungated w2 gradient of one sample)
    Go.zero_()          # dx1^T o
    dmod = torch.zeros((B, 6 * D), dtype=f32, device=dev)
    if dx is None:
        dx = torch.empty_like(x)
    mod = NB.vectors(mod)
    for b in range(B):
        sh1, sc1, g1, sh2, sc2, g2 = [mod[b, i * D:(i + 1) * D] for i in range(6)]
        dsh1, dsc1, dg1, dsh2, dsc2, dg2 = [dmod[b, i * D:(i + 1) * D] for i in range(6)]
        E.scale_rows(w2, g2, out=w2g)
        E.scale_rows(wo, g1, out=wog)
        for w0, nw in _chunks(meta, step):
            r0 = b * rows_per_sample + w0 * meta.L
            n = nw * meta.L
            xc, dyc = x[r0:r0 + n], dy[r0:r0 + n]
            ksplit_tok = -wanted_slices(meta, nw)
            h1, qkv, o, x1, h2, act, lse = _chunk_views(kept, r0, n, meta.heads) if kept is not None else \
                _chunk_views(chunk_bufs, 0, n, meta.heads)
            lse_c = lse.view(nw, meta.heads, meta.L)
            oc, du = o, du_b[:n]
            u = kept["u"][r0:r0 + n] if kept is not None else du
            if kept is None:
                # ---- recompute the chunk's forward internals
                E.modnorm_fwd(xc, sc1, sh1, wn1, mode=meta.mode, eps=meta.eps, out=h1)
                if meta.sp is None:
                    G.gemm(h1, wqkv, out=qkv)
                    if meta.rope is not None:
                        _rope_qk_(qkv, meta, nw)
                    A.attn_fwd(qkv, nw, meta.L, meta.heads, meta.head_dim, out=o, lse=lse_c)
                else:
                    oc, sp_state = _sp_attention_fwd(meta, h1, wqkv, nw, keep_local=True)
                G.gemm(oc, wo, out=x1, epi=G.EPI_GATE_RESID, resid=xc, gate=g1)
            if tp is not None:
                # tensor-parallel MLP half: h2 and dy are gathered over the group inside the two GEMMs that consume
                # them, the partial dh2 is reduced and scattered by the epilogue of the GEMM that produces it
                from ..parallel import tensor as TP
                Mg = tpn * n
                sl = slice(tp.rank * n, (tp.rank + 1) * n)
                x_buf, x_peers = tp.buffer("ag_x", (Mg, D))
                g_buf, g_peers = tp.buffer("ag_dy", (Mg, D))
                E.modnorm_fwd(x1, sc2, sh2, wn2, mode=meta.mode, eps=meta.eps, out=x_buf[sl])
                g_buf[sl].copy_(dyc)
                tp.barrier()
                TP.gemm_allgather_a(tp, x_buf, x_peers, w1, out=act_b[:Mg], epi=G.EPI_SWIGLU_BOTH, aux=du_b[:Mg])
                TP.gemm_allgather_a(tp, g_buf, g_peers, w2g, b_t=True, out=du_b[:Mg], epi=G.EPI_SWIGLU_BWD, resid=du_b[:Mg])
                G.gemm(g_buf, act_b[:Mg], a_t=True, b_t=True, out=G2, epi=G.EPI_ACC_F32, k_splits=ksplit_tok)
                G.gemm(du_b[:Mg], x_buf, a_t=True, b_t=True, out=grads["w1"], epi=G.EPI_ACC_F32, k_splits=ksplit_tok)
                TP.gemm_reduce_scatter(tp, du_b[:Mg], w1, b_t=True, name="rs_dx", out=dh[:n])
            else:
                if kept is None:
                    E.modnorm_fwd(x1, sc2, sh2, wn2, mode=meta.mode, eps=meta.eps, out=h2)
                    G.gemm(h2, w1, out=act, epi=G.EPI_SWIGLU_BOTH, aux=u)     # act and the raw [gate | up]
                # ---- MLP half: y = x1 + g2 * (act @ w2^T)
                G.gemm(dyc, act, a_t=True, b_t=True, out=G2, epi=G.EPI_ACC_F32, k_splits=ksplit_tok)
                # dact = (dy * g2) @ w2 never reaches memory: the epilogue turns it into du (over u unless that is kept)
                G.gemm(dyc, w2g, b_t=True, out=du, epi=G.EPI_SWIGLU_BWD, resid=u)
                G.gemm(du, w1, b_t=True, out=dh[:n])                                # dh2 = du @ w1
                G.gemm(du, h2, a_t=True, b_t=True, out=grads["w1"], epi=G.EPI_ACC_F32, k_splits=ksplit_tok)
            E.modnorm_bwd(x1, dh[:n], dyc, sc2, sh2, wn2, mode=meta.mode, eps=meta.eps, dx=dx1[:n],
                          dscale=dsc2, dshift=dsh2, dw=grads["n2"])
            # ---- attention half: x1 = x + g1 * (o @ wo^T)
            G.gemm(dx1[:n], oc, a_t=True, b_t=True, out=Go, epi=G.EPI_ACC_F32, k_splits=ksplit_tok)
            if meta.sp is None:
                G.gemm(dx1[:n], wog, b_t=True, out=d_o[:n])                            # do = (dx1 * g1) @ wo
                A.attn_bwd(qkv, o, d_o[:n], lse_c, nw, meta.L, meta.heads, meta.head_dim, dqkv=dqkv[:n],
                           delta=delta[:n * meta.heads].view(nw, meta.heads, meta.L))
                if meta.rope is not None:
                    _rope_qk_(dqkv[:n], meta, nw, inverse=True)
                dq_c = dqkv[:n]
            else:
                dq_c = _sp_attention_bwd(meta, dx1[:n], wog, nw, sp_state)
            G.gemm(dq_c, wqkv, b_t=True, out=dh[:n])                                   # dh1 = dqkv @ wqkv
            G.gemm(dq_c, h1, a_t=True, b_t=True, out=grads["to_qkv"], epi=G.EPI_ACC_F32, k_splits=ksplit_tok)
            E.modnorm_bwd(xc, dh[:n], dx1[:n], sc1, sh1, wn1, mode=meta.mode, eps=meta.eps, dx=dx[r0:r0 + n],
                          dscale=dsc1, dshift=dsh1, dw=grads["n1"])
        # per-sample gate handling: dW += g * G ; dg = rowsum(W * G) ; G <- 0
        E.gate_grad_finalize(G2, w2, g2, grads["w2"], dg2)
        E.gate_grad_finalize(Go, wo, g1, grads["wo"], dg1)
    return dx, dmod


def _pool_alloc(peer_fn, gradient: bool = False):
    """The peer-readable buffer allocator that belongs to a halo exchange's ``peer_fn`` (or None)."""
    return getattr(getattr(peer_fn, "__self__", None), "gradient_buffer" if gradient else "output_buffer", None)


# Names that PyTorch does not publish, looked up once: where a version lacks one, everything counts as recorded.
_forward_level = forward_ad if hasattr(forward_ad, "_current_level") else SimpleNamespace(_current_level=0)
_transforms_active = getattr(torch._C, "_are_functorch_transforms_active", lambda: True)
_tracing_state = getattr(torch._C, "_get_tracing_state", lambda: True)


def recorded() -> bool:
    """Whether anything would notice if an autograd function's forward ran as a plain call: a graph under construction, a
    forward-mode level, a function transform, a trace. Sampling has none of them; the wrapper costs about 15 us."""
    return (torch.is_grad_enabled() or _forward_level._current_level >= 0 or _transforms_active()
            or _tracing_state() is not None)


def run_block(x, mod, meta: BlockMeta, wn1, wqkv, wo, wn2, w1, w2, regroup=None, out_alloc=None) -> torch.Tensor:
    """:class:`FusedBlock` where something is recorded, else its forward pass by itself."""
    if recorded():
        return FusedBlock.apply(x, mod, meta, wn1, wqkv, wo, wn2, w1, w2, regroup, out_alloc)
    return _block_output(x, mod, meta, (wn1, wqkv, wo, wn2, w1, w2), regroup, out_alloc, None)[1]


def _block_output(x, mod, meta: BlockMeta, weights, regroup, out_alloc, kept):
    """(block input in the block's own window layout, output); see :meth:`FusedBlock.forward`."""
    out = out_alloc(x.shape[0], x.shape[1], x.dtype) if out_alloc is not None else None
    if regroup is None:
        return x, block_forward(x, mod.float(), meta, *weights, out=out, kept=kept)
    table_fwd, _, peer_fn = regroup
    peers = peer_fn(x, "fwd") if peer_fn is not None else [x.data_ptr()]
    xg = torch.empty((table_fwd.numel(), x.shape[1]), dtype=x.dtype, device=x.device)
    return xg, block_forward(xg, mod.float(), meta, *weights, out=out, gather=(table_fwd, peers, x), kept=kept)


class FusedBlock(torch.autograd.Function):
    """Autograd wrapper: saves the block input and, with ``meta.keep``, the block's internals; weight gradients go to
    ``param.main_grad`` (fp32) when the engine provides one, otherwise they are returned to autograd."""

    @staticmethod
    def forward(ctx, x, mod, meta, wn1, wqkv, wo, wn2, w1, w2, regroup=None, out_alloc=None):
        """``regroup = (table_fwd, table_bwd, peer_fn)`` fuses the preceding window re-partition into this block: the
        incoming stream ``x`` is in the previous layout (published to the WP peers when ``peer_fn`` is given) and the
        first modulate+norm kernel gathers this block's rows from it. ``out_alloc(rows, cols, dtype)``: where to put the
        output when the caller knows that it will be re-partitioned next (a peer-readable buffer: no publish copy)."""
        ctx.meta = meta
        ctx.regroup = regroup
        kept = None
        if meta.keep and any(ctx.needs_input_grad):        # a frozen block has no backward pass to keep anything for
            shapes = _kept_shapes(regroup[0].numel() if regroup is not None else x.shape[0], x.shape[1],
                                  meta.heads * meta.head_dim, meta.heads, w2.shape[1])
            try:
                kept = FreshKept({k: torch.empty(shape, dtype=dt, device=x.device) for k, (shape, dt) in shapes.items()})
            except torch.OutOfMemoryError:
                kept = None            # free in sum but not in pieces of this size: recompute instead
        x, y = _block_output(x, mod, meta, (wn1, wqkv, wo, wn2, w1, w2), regroup, out_alloc, kept)
        ctx.save_for_backward(x, mod, wn1, wqkv, wo, wn2, w1, w2, *([kept[k] for k in KEPT] if kept is not None else ()))
        return y

    @staticmethod
    def backward(ctx, dy):
        x, mod, wn1, wqkv, wo, wn2, w1, w2, *rest = ctx.saved_tensors
        kept = dict(zip(KEPT, rest)) if rest else None
        params = {"n1": wn1, "to_qkv": wqkv, "wo": wo, "n2": wn2, "w1": w1, "w2": w2}
        grads, ret = {}, {}
        for k, p in params.items():
            mg = getattr(p, "main_grad", None)
            if mg is not None:
                grads[k] = mg.view(p.shape) if mg.dim() != p.dim() else mg
                ret[k] = None
            else:
                grads[k] = torch.zeros(p.shape, dtype=torch.float32, device=p.device)
                ret[k] = grads[k]
        x, dy = x.contiguous(), dy.contiguous()        # a saved-tensor hook may hand back other strides
        dx, dmod = block_backward(x, mod.float(), dy, ctx.meta, wn1, wqkv, wo, wn2, w1, w2, grads, dx=dy, kept=kept)
        if ctx.regroup is not None:
            _, table_bwd, peer_fn = ctx.regroup
            peers = peer_fn(dx, "bwd") if peer_fn is not None else [dx.data_ptr()]
            # the gathered gradient is the next (earlier) layer's dy, which that layer turns into its dx in place and
            # publishes in turn: put it into the other peer-readable buffer straight away
            alloc = _pool_alloc(peer_fn, gradient=True)
            back = (alloc(table_bwd.numel(), dx.shape[1], dx.dtype) if alloc is not None else
                    torch.empty((table_bwd.numel(), dx.shape[1]), dtype=dx.dtype, device=dx.device))
            E.gather_rows(table_bwd, peers, back, src_rows=dx.shape[0])
            dx = back
        out = [ret[k].to(params[k].dtype) if ret[k] is not None else None
               for k in ("n1", "to_qkv", "wo", "n2", "w1", "w2")]
        return (dx, dmod.to(mod.dtype), None, *out, None, None)


class GemvLinearFn(torch.autograd.Function):
    """``silu?(x) @ W^T + b`` for the handful of rows of a modulation MLP (one row per sample): the forward streams the
    weight once through the GEMV kernel; one backward kernel adds the rank-B weight gradient to the fp32 gradient buffers
    and streams the weight once more for the gradient of ``x``."""

    @staticmethod
    def forward(ctx, x, W, b, silu_in: bool):
        from ..ops import diffusion as DF
        ctx.silu_in = silu_in
        ctx.save_for_backward(x, W, b)
        return DF.gemv_bias_act(W.detach(), b.detach() if b is not None else None, x.detach(), act=0, silu_in=silu_in)

    @staticmethod
    def backward(ctx, dy):
        dx, rW, rb = _gemv_backward(*ctx.saved_tensors, dy, ctx.silu_in, ctx.needs_input_grad[0])
        return dx, rW, rb, None


def _gemv_backward(x, W, b, dy, silu_in: bool, need_dx: bool):
    """Gradients of ``silu?(x) @ W^T + b``: (dx or None, and dW and db where they do not go to a ``main_grad``)."""
    from ..ops import diffusion as DF
    from .fused_io import _grad_slot, _kernel_target, _settle
    sW, rW = _grad_slot(W)
    sb, rb = _grad_slot(b) if b is not None else (None, None)
    dx = torch.zeros(x.shape, dtype=torch.float32, device=x.device) if need_dx else None
    if DF.gemv_bwd_ok(W, sW):
        tb = _kernel_target(sb) if sb is not None else None
        DF.gemv_bwd(W, x, dy, sW, tb, dx, silu_in)
        if sb is not None:
            _settle(sb, tb)
    else:
        dy, x32 = dy.float(), x.float()
        sig = torch.sigmoid(x32)
        sW.addmm_(dy.t(), x32 * sig if silu_in else x32)
        if sb is not None:
            sb += dy.sum(0)
        if dx is not None:
            dx = dy @ W.float()
            dx = dx * (sig * (1 + x32 * (1 - sig))) if silu_in else dx
    return (dx.to(x.dtype) if dx is not None else None, rW.to(W.dtype) if rW is not None else None,
            rb.to(b.dtype) if rb is not None else None)


class ModulationFn(torch.autograd.Function):
    """``silu(x @ W1^T + b1) @ W2^T + b2``: two :class:`GemvLinearFn` as one node, whose forward is one native call."""

    @staticmethod
    def forward(ctx, x, W1, b1, W2, b2):
        from ..ops import diffusion as DF
        y1, y2 = DF.modulation_mlp(W1.detach(), b1.detach(), x.detach(), W2.detach(), b2.detach())
        ctx.save_for_backward(x, W1, b1, y1, W2, b2)
        return y2

    @staticmethod
    def backward(ctx, dy):
        from ..ops import diffusion as DF
        from .fused_io import _grad_slot, _kernel_target, _settle
        x, W1, b1, y1, W2, b2 = ctx.saved_tensors
        (s1, r1), (sb1, rb1), (s2, r2), (sb2, rb2) = (_grad_slot(p) for p in (W1, b1, W2, b2))
        if DF.gemv_bwd_ok(W1, s1) and DF.gemv_bwd_ok(W2, s2):
            t1, t2 = _kernel_target(sb1), _kernel_target(sb2)
            dx = DF.modulation_mlp_bwd(W1, x, W2, y1, dy, s1, t1, s2, t2, ctx.needs_input_grad[0])
            _settle(sb1, t1)
            _settle(sb2, t2)
            grads = (r.to(p.dtype) if r is not None else None for p, r in zip((W1, b1, W2, b2), (r1, rb1, r2, rb2)))
            return (dx.to(x.dtype) if dx is not None else None, *grads)
        dy1, r2, rb2 = _gemv_backward(y1, W2, b2, dy, True, True)
        dx, r1, rb1 = _gemv_backward(x, W1, b1, dy1, False, ctx.needs_input_grad[0])
        return dx, r1, rb1, r2, rb2


def modulation(seq: torch.nn.Sequential, emb: torch.Tensor) -> torch.Tensor:
    """The AdaLN modulation MLP ``[Linear,] SiLU, Linear`` (src/aeris/models/parallel_swin.py:321-325) on the GEMV kernel
    where that takes all rows of every layer (at most 8 samples), else on stock operators; fp32 result ``[B, out]``."""
    from ..ops import diffusion as DF
    first, *_, last = parts = list(seq)
    w = last.weight
    if not DF.gemv_ok(emb.shape[0], max(emb.shape[1], w.shape[1])):
        return seq(emb.to(w.dtype)).float()
    if len(parts) == 3 and first.bias is not None and last.bias is not None:
        args = (emb, first.weight, first.bias, w, last.bias)
        return ModulationFn.apply(*args) if recorded() else DF.modulation_mlp(*args[1:3], emb, *args[3:])[1]
    x = emb
    if len(parts) == 3:
        x = GemvLinearFn.apply(x, first.weight, first.bias, False)
    return GemvLinearFn.apply(x, w, last.bias, True)


class Regroup(torch.autograd.Function):
    """Row gather between two window layouts through a table; the backward pass is the gather with the inverse
    table. ``peers`` lists the base addresses of every WP rank's source buffer (just the local one without WP)."""

    @staticmethod
    def forward(ctx, x, table_fwd, table_bwd, peer_fn):
        ctx.table_bwd, ctx.peer_fn = table_bwd, peer_fn
        return Regroup.gather(x, table_fwd, peer_fn)

    @staticmethod
    def gather(x, table_fwd, peer_fn):
        out = torch.empty((table_fwd.numel(), x.shape[1]), dtype=x.dtype, device=x.device)
        peers = peer_fn(x, "fwd") if peer_fn is not None else [x.data_ptr()]
        E.gather_rows(table_fwd, peers, out, src_rows=x.shape[0])
        return out

    @staticmethod
    def backward(ctx, dy):
        dy = dy.contiguous()
        peers = ctx.peer_fn(dy, "bwd") if ctx.peer_fn is not None else [dy.data_ptr()]
        alloc = _pool_alloc(ctx.peer_fn, gradient=True)      # the previous layer's dy: see FusedBlock.backward
        out = (alloc(ctx.table_bwd.numel(), dy.shape[1], dy.dtype) if alloc is not None else
               torch.empty((ctx.table_bwd.numel(), dy.shape[1]), dtype=dy.dtype, device=dy.device))
        E.gather_rows(ctx.table_bwd, peers, out, src_rows=dy.shape[0])
        return out, None, None, None
