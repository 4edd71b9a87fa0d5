"""One native call per pass over a transformer block: the launches of :func:`.fused.block_forward` and
:func:`.fused.block_backward` on one GPU, issued by ``csrc/block.cu`` instead of one by one from Python."""
from __future__ import annotations

import ctypes
import math

import torch

from ..ops import elementwise as E
from ..ops import gemm as G
from ..ops import lib as _l

_P, _I, _F, _LL = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_longlong


class BlockArgs(ctypes.Structure):
    """Mirror of ``AerisBlock`` (csrc/api.h)."""
    _fields_ = ([(n, _I) for n in ("D", "F", "heads", "head_dim", "L", "mode", "n_win", "batch", "step", "merged",
                                   "slice_windows", "kept", "two_cta", "n_peers")]
                + [("eps", _F), ("scale", _F), ("mod_vec", _LL), ("mod_sample", _LL)]
                + [(n, _P) for n in ("mod", "wn1", "wqkv", "wo", "wn2", "w1", "w2", "rope_cos", "rope_sin", "x", "y",
                                     "table", "peers", "h1", "qkv", "o", "lse", "x1", "h2", "act", "u", "status", "stream")])


class BlockGradArgs(ctypes.Structure):
    """Mirror of ``AerisBlockGrad`` (csrc/api.h)."""
    _fields_ = [(n, _P) for n in ("dy", "dx", "du", "dh", "dx1", "d_o", "dqkv", "w2g", "wog", "delta", "G2", "Go", "dmod",
                                  "n1", "to_qkv", "wo", "n2", "w1", "w2")]


def _plain(t: torch.Tensor, dtype: torch.dtype) -> bool:
    return t.dtype == dtype and t.is_cuda and t.is_contiguous()


def takes(meta, x: torch.Tensor, mod: torch.Tensor, weights, grads=()) -> bool:
    """Whether the native call takes this block: bf16 operands without gaps, fp32 modulation and gradients, heads of whole
    16-byte vectors, none of the exchanges of the parallel paths. Everything else is issued (or refused) call by call."""
    d = meta.head_dim
    if not (meta.sp is None and meta.tp is None and (d in (64, 128) or (d % 8 == 0 and 0 < d < 128))
            and mod.dtype == torch.float32 and mod.is_cuda and _plain(x, torch.bfloat16)):
        return False
    for w in weights:
        if not _plain(w, torch.bfloat16):
            return False
    for g in grads:
        if not _plain(g, torch.float32):
            return False
    return True


WEIGHTS = ("n1", "to_qkv", "wo", "n2", "w1", "w2")


def fits(meta, x: torch.Tensor, mod: torch.Tensor, weights, rows=(), grads=None, table=None) -> bool:
    """Whether every operand has the extents that the native call derives from ``x``, ``w2`` and ``meta``: it has no other
    check. ``rows``: tensors shaped like ``x``; ``grads``: as :func:`.fused.block_backward` takes them. What does not fit
    goes launch by launch, where each is checked by itself. Every pass over a block asks: what :func:`takes` has found to be
    whole is compared by its number of elements where another shape of as many reads the same."""
    n1, to_qkv, wo, n2, w1, w2 = weights
    xs, ms, w2_shape, HD = x.shape, mod.shape, w2.shape, meta.heads * meta.head_dim
    (T, D), F = xs, w2_shape[1]
    qkv_shape, w1_shape = (3 * HD, D), (2 * F, D)
    if (T != ms[0] * meta.n_win_per_sample * meta.L or ms != (ms[0], 6 * D) or to_qkv.shape != qkv_shape
            or wo.shape != (D, HD) or w1.shape != w1_shape or w2_shape != (D, F) or n1.numel() != D or n2.numel() != D
            or (table is not None and table.numel() != T)):
        return False
    for r in rows:
        if r.shape != xs:
            return False
    return grads is None or (grads["to_qkv"].shape == qkv_shape and grads["w1"].shape == w1_shape
                             and grads["wo"].numel() == D * HD and grads["w2"].numel() == D * F
                             and grads["n1"].numel() == D and grads["n2"].numel() == D)


def refuse_misfits(meta, x: torch.Tensor, mod: torch.Tensor, weights, dx=None, grads=None, table=None) -> None:
    """Raises for the extents that no launch checks by itself, where kernels would read or write out of range."""
    (T, D), need = x.shape, mod.shape[0] * meta.n_win_per_sample * meta.L
    wrong = [k for k, w in zip(WEIGHTS, weights) if k in ("n1", "n2") and w.numel() != D]
    if T < need:
        wrong.append("x")
    if mod.numel() < mod.shape[0] * 6 * D or (grads is not None and (mod.dim() != 2 or mod.shape[1] < 6 * D)):
        wrong.append("mod")
    if dx is not None and (dx.shape[0] < need or dx.shape[1] != D):
        wrong.append("dx")
    if grads is not None:
        wrong += [f"grads[{k}]" for k, w in zip(WEIGHTS, weights) if grads[k].numel() != w.numel()]
    if table is not None and table.numel() < T:
        wrong.append("gather table")
    if wrong:
        raise ValueError(f"operands that do not fit a block of {T} rows of {D}: {', '.join(wrong)}")


def vectors(mod: torch.Tensor) -> torch.Tensor:
    """``mod`` as the kernels of both directions read it: without gaps, from a 16-byte boundary on (vectors of four)."""
    mod = mod.contiguous()
    return mod if mod.data_ptr() % 16 == 0 else mod.clone()


def _args(meta, x, mod, B, D, F, step, weights, bufs: dict[str, int], kept: bool, stream: int) -> tuple[BlockArgs, tuple]:
    """The arguments both directions share, and what has to live until the call returns. ``bufs``: addresses of internals."""
    wn1, wqkv, wo, wn2, w1, w2 = weights
    cos = sin = None
    if meta.rope is not None:
        cos, sin = (t.float().contiguous() for t in meta.rope)
        assert cos.shape == (meta.L, meta.head_dim // 2)
    a = BlockArgs(D=D, F=F, heads=meta.heads, head_dim=meta.head_dim, L=meta.L, mode=meta.mode, n_win=meta.n_win_per_sample,
                  batch=B, step=step, slice_windows=max(1, min(meta.chunk_windows, meta.n_win_per_sample)), kept=kept,
                  two_cta=G.TWO_CTA_DEFAULT, eps=meta.eps, scale=1.0 / math.sqrt(meta.head_dim), mod_vec=D, mod_sample=6 * D,
                  mod=mod.data_ptr(), wn1=wn1.data_ptr(), wqkv=wqkv.data_ptr(), wo=wo.data_ptr(), wn2=wn2.data_ptr(),
                  w1=w1.data_ptr(), w2=w2.data_ptr(), x=x.data_ptr(), status=_l.status_word().data_ptr(), stream=stream,
                  **bufs)
    if cos is not None:
        a.rope_cos, a.rope_sin = cos.data_ptr(), sin.data_ptr()
    return a, (mod, cos, sin)


def _issued(rc: int, what: str) -> None:
    _l.check(min(rc, 0), what, kernels=max(rc, 0))


def forward(meta, x, mod, weights, y, step: int, merged: bool, bufs: dict[str, int], kept: bool, gather=None) -> None:
    """``mod`` [B, 6 D] fp32, read in place: samples that run in one launch find their vectors 6 D apart. ``gather``: see
    :func:`.fused.block_forward`."""
    B, D, F = mod.shape[0], x.shape[1], weights[5].shape[1]
    mod = vectors(mod)
    a, alive = _args(meta, x, mod, B, D, F, step, weights, bufs, kept, _l.raw_stream())
    a.merged, a.y = merged, y.data_ptr()
    if gather is not None:
        table, peers, src = gather
        if E._CHECKED:
            E.set_gather_bounds(src.shape[0])
        arr = E._peer_array(peers)
        a.table, a.peers, a.n_peers = table.data_ptr(), ctypes.addressof(arr), len(peers)
    _issued(_l.lib().aeris_block_forward(ctypes.byref(a)), "aeris_block_forward")


def issue_forward(records: ctypes.Array, mod_offset: int) -> None:
    """The forward passes over consecutive blocks in one call, on the current stream: ``records`` as :func:`_args` lays them
    out, with ``mod_offset`` elements added to each one's modulation vectors."""
    _issued(_l.lib().aeris_blocks_forward(records, len(records), _LL(mod_offset), _l.stream_ptr()), "aeris_blocks_forward")


def backward(meta, x, mod, dy, weights, step: int, bufs: dict[str, int], kept: bool, work: dict[str, int], dx, dmod,
             grads: dict[str, torch.Tensor]) -> None:
    """``work``: addresses of the gradient workspaces; ``dmod`` [B, 6 D] fp32 is overwritten."""
    mod = vectors(mod)
    a, alive = _args(meta, x, mod, mod.shape[0], x.shape[1], weights[5].shape[1], step, weights, bufs, kept, _l.raw_stream())
    g = BlockGradArgs(dy=dy.data_ptr(), dx=dx.data_ptr(), dmod=dmod.data_ptr(), **work,
                      **{k: t.data_ptr() for k, t in grads.items()})
    _issued(_l.lib().aeris_block_backward(ctypes.byref(a), ctypes.byref(g)), "aeris_block_backward")
