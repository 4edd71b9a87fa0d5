"""How many blocks keep their internals for the backward pass, and how small a chunk may get."""
import pytest
import torch

from aeris_gb_b200.models import fused
from aeris_gb_b200.ops import elementwise as E


@pytest.mark.parametrize("free,want", [(100 << 30, 10), (30 << 30, 5), (11 << 30, 0), (5 << 30, 0), (12 << 30, 0)])
def test_kept_blocks_take_at_most_half_of_the_free_memory(free, want):
    # 10 blocks of 2 GiB next to 10 GiB that the step needs anyway
    n = fused.n_kept(10, 2 << 30, 10 << 30, free)
    assert n == want and n * (2 << 30) <= max(0, free - (10 << 30)) / 2


def test_a_block_keeps_every_recomputed_internal():
    per_row = 3 * 1536 * 2 + 4 * 1536 * 2 + 3 * 4096 * 2 + 24 * 4        # h1, x1, h2 | qkv, o | act, u | lse
    assert fused.kept_bytes(1000, 1536, 1536, 24, 4096) == 1000 * per_row
    assert set(fused._kept_shapes(8, 16, 16, 2, 32)) == set(fused.KEPT)


@pytest.mark.parametrize("dim,heads,mlp,L,chunk,n_win,want", [
    (1536, 24, 4096, 900, 72, 288, 72),       # the caller's bound holds where a chunk is large
    (1536, 24, 4096, 900, 4, 288, 12),        # 512 MiB of internals: 12 windows
    (128, 4, 256, 64, 8, 32, 32),             # a toy sample is one chunk
    (5120, 40, 13696, 900, 72, 32, 32)])
def test_chunks_below_half_a_gigabyte_are_merged(dim, heads, mlp, L, chunk, n_win, want):
    meta = fused.BlockMeta(n_win, L, heads, dim // heads, E.MODE_MOD_THEN_NORM, 1e-6, chunk)
    step = fused.chunk_step(meta, dim, mlp)
    assert step == want
    spans = list(fused._chunks(meta, step))
    assert sum(n for _, n in spans) == n_win and [w for w, _ in spans] == list(range(0, n_win, step))


@pytest.mark.parametrize("win,dim,mlp", [((1, 1), 128, 256), ((1, 2), 128, 256), ((2, 2), 64, 64)])
def test_merged_chunks_stay_within_the_attention_grid(win, dim, mlp):
    """Windows of a few tokens on the full 720 x 1440 image: half a gigabyte of them is more than the grid's 65,535 layers."""
    L = win[0] * win[1]
    n_win = 720 * 1440 // L
    meta = fused.BlockMeta(n_win, L, 2, dim // 2, E.MODE_MOD_THEN_NORM, 1e-6, 64)
    step = fused.chunk_step(meta, dim, mlp)
    assert fused.MIN_CHUNK_BYTES // (fused.kept_bytes(1, dim, dim, 2, mlp) * L) > 65535 and step == 65535
    assert all(nw <= 65535 for b, _, nw, _ in fused._forward_spans(meta, 2, step, dim, mlp, True))


@pytest.mark.parametrize("trains", ["x", "mod", "weight", None])
def test_internals_are_kept_only_for_a_backward_pass_that_can_come(trains, monkeypatch):
    """A frozen block on inputs without gradients, called without no_grad: nothing is kept. Any differentiable input: all is."""
    seen = []

    def forward(x, mod, meta, *weights, out=None, gather=None, kept=None):
        seen.append(kept)
        return torch.zeros_like(x)

    monkeypatch.setattr(fused, "block_forward", forward)
    meta = fused.BlockMeta(2, 4, 2, 8, E.MODE_MOD_THEN_NORM, 1e-6, 64, keep=True)
    bf = dict(dtype=torch.bfloat16)
    x, mod = torch.zeros(8, 16, requires_grad=trains == "x", **bf), torch.zeros(1, 96, requires_grad=trains == "mod")
    ws = [torch.zeros(16, **bf), torch.zeros(48, 16, **bf), torch.zeros(16, 16, **bf), torch.zeros(16, **bf),
          torch.zeros(64, 16, **bf), torch.zeros(16, 32, requires_grad=trains == "weight", **bf)]
    y = fused.FusedBlock.apply(x, mod, meta, *ws)
    assert y.requires_grad == (trains is not None)
    assert (seen[0] is not None) == (trains is not None)
    if trains:
        assert set(seen[0]) == set(fused.KEPT) and seen[0]["u"].shape == (8, 64)


@pytest.mark.parametrize("recompute,first", [(False, 1), (True, 4)])
def test_an_explicit_request_to_recompute_is_followed(recompute, first, monkeypatch):
    """``model.act_ckpt: true`` reaches the CUDA path: no block keeps anything and the memory is not even asked about."""
    from aeris_gb_b200.models import aeris as M
    from aeris_gb_b200.utils import config as C
    run = C.compose("train", ["experiment=tiny_cpu", f"model.act_ckpt={str(recompute).lower()}"])
    cfg = C.model_config(run)
    assert cfg.recompute == recompute and cfg.oracle_checkpoint == recompute and cfg.n_blocks == 4
    model = M.AerisModel(cfg)
    ctx = M.StreamContext(cfg, 1)
    monkeypatch.setattr(M, "use_fused", lambda x: True)
    monkeypatch.setattr(fused, "plan_kept_blocks", lambda *a: pytest.fail("asked") if recompute else 3)
    assert model._first_kept_block(torch.zeros(8, cfg.dim), ctx) == first
