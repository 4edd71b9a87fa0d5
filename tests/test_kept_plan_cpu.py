"""How many blocks keep their internals for the backward pass, and how small a chunk may get."""
import math

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
    shapes = fused._kept_shapes(1000, 1536, 1280, 20, 4104).values()
    assert fused.kept_bytes(1000, 1536, 1280, 20, 4104) == sum(math.prod(sh) * dt.itemsize for sh, dt in shapes)


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
    """Windows of a few tokens on the full 720 x 1440 image: half a gigabyte of them is more than the grid's 65,535
    layers."""
    L = win[0] * win[1]
    n_win = 720 * 1440 // L
    meta = fused.BlockMeta(n_win, L, 2, dim // 2, E.MODE_MOD_THEN_NORM, 1e-6, 64)
    step = fused.chunk_step(meta, dim, mlp)
    assert fused.MIN_CHUNK_BYTES // (fused.kept_bytes(1, dim, dim, 2, mlp) * L) > 65535 and step == 65535
    assert all(nw <= 65535 for b, _, nw, _ in fused._forward_spans(meta, 2, step, dim, mlp, True))


@pytest.mark.parametrize("trains", ["x", "mod", "weight", None])
def test_internals_are_kept_only_for_a_backward_pass_that_can_come(trains, monkeypatch):
    """A frozen block on inputs without gradients, called without no_grad: nothing is kept. Any differentiable input: all
    is."""
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


GB, MB = 1 << 30, 1 << 20


class _Memory:
    """Stands in for the allocator and the driver."""

    def __init__(self, monkeypatch, driver, cached=0, fragments=0):
        self.asked = 0
        stat = lambda n: {"all": {"current": n}}
        monkeypatch.setattr(fused, "_WS", fused.Workspace())
        stats = {"reserved_bytes": stat(7 * GB + cached), "allocated_bytes": stat(7 * GB),
                 "inactive_split_bytes": stat(fragments)}
        monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda d: stats)

        def ask(device):
            self.asked += 1
            return driver, 180 * GB
        monkeypatch.setattr(torch.cuda, "mem_get_info", ask)


# the medium model: 2 samples of 32 windows x 900 tokens, 6 blocks
META = fused.BlockMeta(32, 900, 12, 64, E.MODE_MOD_THEN_NORM, 1e-6, 64)
D, FF, BLOCKS, ROWS = 768, 2048, 6, 2 * 32 * 900
NEED = BLOCKS * fused.kept_bytes(ROWS, D, D, 12, FF)
STREAM = ROWS * D * 2
PEAK = (BLOCKS + 2) * STREAM
# chunks of one sample: bytes per row of the gradient workspaces and of the recompute's, and the weight-sized ones
GRADS = 32 * 900 * ((2 * FF + 2 * D + 4 * D) * 2 + 12 * 4) + D * (FF + D) * 6
CHUNK = 32 * 900 * ((3 * D + 4 * D + FF) * 2 + 12 * 4)


def _plan(meta=META, batch=2, d=D, f=FF, blocks=BLOCKS):
    return fused.plan_kept_blocks(meta, batch, d, f, blocks, torch.device("cpu"))


def test_a_cache_that_covers_the_whole_step_needs_no_question(monkeypatch):
    """Whole or in fragments, in which the earlier step's tensors lay."""
    for fragments in (0, NEED):
        mem = _Memory(monkeypatch, driver=0, cached=NEED + PEAK + GRADS, fragments=fragments)
        assert _plan() == BLOCKS and mem.asked == 0


@pytest.mark.parametrize("cached", [NEED, NEED + BLOCKS * STREAM, NEED + PEAK + GRADS - 1])
def test_a_cache_that_covers_only_what_is_kept_leaves_room_for_the_step(cached, monkeypatch):
    """The internals alone, or with the block inputs, fit the cache and the driver has nothing left: what the step needs
    besides comes first."""
    mem = _Memory(monkeypatch, driver=0, cached=cached)
    base = PEAK + 2 * STREAM + GRADS + CHUNK
    want = max(0, (cached - base) // 2 // (NEED // BLOCKS))
    assert _plan() == want < BLOCKS and mem.asked == 1
    assert want == 0 or want * (NEED // BLOCKS) + base <= cached


def test_workspaces_that_are_there_are_not_counted_again(monkeypatch):
    mem = _Memory(monkeypatch, driver=0, cached=NEED + PEAK)
    assert _plan() < BLOCKS and mem.asked == 1
    for name, (shape, dtype) in fused._grad_shapes(32 * 900, D, D, 12, FF).items():
        fused._WS._buf[name] = torch.empty(shape, dtype=dtype, device="meta").flatten()
    monkeypatch.setattr(fused._WS, "missing", lambda shapes, device: fused.Workspace.missing(fused._WS, shapes, "meta"))
    assert _plan() == BLOCKS and mem.asked == 1


def test_fragments_are_not_free_memory_where_the_driver_is_asked(monkeypatch):
    mem = _Memory(monkeypatch, driver=0, cached=NEED + PEAK + GRADS - 1, fragments=NEED)
    assert _plan() == 0 and mem.asked == 1


def test_the_driver_s_memory_is_shared_half_and_half(monkeypatch):
    free = PEAK + 2 * STREAM + GRADS + CHUNK + NEED       # half of the rest: three of six blocks
    mem = _Memory(monkeypatch, driver=free)
    assert _plan() == BLOCKS // 2 and mem.asked == 1
    _Memory(monkeypatch, driver=free + NEED)
    assert _plan() == BLOCKS


def test_a_small_model_on_a_full_device_recomputes(monkeypatch):
    """Needs below 1/256 of the device are not exempt: with 100 MB left in all, a step that needs more keeps nothing."""
    meta = fused.BlockMeta(8, 900, 4, 64, E.MODE_MOD_THEN_NORM, 1e-6, 4)
    assert 2 * fused.kept_bytes(7200, 256, 256, 4, 512) < 180 * GB // 256
    mem = _Memory(monkeypatch, driver=100 * MB)
    assert _plan(meta, 1, 256, 512, 2) == 0 and mem.asked == 1


def test_internals_that_find_no_room_are_recomputed(monkeypatch):
    """The plan counts bytes; where the pieces are too small after all, the block runs without kept internals."""
    seen = []
    monkeypatch.setattr(fused, "block_forward", lambda x, *a, kept=None, **k: seen.append(kept) or torch.zeros_like(x))
    monkeypatch.setattr(fused, "_kept_shapes", lambda *a: {k: ((1 << 60,), torch.uint8) for k in fused.KEPT})
    real = torch.empty

    def empty(shape, **kw):
        if shape == (1 << 60,):
            raise torch.OutOfMemoryError("no room")
        return real(shape, **kw)
    monkeypatch.setattr(torch, "empty", empty)
    meta = fused.BlockMeta(2, 4, 2, 8, E.MODE_MOD_THEN_NORM, 1e-6, 64, keep=True)
    ws = [torch.zeros(s, dtype=torch.bfloat16) for s in ((16,), (48, 16), (16, 16), (16,), (64, 16), (16, 32))]
    y = fused.FusedBlock.apply(torch.zeros(8, 16, requires_grad=True), torch.zeros(1, 96), meta, *ws)
    assert seen == [None] and len(y.grad_fn.saved_tensors) == 8


def test_the_plan_counts_the_workspaces_that_the_passes_use(monkeypatch):
    """The tables behind the plan are the ones that the passes allocate from, merged samples included."""
    asked = {}

    class Spy(fused.Workspace):
        def get(self, name, shape, dtype, device, zero=False):
            asked[name] = max(asked.get(name, 0), math.prod(shape) * dtype.itemsize)
            return super().get(name, shape, dtype, device, zero)

    monkeypatch.setattr(fused, "_WS", Spy())
    for mod, names in ((fused.E, ("modnorm_fwd", "modnorm_bwd", "scale_rows", "gate_grad_finalize")),
                       (fused.G, ("gemm",)), (fused.A, ("attn_fwd", "attn_bwd"))):
        for n in names:
            monkeypatch.setattr(mod, n, lambda *a, **k: None)
    meta = fused.BlockMeta(4, 16, 2, 8, E.MODE_MOD_THEN_NORM, 1e-6, 64)
    bf = torch.bfloat16
    ws = [torch.zeros(s, dtype=bf) for s in ((16,), (48, 16), (16, 16), (16,), (64, 16), (16, 32))]
    x, mod = torch.zeros(2 * 64, 16, dtype=bf), torch.zeros(2, 96)
    fused.block_forward(x, mod, meta, *ws)
    grads = {k: torch.zeros(w.shape) for k, w in zip(("n1", "to_qkv", "wo", "n2", "w1", "w2"), ws)}
    fused.block_backward(x, mod, x.clone(), meta, *ws, grads)
    shapes = {**fused._chunk_shapes(128, 16, 16, 2, 32), **fused._grad_shapes(64, 16, 16, 2, 32)}
    assert asked["h"] == math.prod(shapes["h"][0]) * 2 and set(asked) == set(shapes)
    empty = fused.Workspace()
    assert sum(asked.values()) <= empty.missing(shapes, "cpu")


def _slices(tiles, kb, units=74, most=64, want=0):
    from aeris_gb_b200.ops import lib as L
    return L.lib().aeris_choose_k_splits(tiles, kb, units, most, want)


@pytest.mark.parametrize("tiles,kb,units,most,want,got", [
    (1, 32, 148, 4, 4, 4), (4, 32, 148, 4, 16, 16),     # a toy's weight: one chunk of 2,048 rows for four of 512
    (4, 113, 74, 64, 8, 13),                            # the cheapest number is above what is wanted
    (64, 141, 74, 64, 12, 4), (32, 431, 74, 64, 204, 9),    # finer slices have a price
    (1, 288, 74, 64, 288, 72),                          # finer slices for nothing
    (192, 1013, 74, 64, 4, 5), (108, 1013, 74, 64, 4, 4),   # nothing merged: the cheapest number
    (9, 1, 74, 64, 4, 1), (9, 3, 74, 64, 400, 3), (9, 4, 74, 64, 0, 4)])
def test_slices_of_a_weight_gradient(tiles, kb, units, most, want, got):
    """No empty slice, at least four where there are four k-blocks, and for merged chunks towards the slices of the shorter
    sums."""
    assert _slices(tiles, kb, units, most, want) == got
    assert (got - 1) * -(-kb // got) < kb


@pytest.mark.parametrize("chunk,n_win,nw,want", [(8, 32, 32, 16), (64, 32, 32, 4), (5, 32, 32, 28), (0, 32, 32, 128)])
def test_slices_that_a_merged_chunk_asks_for(chunk, n_win, nw, want):
    """Four per chunk that ``chunk_windows`` names; 0 leaves the chunk to the floor in bytes and must not divide."""
    meta = fused.BlockMeta(n_win, 64, 4, 32, E.MODE_MOD_THEN_NORM, 1e-6, chunk)
    assert fused.chunk_step(meta, 128, 256) == nw
    assert fused.wanted_slices(meta, nw) == want


def test_every_wanted_number_is_met_or_has_a_price():
    cost = lambda t, kb, s: -(-t * s // 74) * (-(-kb // s) + 10)
    for tiles in (1, 7, 33, 74, 75, 500):
        for kb in (1, 5, 57, 200, 1013):
            best = _slices(tiles, kb)
            for want in (4, 9, 50, 1000):
                s = _slices(tiles, kb, want=want)
                assert best <= s <= max(best, want) and cost(tiles, kb, s) <= cost(tiles, kb, best)
                per = -(-kb // min(want, kb))
                finer = {-(-kb // p) for p in range(per, kb + 1)}
                assert not [f for f in finer if s < f and cost(tiles, kb, f) <= cost(tiles, kb, best)]


def test_chunk_windows_bounds_a_chunk_when_asked_to(monkeypatch):
    """``model.min_chunk_bytes: 0``: small chunks are not merged, neither windows nor samples, whatever reads the bound."""
    from aeris_gb_b200.models import aeris as M
    from aeris_gb_b200.utils import config as C
    cfg = C.model_config(C.compose("train", ["experiment=tiny_cpu", "+model.min_chunk_bytes=0", "model.chunk_windows=3",
                                               "model.act_ckpt=false"]))
    assert cfg.min_chunk_bytes == 0
    assert C.model_config(C.compose("train", ["experiment=tiny_cpu"])).min_chunk_bytes is None
    meta = fused.BlockMeta(8, 16, 4, 32, E.MODE_MOD_THEN_NORM, 1e-6, 3, min_chunk_bytes=0)
    step = fused.chunk_step(meta, 128, 256)
    assert step == 3 and [n for _, n in fused._chunks(meta, step)] == [3, 3, 2]
    whole = fused.BlockMeta(8, 16, 4, 32, E.MODE_MOD_THEN_NORM, 1e-6, 8, min_chunk_bytes=0)
    assert len(fused._forward_spans(whole, 2, 8, 128, 256, False)) == 2
    seen = {}
    monkeypatch.setattr(M, "use_fused", lambda x: True)
    monkeypatch.setattr(fused, "plan_kept_blocks", lambda meta, *a: seen.update(meta=meta) or 0)
    M.AerisModel(cfg)._first_kept_block(torch.zeros(8, cfg.dim), M.StreamContext(cfg, 1))
    assert seen["meta"].min_chunk_bytes == 0 and seen["meta"].chunk_windows == 3
