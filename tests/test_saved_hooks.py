"""Saved tensors that come back from a hook with other strides, or as something else, where kernels read them by address."""
import pytest
import torch

from conftest import rel_err
from aeris_gb_b200.models import fused
from aeris_gb_b200.ops import elementwise as E

DEV = "cuda"


def _other_strides(t):
    """The same values, column by column; odd starts for what has one dimension."""
    if t.dim() == 2 and min(t.shape) > 1:
        return t.t().contiguous().t()
    return torch.cat([t.flatten()[:1], t.flatten()])[1:].view_as(t)


def test_kept_internals_are_whole_or_refused():
    T, D, HD, heads, F = 32, 16, 64, 1, 24
    kept = {k: torch.randn(s).to(dt) for k, (s, dt) in fused._kept_shapes(T, D, HD, heads, F).items()}
    want = lambda ks: fused._whole_kept(ks, fused._kept_shapes(T, D, HD, heads, F), torch.device("cpu"))
    assert all(want(kept)[k] is kept[k] for k in kept)                     # nothing is copied where nothing has to be
    got = want({k: _other_strides(t) for k, t in kept.items()})
    assert all(torch.equal(got[k], kept[k]) and got[k].is_contiguous() and got[k].data_ptr() % 16 == 0 for k in kept)
    for k, t in kept.items():
        for bad in (t.double(), t[1:], t.to("meta")):
            with pytest.raises(ValueError):
                want({**kept, k: bad})


def test_internals_that_do_not_fit_are_not_written_by_address(monkeypatch):
    """Forward: the native call takes whole buffers only; others go launch by launch, which refuse them."""
    from aeris_gb_b200.models import block
    from aeris_gb_b200.ops import lib

    class Library:
        def __getattr__(self, entry):
            return lambda *a: 0

    native = []
    monkeypatch.setattr(lib, "lib", Library)
    monkeypatch.setattr(lib, "raw_stream", lambda: 0)
    monkeypatch.setattr(lib, "status_word", lambda: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(block, "takes", lambda *a: True)
    monkeypatch.setattr(block, "forward", lambda *a: native.append(1))
    T, D, heads, d, F = 64, 32, 2, 64, 48
    HD = heads * d
    meta = fused.BlockMeta(2, 16, heads, d, E.MODE_MOD_THEN_NORM, 1e-6, 64)
    z = lambda *s: torch.zeros(s, dtype=torch.bfloat16)
    ws = [z(D), z(3 * HD, D), z(D, HD), z(D), z(2 * F, D), z(D, F)]
    whole = lambda: {k: torch.zeros(s, dtype=dt) for k, (s, dt) in fused._kept_shapes(T, D, HD, heads, F).items()}
    fused.block_forward(z(T, D), torch.zeros(2, 6 * D), meta, *ws, kept=whole())
    assert native == [1]
    for k in fused.KEPT:
        if k != "lse":
            with pytest.raises((AssertionError, RuntimeError, ValueError)):
                fused.block_forward(z(T, D), torch.zeros(2, 6 * D), meta, *ws, kept={**whole(), k: whole()[k][:32]})
    assert native == [1]


@pytest.mark.gpu
@pytest.mark.parametrize("B,L", [(1, 225), (2, 72)])
def test_block_with_kept_internals(B, L):
    heads, d, F, wins = 4, 64, 512, 2
    D = HD = heads * d
    meta = fused.BlockMeta(wins, L, heads, d, E.MODE_MOD_THEN_NORM, 1e-6, 64, keep=True)
    torch.manual_seed(L)
    rnd = lambda *s: (torch.randn(*s, device=DEV) * s[-1] ** -0.5).bfloat16()
    ws = [(1 + rnd(D)), rnd(3 * HD, D), rnd(D, HD), (1 + rnd(D)), rnd(2 * F, D), rnd(D, F)]
    x, dy = torch.randn(2, B * wins * L, D, device=DEV).bfloat16()
    mod = torch.randn(B, 6 * D, device=DEV)

    def grads():
        leaves = [t.clone().requires_grad_(True) for t in (x, mod, *ws)]
        y = fused.FusedBlock.apply(leaves[0], leaves[1], meta, *leaves[2:])
        return torch.autograd.grad(y, leaves, dy.clone())

    want = grads()
    skip = {tuple(w.shape) for w in ws}                # weights of other strides are refused

    def unpack(t):
        return t if tuple(t.shape) in skip else _other_strides(t)

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        got = grads()
    assert torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):                # fp32 sums by atomics, rounded to the parameters' bf16
        assert rel_err(a, b) < 1e-3


def test_modulation_mlp_reads_the_first_layer_in_order(monkeypatch):
    """The address handed on is that of dense rows, whatever strides a hook gave the first layer's result."""
    import ctypes
    from aeris_gb_b200.ops import diffusion as DF
    from aeris_gb_b200.ops import lib
    B, K, N1, N2 = 3, 8, 12, 16
    seen = []

    class Library:
        def aeris_modulation_mlp_bwd(self, *a):
            seen.append(list((ctypes.c_float * (B * N1)).from_address(a[10].value)))
            return 0

    monkeypatch.setattr(lib, "lib", Library)
    monkeypatch.setattr(lib, "raw_stream", lambda: 0)
    x, y1, dy = torch.randn(B, K), torch.randn(B, N1), torch.randn(B, N2)
    z = torch.zeros
    for t in (y1, _other_strides(y1), y1.double()):
        DF.modulation_mlp_bwd(z(N1, K), x, z(N2, N1), t, dy, z(N1, K), z(N1), z(N2, N1), z(N2), True)
    assert seen == [y1.flatten().tolist()] * 3


@pytest.mark.gpu
@pytest.mark.parametrize("B", [1, 2, 5])
@pytest.mark.parametrize("K,N1,N2", [(64, 128, 96), (128, 64, 6 * 128)])
def test_modulation_mlp(B, K, N1, N2):
    x, W1, b1, W2, b2 = (torch.randn(*s, device=DEV) for s in ((B, K), (N1, K), (N1,), (N2, N1), (N2,)))
    dy = torch.randn(B, N2, device=DEV)

    def grads():
        leaves = [t.clone().requires_grad_(True) for t in (x, W1, b1, W2, b2)]
        return torch.autograd.grad(fused.ModulationFn.apply(*leaves), leaves, dy)

    want = grads()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, _other_strides):
        got = grads()
    for a, b in zip(got, want):          # other strides of a weight take the PyTorch formulas: 2e-7, and fast exponentials
        assert rel_err(a, b) < 4e-6
    keep = lambda t: t if t.shape in (W1.shape, W2.shape) and t.shape != (B, N1) else _other_strides(t)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, keep):       # y1 with other strides on the kernels
        got = grads()
    for a, b in zip(got, want):
        assert rel_err(a, b) < 1e-6
