"""Gradients that kernels add by address: a ``main_grad`` of another type or layout gets its sum, never a foreign write. The
kernels are stand-ins that check what they are handed."""
from types import SimpleNamespace

import pytest
import torch

from aeris_gb_b200.models import fused, fused_io
from aeris_gb_b200.ops import diffusion as DF

LAYOUTS = {"fp32": lambda *s: torch.zeros(*s), "bf16": lambda *s: torch.zeros(*s, dtype=torch.bfloat16),
           "fp64": lambda *s: torch.zeros(*s, dtype=torch.float64),
           "strided": lambda *s: torch.zeros(*s, 2)[..., 0]}


def _add_ones(*targets):
    for t in targets:
        if t is not None:
            assert t.dtype == torch.float32 and t.is_contiguous()
            t += 1


def _param(layout, *shape):
    p = torch.nn.Parameter(torch.randn(*shape))
    p.main_grad = LAYOUTS[layout](*shape)
    return p


@pytest.mark.parametrize("layout", LAYOUTS)
def test_modulation_bias(layout, monkeypatch):
    monkeypatch.setattr(DF, "gemv_bias_act", lambda W, b, x, act, silu_in: x @ W.t() + b)
    monkeypatch.setattr(DF, "gemv_bwd", lambda W, x, dy, dW, db, dx, silu_in: _add_ones(dW, db, dx))
    W, b = _param("fp32", 6, 8), _param(layout, 6)
    fused.GemvLinearFn.apply(torch.randn(2, 8, requires_grad=True), W, b, True).sum().backward()
    assert (b.main_grad == 1).all() and (W.main_grad == 1).all()


def test_modulation_weight_gradients_of_another_type_are_not_for_the_kernel():
    W = torch.zeros(6, 8)
    assert DF.gemv_bwd_ok(W, torch.zeros(6, 8))
    assert not DF.gemv_bwd_ok(W, torch.zeros(6, 8, dtype=torch.bfloat16))
    assert not DF.gemv_bwd_ok(W, torch.zeros(8, 6).t())
    rows = 65535 * 16
    assert DF.gemv_bwd_ok(torch.zeros(rows, 4), torch.zeros(rows, 4))
    assert not DF.gemv_bwd_ok(torch.zeros(rows + 1, 4), torch.zeros(rows + 1, 4))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_input_projection(layout, monkeypatch):
    monkeypatch.setattr(DF, "embed_pack", lambda *a, **k: None)
    monkeypatch.setattr(fused_io.G, "gemm", lambda *a, **k: None)
    monkeypatch.setattr(DF, "fold_embed_grad", lambda G, dW, db: _add_ones(dW, db))
    W, b = _param(layout, 16, 4), _param(layout, 16)
    plan = SimpleNamespace(geom=SimpleNamespace(rows=8), ape_y=None, ape_x=None, seed=0, sigma_data=1.0, noise=False)
    ctx = SimpleNamespace(plan=plan, saved_tensors=(None, None, None, W, b))
    fused_io.EmbedFn.backward(ctx, torch.zeros(8, 16, dtype=torch.bfloat16))
    assert (W.main_grad == 1).all() and (b.main_grad == 1).all()


@pytest.mark.parametrize("layout", LAYOUTS)
def test_output_norm(layout, monkeypatch):
    monkeypatch.setattr(DF, "pack_head_weights", lambda w, rows: torch.zeros(rows, 3 * w.shape[1], dtype=torch.bfloat16))
    monkeypatch.setattr(fused_io.G, "gemm", lambda *a, **k: None)
    monkeypatch.setattr(fused_io.E, "modnorm_fwd", lambda *a, **k: None)
    monkeypatch.setattr(fused_io.E, "modnorm_bwd", lambda *a, dw, **k: _add_ones(dw))
    D, T, B = 16, 8, 2
    norm, head = _param(layout, D), _param("fp32", 3, D)
    mod = torch.zeros(B, D)
    ctx = SimpleNamespace(plan=SimpleNamespace(eps=1e-6),
                          saved_tensors=(torch.zeros(T, D, dtype=torch.bfloat16), mod, mod, norm, head,
                                         torch.zeros(T, fused_io.PAD_N, dtype=torch.bfloat16)))
    fused_io.HeadLossFn.backward(ctx, torch.ones(()))
    assert (norm.main_grad == B).all()          # one call per sample
