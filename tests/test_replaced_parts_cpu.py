"""`predict_images` and the forecast's evaluations look past a part of the model only where it is the stock one: what a caller
put in its place, on an instance or on the class, is called as before."""
import pytest
import torch

from aeris_gb_b200.models import aeris as A

CFG = dict(img=(16, 32), window=(8, 8), in_channels=10, out_channels=4, dim=32, heads=2, head_dim=16, mlp_dim=64, sublayers=1)


def _predict(monkeypatch, replace, n_layers):
    """Calls `predict_images` with an input stage and an output stage that need no kernels; (result, the whole trunk's rows)."""
    torch.manual_seed(0)
    model = A.AerisModel(A.AerisConfig(**CFG, n_layers=n_layers)).eval()
    ctx = A.StreamContext(model.cfg, 1)
    x = torch.randn(16 * 32, 32, dtype=model.cfg.model_dtype)
    dt = torch.randn(1, 32, dtype=model.cfg.model_dtype)
    with torch.no_grad():
        whole = model.trunk(x, dt, ctx)
    model.input_stage.forward_images = lambda *a: (x, dt)
    replace(model, ctx)
    return model.predict_images(torch.zeros(1, 16, 32, 4), None, None, ctx, None), whole


@pytest.mark.parametrize("n_layers", [1, 2])            # without and with a shifted partition at the end
@pytest.mark.parametrize("where", ["instance", "class"])
def test_an_output_stage_of_two_arguments(monkeypatch, where, n_layers):
    def replace(model, ctx):
        if where == "instance":
            model.output_stage.predict_tokens = lambda x, dt: (x, dt.shape)
        else:
            monkeypatch.setattr(A.OutputStage, "predict_tokens", lambda self, x, dt: (x, dt.shape))
    (rows, _), whole = _predict(monkeypatch, replace, n_layers)
    assert torch.equal(rows, whole)


def test_an_output_stage_that_ignores_further_arguments(monkeypatch):
    def replace(model, ctx):
        model.output_stage.predict_tokens = lambda x, *_: x
    rows, whole = _predict(monkeypatch, replace, 2)
    assert torch.equal(rows, whole)


@pytest.mark.parametrize("where", ["trunk", "trunk of the class", "way back"])
def test_a_trunk_of_another_kind(monkeypatch, where):
    calls = []

    def replace(model, ctx):
        if where == "way back":
            own = ctx.regroup_unfused
            ctx.regroup_unfused = lambda *a: calls.append(1) or own(*a)
        else:
            own = A.AerisModel.trunk
            if where == "trunk":
                model.trunk = lambda *a: calls.append(1) or own(model, *a)
            else:
                monkeypatch.setattr(A.AerisModel, "trunk", lambda *a: calls.append(1) or own(*a))
        monkeypatch.setattr("aeris_gb_b200.models.fused.modulation", lambda *a: torch.zeros(1, 64))
        monkeypatch.setattr("aeris_gb_b200.models.fused_io.head_forward", lambda x, *a, table=None, **k: (x, table))
    (rows, table), whole = _predict(monkeypatch, replace, 2)
    assert calls[-1:] == [1] and table is None and torch.equal(rows, whole)


@pytest.mark.parametrize("kind", [A.AerisModel, A.InputStage, A.OutputStage, A.SwinLayer])
def test_what_counts_as_replaced(monkeypatch, kind):
    model = A.AerisModel(A.AerisConfig(**CFG, n_layers=1))
    part = next(m for m in model.modules() if type(m) is kind)
    assert not A.replaced(part, kind)
    for other in (lambda *a: None, kind.forward.__get__(object())):
        part.forward = other
        assert A.replaced(part, kind) and A.replaced(part, kind, "forward") and not A.replaced(part, kind, "__init__")
        del part.forward
    assert not A.replaced(part, kind)
    monkeypatch.setattr(kind, "forward", lambda self, *a: None)
    assert A.replaced(part, kind)
    monkeypatch.undo()
    assert not A.replaced(part, kind)
    part.__class__ = type("Own", (kind,), {})
    assert A.replaced(part, kind) and not A.replaced(part, kind, "forward")
