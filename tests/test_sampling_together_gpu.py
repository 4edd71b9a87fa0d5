"""A sampler run whose evaluations are laid out together, against the same run one evaluation at a time: the same kernels on
the same values, so bit for bit the same forecast."""
import pytest
import torch

from aeris_gb_b200.diffusion.rollout import DeviceForecaster, SamplerConfig
from aeris_gb_b200.models import aeris as A
from aeris_gb_b200.models.sampling import Evaluations
from aeris_gb_b200.ops import diffusion as DF

pytestmark = pytest.mark.gpu
C = 16


def _model(**over):
    kw = dict(img=(32, 64), window=(8, 8), in_channels=2 * C + 2, out_channels=C, dim=128, heads=4, head_dim=32, mlp_dim=256,
              n_layers=2, sublayers=1)
    torch.manual_seed(0)
    with torch.device("cuda"):
        model = A.AerisModel(A.AerisConfig(**{**kw, **over})).eval()
    torch.nn.init.normal_(model.output_stage.head.weight, std=0.05)
    return model


def _forecast(model, batch, sampler):
    cfg = model.cfg
    gen = torch.Generator(device="cuda").manual_seed(1)
    state, forcing = (torch.randn(batch, *cfg.img, c, device="cuda", generator=gen) for c in (C, 2))
    stats = {k: torch.full((C,), float("std" in k), device="cuda") for k in ("x_mean", "x_std", "t_mean", "t_std")}
    fc = DeviceForecaster(model, A.StreamContext(cfg, batch), stats, sampler, C, seed=3)
    return fc.step(fc.step(state, forcing), forcing)


def _both(model, batch, sampler, monkeypatch):
    """(result, how many runs were laid out together), and the result one by one."""
    prepare, taken = Evaluations.prepare, []
    monkeypatch.setattr(Evaluations, "prepare", lambda *a: taken.append(prepare(*a)) or taken[-1])
    together = _forecast(model, batch, sampler)
    monkeypatch.setattr(Evaluations, "prepare", lambda *a: None)
    return together, sum(t is not None for t in taken), _forecast(model, batch, sampler)


@pytest.mark.parametrize("batch,sampler,over", [
    (1, dict(n_steps=1), dict(n_layers=1)),                                    # one evaluation, no shifted layer
    (2, dict(n_steps=2), {}),                                                  # back from the shifted partition at the end
    (3, dict(n_steps=3), dict(n_layers=3, sublayers=2)),
    (2, dict(n_steps=5, heun=False), dict(after_mod_norm=False)),
    (1, dict(n_steps=6), dict(use_rope=True)),                                 # eleven levels: two passes of eight
    (2, dict(n_steps=3, s_churn=2.0), dict(heads=2, head_dim=64)),
    (2, dict(n_steps=2), dict(chunk_windows=3, min_chunk_bytes=0)),            # chunks, a ragged last one
    (2, dict(n_steps=2), dict(dim=384, heads=3, head_dim=128, mlp_dim=640)),
    (8, dict(n_steps=2), {}),
])
def test_equal_to_one_by_one(batch, sampler, over, monkeypatch):
    together, taken, alone = _both(_model(**over), batch, SamplerConfig(**sampler), monkeypatch)
    assert taken == 2 and torch.isfinite(alone).all() and torch.equal(together, alone)


@pytest.mark.parametrize("batch,over", [(2, dict(layerwise_t_emb=False)), (9, {})])
def test_what_goes_one_by_one(batch, over, monkeypatch):
    together, taken, alone = _both(_model(**over), batch, SamplerConfig(n_steps=2), monkeypatch)
    assert taken == 0 and torch.equal(together, alone)


def test_hooks_and_replaced_parts_are_called(monkeypatch):
    model, calls = _model(), []
    plain = _forecast(model, 1, SamplerConfig(n_steps=2))
    handle = model.layers[1].register_forward_hook(lambda *_: calls.append(1))
    assert torch.equal(_forecast(model, 1, SamplerConfig(n_steps=2)), plain) and len(calls) == 2 * 3
    handle.remove()
    own = model.predict_images
    model.predict_images = lambda *a: calls.append(2) or own(*a)
    assert torch.equal(_forecast(model, 1, SamplerConfig(n_steps=2)), plain) and calls.count(2) == 2 * 3


def test_new_weights_between_steps():
    model = _model()
    first = _forecast(model, 1, SamplerConfig(n_steps=2))
    with torch.no_grad():
        model.layers[0].blocks()[0][1].wo.weight.mul_(2)
        model.output_stage.head.weight.mul_(1.5)
    assert not torch.equal(first, _forecast(model, 1, SamplerConfig(n_steps=2)))


def test_without_memory_for_all_buffers(monkeypatch):
    def full(*a):
        raise torch.OutOfMemoryError("no memory for three streams")
    model = _model()
    plain = _forecast(model, 1, SamplerConfig(n_steps=2))
    monkeypatch.setattr(Evaluations, "_lay_out_blocks", full)
    assert torch.equal(plain, _forecast(model, 1, SamplerConfig(n_steps=2)))


@pytest.mark.parametrize("n", [1, 64, 65])
def test_levels_that_travel_with_the_launch(n):
    t = torch.linspace(0.01, 1.57, n)
    for dtype in (torch.float32, torch.bfloat16):
        assert torch.equal(DF.noise_embedding_of(t.tolist(), 96, 1e4, dtype, "cuda"),
                           DF.noise_embedding(t.cuda(), 96, 1e4, dtype))
