"""Whole steps, whose kernels may start while the one before them still runs, against the same steps with a wait after every
launch: packing of the input, modulation vectors both ways, blocks, head and loss, sampler updates."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _config(**kw):
    from aeris_gb_b200.models.aeris import AerisConfig
    return AerisConfig(img=(60, 120), window=(30, 30), in_channels=20, out_channels=9, dim=256, heads=4, head_dim=64,
                       mlp_dim=512, n_layers=2, sublayers=1, chunk_windows=4, **kw)


def _wait_after_each_launch(monkeypatch):
    from aeris_gb_b200.models import block
    from aeris_gb_b200.ops import lib
    check, waits = lib.check, []
    monkeypatch.setattr(block, "takes", lambda *a: False)             # no calls that issue several blocks' launches at once
    monkeypatch.setattr(lib, "check", lambda *a, **k: (check(*a, **k), torch.cuda.synchronize(), waits.append(1))[0])
    return waits


@pytest.mark.parametrize("after_mod_norm", [True, False])
def test_training_steps(after_mod_norm, monkeypatch):
    from aeris_gb_b200.engine.optim import OptimConfig
    from aeris_gb_b200.engine.trainer import DiffusionConfig, Trainer
    gen = torch.Generator().manual_seed(1)
    x, c = (torch.randn(2, 60, 120, n, generator=gen).pin_memory() for n in (9, 11))

    def steps():
        torch.manual_seed(0)
        tr = Trainer(_config(after_mod_norm=after_mod_norm), OptimConfig(), DiffusionConfig(cond_channels=11), "cuda", seed=3)
        # the first step: later ones start from weights that AdamW has moved by the sign of gradients near zero
        return tr.train_step(x, c), [s.m.clone() for s in tr.opt.segments]

    chained = [steps() for _ in range(2)]
    waits = _wait_after_each_launch(monkeypatch)
    loss, m = steps()
    assert len(waits) > 50
    for loss0, m0 in chained:
        assert abs(float(loss0) - float(loss)) <= 1e-5 * abs(float(loss))
        for a, b in zip(m0, m):
            assert rel_err(a, b) < 1e-4                   # fp32 atomics in another order each time, and what bf16 makes of it


def test_sampler_steps(monkeypatch):
    from aeris_gb_b200.diffusion.rollout import DeviceForecaster, SamplerConfig
    from aeris_gb_b200.models.aeris import AerisModel, StreamContext
    torch.manual_seed(0)
    cfg = _config()
    with torch.device("cuda"):
        model = AerisModel(cfg).eval()
    stats = {k: torch.zeros(9, device="cuda") if "mean" in k else torch.ones(9, device="cuda")
             for k in ("x_mean", "x_std", "t_mean", "t_std")}
    state, forcing = torch.randn(2, 60, 120, 9, device="cuda"), torch.randn(2, 60, 120, 2, device="cuda")

    def step():
        fc = DeviceForecaster(model, StreamContext(cfg, 2), stats, SamplerConfig(n_steps=3, s_churn=1.0), 9, seed=5)
        return fc.step(state, forcing).clone()

    chained = [step() for _ in range(3)]
    waits = _wait_after_each_launch(monkeypatch)
    want = step()
    assert len(waits) > 50 and bool(want.isfinite().all())
    for got in chained:
        assert torch.equal(got, want)
