"""Routes of the noise-level embedding: the kernel works on plain values only, everything that carries a derivative or a
hidden dimension takes the formulas."""
import pytest
import torch
from torch.autograd import forward_ad

from aeris_gb_b200.models import aeris as M
from aeris_gb_b200.ops import diffusion as DF


@pytest.fixture(params=[True, False], ids=["layerwise", "shared"])
def stage(request, monkeypatch):
    """An input stage that believes it runs on the GPU, with the kernel replaced by NaN."""
    cfg = M.AerisConfig(img=(8, 16), window=(4, 4), in_channels=6, out_channels=2, dim=16, heads=2, head_dim=8, mlp_dim=32,
                        n_layers=1, sublayers=1, layerwise_t_emb=request.param, model_dtype=torch.float32)
    monkeypatch.setattr(M, "use_fused", lambda t: True)
    monkeypatch.setattr(DF, "noise_embedding", lambda t, dim, *_: torch.full((t.shape[0], dim), float("nan")))
    return M.InputStage(cfg)


T = torch.tensor([0.3, 1.2])


def _formulas(stage, t):
    e = M.O.timestep_embedding(t, stage.cfg.dim, stage.cfg.max_period)
    return e if stage.cfg.layerwise_t_emb else stage.latent_embed(e)


def test_plain_values_take_the_kernel(stage):
    assert stage.noise_embedding(T).isnan().all()


def test_forward_mode_keeps_its_tangent(stage):
    with forward_ad.dual_level():
        got = forward_ad.unpack_dual(stage.noise_embedding(forward_ad.make_dual(T, torch.ones(2))))
        want = forward_ad.unpack_dual(_formulas(stage, forward_ad.make_dual(T, torch.ones(2))))
    assert torch.equal(got.primal, want.primal) and torch.equal(got.tangent, want.tangent)
    assert want.tangent.abs().max() > 0.01


def test_function_transforms_take_the_formulas(stage):
    jac = torch.func.jacfwd(lambda t: _formulas(stage, t))(T)
    torch.testing.assert_close(torch.func.jacfwd(stage.noise_embedding)(T), jac)
    torch.testing.assert_close(torch.func.jacrev(stage.noise_embedding)(T), jac)
    got = torch.func.vmap(stage.noise_embedding)(T.view(2, 1))
    torch.testing.assert_close(got, _formulas(stage, T).view(2, 1, -1))


def test_reverse_mode_takes_the_formulas(stage):
    t = T.clone().requires_grad_()
    stage.noise_embedding(t).sum().backward()
    assert t.grad.isfinite().all() and t.grad.abs().min() > 0
