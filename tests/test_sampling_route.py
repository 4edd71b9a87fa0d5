"""What sampling issues without autograd nodes, and workspaces handed on by address."""
import pytest
import torch

from aeris_gb_b200.diffusion.rollout import DeviceForecaster, SamplerConfig
from aeris_gb_b200.models import aeris as A
from aeris_gb_b200.models import fused


def test_whole_buffers_are_those_behind_the_views():
    ws = fused.Workspace()
    big = ws.whole("a", (4, 6), torch.float32, "cpu")
    assert big.numel() == 24 and ws.get("a", (2, 6), torch.float32, "cpu").data_ptr() == big.data_ptr()
    assert ws.whole("a", (2, 6), torch.float32, "cpu") is big                      # never smaller than asked for
    larger = ws.whole("a", (5, 6), torch.float32, "cpu")
    assert larger is not big and larger.numel() == 30
    assert ws.whole("a", (5, 6), torch.bfloat16, "cpu").dtype == torch.bfloat16


@pytest.mark.gpu
@pytest.mark.parametrize("batch,layers", [(1, 1), (2, 2)])      # without and with the return from a shifted partition
def test_sampling_equals_the_recorded_route(batch, layers, monkeypatch):
    """The same kernels on the same values: bit for bit the same forecast."""
    cfg = A.AerisConfig(img=(32, 64), window=(8, 8), in_channels=34, out_channels=16, dim=128, heads=4, head_dim=32,
                        mlp_dim=256, n_layers=layers, sublayers=1)
    torch.manual_seed(0)
    with torch.device("cuda"):
        model = A.AerisModel(cfg).eval()
    x = torch.randn(batch, 32, 64, 16, device="cuda")
    forcing = torch.randn(batch, 32, 64, 2, device="cuda")
    stats = {k: torch.full((16,), float("std" in k), device="cuda") for k in ("x_mean", "x_std", "t_mean", "t_std")}

    def forecast():
        fc = DeviceForecaster(model, A.StreamContext(cfg, batch), stats, SamplerConfig(n_steps=2), 16, seed=3)
        return fc.step(x.clone(), forcing)

    plain = forecast()
    monkeypatch.setattr(fused, "recorded", lambda: True)
    assert torch.equal(plain, forecast())
