"""Which modulation MLPs run on the GEMV kernel."""
import pytest
import torch

from aeris_gb_b200.models import fused
from aeris_gb_b200.ops import diffusion as DF


@pytest.mark.parametrize("B,K,ok", [(1, 5120, True), (3, 5120, True), (8, 5120, True), (8, 6400, True), (5, 6401, False),
                                    (4, 12800, True), (3, 12801, False), (8, 8192, False), (9, 16, False)])
def test_rows_that_the_kernel_takes(B, K, ok):
    assert DF.gemv_ok(B, K) == ok


@pytest.mark.parametrize("B,dims", [(9, (16, 16)), (8, (8192,)), (8, (16, 8192))])
def test_modulation_the_kernel_does_not_take_runs_on_stock_operators(B, dims, monkeypatch):
    """Too many samples, or rows too wide for the kernel in either layer: the module itself, not an error."""
    monkeypatch.setattr(fused.GemvLinearFn, "apply", lambda *a: pytest.fail("kernel route"))
    linear = [torch.nn.Linear(k, n) for k, n in zip(dims, (*dims[1:], 12))]
    seq = torch.nn.Sequential(linear[0], torch.nn.SiLU(), *linear[1:]) if len(dims) == 2 else \
        torch.nn.Sequential(torch.nn.SiLU(), linear[0])
    emb = torch.randn(B, dims[0])
    assert torch.equal(fused.modulation(seq, emb), seq(emb).float())
