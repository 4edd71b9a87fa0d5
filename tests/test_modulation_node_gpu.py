"""The modulation MLP as one autograd node: all five gradients against 64 bits, with and without an engine's buffers."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,K,N1,N2", [(1, 64, 128, 96), (2, 1536, 1536, 70), (3, 100, 260, 1552), (8, 256, 64, 1536),
                                       (2, 101, 64, 40), (2, 64, 101, 40)])      # 101: a layer on the PyTorch formulas
@pytest.mark.parametrize("target", [None, "whole", "strided"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradients(B, K, N1, N2, target, dtype):
    from aeris_gb_b200.models.fused import ModulationFn
    torch.manual_seed(K)
    params = [torch.nn.Parameter((torch.randn(*s, device=DEV) * s[-1] ** -0.5).to(dtype))
              for s in ((N1, K), (N1,), (N2, N1), (N2,))]
    x = torch.randn(B, K, device=DEV, requires_grad=True)
    dy = torch.randn(B, N2, device=DEV)
    if target is not None:
        for p in params:        # strided: every second column, the PyTorch formulas
            p.main_grad = torch.ones((*p.shape, 2), device=DEV)[..., 0]
            if target == "whole":
                p.main_grad = p.main_grad.contiguous()
    y = ModulationFn.apply(x, *params)
    y.backward(dy)
    ex = [t.detach().double().requires_grad_(True) for t in (x, *params)]
    W1, b1, W2, b2 = ex[1:]
    ref = torch.nn.functional.silu(ex[0] @ W1.t() + b1) @ W2.t() + b2
    ref.backward(dy.double())
    # fp32 sums of K (N1, N2) terms, fast exponentials in the SiLU, as for the single layers
    tol = 4e-6
    assert rel_err(y, ref) < tol and rel_err(x.grad, ex[0].grad) < tol
    for p, e in zip(params, ex[1:]):
        if target is None:
            assert rel_err(p.grad, e.grad) < (tol if dtype == torch.float32 else 3e-3)       # rounded to bf16 at the end
        else:
            assert p.grad is None
            assert rel_err(p.main_grad, e.grad + 1) < tol
