"""Epilogues of the two-CTA GEMM that request their second operand (u = [gate | up], or the residual) one step ahead."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 4e-3      # one rounding to bf16 of the result (2^-9 at most), and of the products' operands' share in it


@pytest.mark.parametrize("M,F,D", [(1, 256, 64), (257, 512, 128), (300, 2176, 256), (31, 2048, 192), (19000, 768, 768)])
@pytest.mark.parametrize("in_place", [False, True])
def test_swiglu_backward(M, F, D, in_place):
    """Row and column remainders (2176: the last tile is half empty, one of the two warps of a row has nothing to do there),
    more tiles than CTA pairs, and the gradient written over the operand."""
    from aeris_gb_b200.ops import gemm as G
    torch.manual_seed(M)
    dy, w2 = torch.randn(M, D, device=DEV).bfloat16(), (torch.randn(D, F, device=DEV) * D ** -0.5).bfloat16()
    u = torch.randn(M, 2 * F, device=DEV).bfloat16()
    uf = u.float().requires_grad_(True)
    (torch.nn.functional.silu(uf[:, :F]) * uf[:, F:]).backward(dy.float() @ w2.float())
    du = u if in_place else torch.empty_like(u)
    G.gemm(dy, w2, b_t=True, out=du, epi=G.EPI_SWIGLU_BWD, resid=u)
    assert rel_err(du, uf.grad) < TOL


@pytest.mark.parametrize("M,N,K,per", [(1, 256, 64, 0), (255, 512, 192, 85), (300, 2176, 256, 100), (31, 2048, 1024, 0),
                                       (19000, 768, 768, 9500), (600, 512, 1088, 0)])
@pytest.mark.parametrize("in_place", [False, True])
def test_gated_residual(M, N, K, per, in_place):
    """As above, with gates per group of rows, on both sides of the line (reductions up to 1024 request ahead)."""
    from aeris_gb_b200.ops import gemm as G
    torch.manual_seed(M)
    a, b = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) * K ** -0.5).bfloat16()
    x = torch.randn(M, N, device=DEV).bfloat16()
    rows = per or M
    gate = torch.randn(-(-M // rows), N, device=DEV)
    ref = x.float() + gate.repeat_interleave(rows, 0)[:M] * (a.float() @ b.float().t())
    y = x if in_place else torch.empty_like(x)
    G.gemm(a, b, out=y, epi=G.EPI_GATE_RESID, resid=x, gate=gate, rows_per_gate=per)
    assert rel_err(y, ref) < TOL
