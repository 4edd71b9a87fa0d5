"""Two-CTA GEMM: bf16 outputs leave as tiled stores of 32 rows. Rows that end inside a tile of 32, inside a CTA's and a
pair's rows, a last column tile that is half empty, outputs that are slices of wider tensors (nothing beside them is written),
short and long reductions (eight and four epilogue warps), the SwiGLU backward in place."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _wide(rows, cols):
    """A [rows, cols] slice of a larger tensor of sevens, and a check that only the slice was written."""
    w = torch.full((rows + 8, cols + 32), 7.0, device=DEV, dtype=torch.bfloat16)

    def untouched():
        return all(float((x - 7).abs().max()) == 0 for x in (w[rows:], w[:rows, :16], w[:rows, 16 + cols:]))
    return w[:rows, 16:16 + cols], untouched


# a bf16 result of fp32 sums: half a unit in the last place, 2^-9, about half of that in the 2-norm
TOL = 4e-3


@pytest.mark.parametrize("M", [1, 31, 33, 128, 129, 257, 700])
@pytest.mark.parametrize("K", [64, 768, 2624])
@pytest.mark.parametrize("N,F", [(256, 256), (2176, 2176)])
def test_outputs(M, N, F, K):
    from aeris_gb_b200.ops import gemm as G
    torch.manual_seed(M + K)
    r = lambda *s: torch.randn(*s, device=DEV).bfloat16()
    a, b, x, g = r(M, K), r(N, K), r(M, N), torch.randn(1, N, device=DEV)
    c, ok = _wide(M, N)
    ref = a.double() @ b.double().t()
    G.gemm(a, b, out=c, two_cta=True)
    assert rel_err(c, ref) < TOL and ok()
    c, ok = _wide(M, N)
    G.gemm(a, b, out=c, epi=G.EPI_GATE_RESID, resid=x, gate=g, two_cta=True)
    assert rel_err(c, x.double() + g.double() * ref) < TOL and ok()
    # SwiGLU: gate and up rows of the weights, activation and raw columns
    f = F if F % 256 == 0 else 256
    w = r(2 * f, K)
    u = a.double() @ w.double().t()
    act, ok = _wide(M, f)
    raw, ok2 = _wide(M, 2 * f)
    G.gemm(a, w, out=act, epi=G.EPI_SWIGLU_BOTH, aux=raw, two_cta=True)
    assert rel_err(act, torch.nn.functional.silu(u[:, :f]) * u[:, f:]) < TOL and rel_err(raw, u) < TOL and ok() and ok2()
    act2, ok = _wide(M, f)
    G.gemm(a, w, out=act2, epi=G.EPI_SWIGLU, two_cta=True)
    assert torch.equal(act2, act) and ok()
    # its backward: d(act) = a b^T over N columns, operand u and gradient in place
    du, ok = _wide(M, 2 * N)
    uu = r(M, 2 * N)
    du.copy_(uu)
    G.gemm(a, b.t().contiguous(), b_t=True, out=du, epi=G.EPI_SWIGLU_BWD, resid=du, two_cta=True)
    ud = uu.double().requires_grad_(True)
    (torch.nn.functional.silu(ud[:, :N]) * ud[:, N:]).backward(ref)
    assert rel_err(du, ud.grad) < TOL and ok()
