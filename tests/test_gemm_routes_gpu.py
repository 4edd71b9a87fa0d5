"""Which GEMM kernel takes a product is decided by its size alone: sizes on both sides of every line (one wave of tiles or
several, half-empty last tiles, short and long sums), on the route that they take and on the other one, against 64 bits."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 4e-3      # a bf16 result of fp32 sums: half a unit in the last place, 2^-9, about half of that in the 2-norm


@pytest.mark.parametrize("M,N,K,plain,swiglu,bwd,wgrad", [
    (1, 128, 128, "one", None, "pairs", "one"),
    (248, 256, 384, "one", "one", "pairs", "pairs"),
    (3600, 512, 392, "one", "pairs", "pairs", "pairs"),
    (9480, 384, 896, "one", None, "pairs", "one"),          # two waves of either
    (9473, 256, 256, "pairs", "one", "pairs", "pairs"),     # 150 small tiles: two waves against one
    (28799, 384, 64, "pairs", None, "pairs", "one"),        # five against four
    (136, 2176, 384, "one", None, "pairs", "pairs"),
    (384, 640, 20000, "one", None, "pairs", "pairs")])
def test_products(M, N, K, plain, swiglu, bwd, wgrad):
    from aeris_gb_b200.ops import gemm as G
    from aeris_gb_b200.ops.lib import lib
    torch.manual_seed(M)
    r = lambda *s: torch.randn(*s, device=DEV).bfloat16()
    a, b, x, g = r(M, K), r(N, K), r(M, N), torch.randn(1, N, device=DEV)
    bt = b.t().contiguous()
    for epi, path in ((G.EPI_STORE, plain), (G.EPI_STORE_F32, plain), (G.EPI_GATE_RESID, plain), (G.EPI_SWIGLU, swiglu),
                      (G.EPI_SWIGLU_BWD, bwd), (G.EPI_ACC_F32, wgrad)):
        if path:
            assert lib().aeris_gemm_takes_pairs(M, N, K, epi, 1) == (path == "pairs")
            assert lib().aeris_gemm_takes_pairs(M, N, K, epi, 2) and not lib().aeris_gemm_takes_pairs(M, N, K, epi, 0)
    ref = a.double() @ b.double().t()
    for route in (None, False, True):
        kw = dict(two_cta=route)
        c = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)

        def check(out, want, tol=TOL):
            assert rel_err(out, want) < tol
        check(G.gemm(a, b, out=c, **kw), ref)
        check(G.gemm(a, bt, b_t=True, out=c, **kw), ref)
        # fp32 sums of K products of bf16 values, exact each
        check(G.gemm(a, b, epi=G.EPI_STORE_F32, **kw), ref, 2.0 ** -23 * K ** 0.5 * 4)
        check(G.gemm(a, b, out=c, epi=G.EPI_GATE_RESID, resid=x, gate=g, **kw), x.double() + g.double() * ref)
        u, du = r(M, 2 * N), torch.empty(M, 2 * N, device=DEV, dtype=torch.bfloat16)
        ud = u.double().requires_grad_(True)
        (torch.nn.functional.silu(ud[:, :N]) * ud[:, N:]).backward(ref)
        check(G.gemm(a, bt, b_t=True, out=du, epi=G.EPI_SWIGLU_BWD, resid=u, **kw), ud.grad)
        if swiglu:
            act = torch.empty(M, N // 2, device=DEV, dtype=torch.bfloat16)
            check(G.gemm(a, b, out=act, epi=G.EPI_SWIGLU, **kw), torch.nn.functional.silu(ref[:, :N // 2]) * ref[:, N // 2:])
        # [M, N] += [K, M]^T [K, N]
        at, w = a.t().contiguous() if M % 8 == 0 else None, torch.zeros(M, N, device=DEV)
        if at is not None:
            check(G.gemm(at, bt, a_t=True, b_t=True, out=w, epi=G.EPI_ACC_F32, k_splits=0, **kw), ref,
                  2.0 ** -23 * K ** 0.5 * 4)
