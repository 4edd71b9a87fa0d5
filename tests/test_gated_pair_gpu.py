"""What a block's backward pass does with its two gated matrices before and after a sample's products, against 64 bits."""
import pytest
import torch

from aeris_gb_b200.ops import lib as L

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -24


@pytest.mark.parametrize("R,C2,Co", [(1, 8, 8), (3, 8, 2048), (130, 1032, 40), (257, 4096, 1536), (1536, 384, 4104)])
def test_gated_matrices(R, C2, Co):
    torch.manual_seed(R)
    P, st = L.ptr, L.stream_ptr()
    W = [torch.randn(R, c, device=DEV).bfloat16() for c in (C2, Co)]
    g = [torch.randn(R, device=DEV) for _ in W]
    Wg, G = [torch.full_like(w, 7) for w in W], [torch.full(w.shape, 7.0, device=DEV) for w in W]
    zero = torch.full((6 * R + 2,), 7.0, device=DEV)
    rc = L.lib().aeris_gate_prepare(P(W[0]), P(g[0]), P(Wg[0]), P(G[0]), C2, P(W[1]), P(g[1]), P(Wg[1]), P(G[1]), Co, R,
                                    P(zero), 6 * R, st)
    assert rc == 0
    for w, gi, wg, Gi in zip(W, g, Wg, G):
        exact = w.double() * gi.double()[:, None]
        # the fp32 product and one rounding to bf16 (eight significant bits)
        assert ((wg.double() - exact).abs() <= exact.abs() * (2.0 ** -8 + 2 * U)).all()
        assert float(Gi.abs().max()) == 0
    assert float(zero[:6 * R].abs().max()) == 0 and float((zero[6 * R:] - 7).abs().max()) == 0
    G = [torch.randn(w.shape, device=DEV) for w in W]
    dW, dg = [torch.randn(w.shape, device=DEV) for w in W], [torch.randn(R, device=DEV) for _ in W]
    dW0, dg0 = [t.clone() for t in dW], [t.clone() for t in dg]
    rc = L.lib().aeris_gate_finalize_pair(P(G[0]), P(W[0]), P(g[0]), P(dW[0]), P(dg[0]), C2, P(G[1]), P(W[1]), P(g[1]),
                                          P(dW[1]), P(dg[1]), Co, R, st)
    assert rc == 0
    for w, gi, Gi, a, a0, b, b0 in zip(W, g, G, dW, dW0, dg, dg0):
        add = gi.double()[:, None] * Gi.double()
        assert ((a.double() - a0.double() - add).abs() <= U * (add + a0.double()).abs() + 1e-30).all()      # one fma
        terms = w.double() * Gi.double()
        # a sum of C products in any order, and the addition to what was there
        tol = (w.shape[1] + 2) * U * terms.abs().sum(1) + U * (b0.double() + terms.sum(1)).abs()
        assert ((b.double() - b0.double() - terms.sum(1)).abs() <= tol).all()
