"""CTA pairs that give up because another kernel has. A wait that has gone on for some 15 us looks for that; sums of 4096 out
of memory take longer for part of the tiles. The pairs leave with nothing under way, and the launch behind them finds all as it
should be. (Waits of products with requests ahead are shorter than that: their way out has not been seen.)"""
import ctypes

import pytest
import torch

from aeris_gb_b200.ops import gemm as G
from aeris_gb_b200.ops import lib as L
from conftest import rel_err

pytestmark = pytest.mark.gpu
V = ctypes.c_void_p
TOL = 4e-3      # one rounding to bf16 of the result


@pytest.mark.parametrize("epi", [G.EPI_STORE, G.EPI_GATE_RESID, G.EPI_SWIGLU_BWD])
def test_a_launch_behind_pairs_that_gave_up(epi):
    torch.manual_seed(0)
    M, N, K, dev = 256 * 74 * 2 + 100, 256, 4096, "cuda"
    bwd = epi == G.EPI_SWIGLU_BWD
    a = torch.randn(M, K, device=dev).bfloat16()
    b = (torch.randn(*((K, N) if bwd else (N, K)), device=dev) * K ** -0.5).bfloat16()
    x = torch.randn(M, 2 * N if bwd else N, device=dev).bfloat16()
    gate = torch.randn(1, N, device=dev)
    prod = a.float() @ (b.float() if bwd else b.float().t())
    if epi == G.EPI_STORE:
        ref = prod
    elif epi == G.EPI_GATE_RESID:
        ref = x.float() + gate * prod
    else:
        u = x.float().requires_grad_(True)
        (torch.nn.functional.silu(u[:, :N]) * u[:, N:]).backward(prod)
        ref = u.grad
    out, word = torch.empty_like(x), torch.zeros(1, dtype=torch.int32, device=dev)
    flush = torch.empty(64 << 20, device=dev)

    def launch():
        rc = L.lib().aeris_gemm_auto(
            L.ptr(a), L.ptr(b), L.ptr(out), M, N, K, K, b.stride(0), out.stride(0), 0, int(bwd), epi,
            V(0) if epi == G.EPI_STORE else L.ptr(x), x.stride(0), L.ptr(gate), M, N, V(0), 0, N if bwd else 0, 1, 0, 2,
            L.ptr(word), L.stream_ptr())
        assert rc == 0

    for i in range(4):
        word.fill_(1)
        flush.fill_(float(i))          # nothing of the operands is in L2
        launch()
        torch.cuda.synchronize()
        assert int(word) == 1          # the first failure stays on record
        out.zero_(), word.zero_()
        launch()
        torch.cuda.synchronize()
        assert int(word) == 0 and rel_err(out, ref) < TOL
