"""A kernel behind one that gave up keeps its results to itself, also where it started while that one was still running. Here
the word that tells it is part of what a long product of one tile writes: zero while the kernel behind it starts on the other
multiprocessors, not zero when its turn comes."""
import ctypes

import pytest
import torch

from aeris_gb_b200.ops import gemm as G
from aeris_gb_b200.ops import lib as L

pytestmark = pytest.mark.gpu
V = ctypes.c_void_p
K_LONG = 1 << 18                # 4,096 steps of 64, one after the other
SENTINEL = 2.0 ** 100


def _gemm(a, b, c, status, epi, bn=0):
    M, K = a.shape
    N = b.shape[0]
    return lambda: L.lib().aeris_gemm_auto(
        L.ptr(a), L.ptr(b), L.ptr(c), M, N, K, K, K, N, 0, 0, epi, V(0), 0, V(0), 0, 0, V(0), 0, 0, 1, bn, 0, status,
        L.stream_ptr())


def _behind_a_failure(make):
    """``make(status)``: (a launch, its outputs); the launch is issued right behind the long product."""
    one = torch.ones(128, K_LONG, dtype=torch.bfloat16, device="cuda")
    word = torch.zeros(128, 128, device="cuda")
    first = _gemm(one, one, word, V(0), G.EPI_STORE_F32)
    launch, outs = make(L.ptr(word))
    assert first() == 0 and word.zero_() is word and launch() == 0         # both are loaded: no pause between them below
    word.zero_()
    for o in outs:
        o.fill_(SENTINEL)
    torch.cuda.synchronize()
    rcs = (first(), launch())
    torch.cuda.synchronize()
    assert rcs == (0, 0) and bool((word == K_LONG).all())
    for o in outs:
        assert bool((o == SENTINEL).all())
    # and with nothing wrong before it the same launch writes
    word.zero_()
    assert launch() == 0
    torch.cuda.synchronize()
    for o in outs:
        assert not bool((o == SENTINEL).any())


@pytest.mark.parametrize("N,bn", [(128, 0), (256, 128), (256, 256)])
def test_product(N, bn):
    a, b = (torch.randn(n, 256, device="cuda").bfloat16() for n in (4096, N))
    c = torch.empty(4096, N, device="cuda")
    _behind_a_failure(lambda status: (_gemm(a, b, c, status, G.EPI_STORE_F32, bn), [c]))


def _attention(n_win, N, H, d):
    qkv = torch.randn(n_win * N, 3 * H * d, device="cuda").bfloat16()
    o = torch.empty(n_win * N, H * d, dtype=torch.bfloat16, device="cuda")
    return qkv, o, torch.empty(n_win, H, N, device="cuda")


# one query tile, two in turn, four at a time
@pytest.mark.parametrize("n_win,N,H,d", [(8, 100, 2, 64), (8, 100, 2, 128), (8, 250, 2, 64), (8, 200, 2, 128),
                                         (50, 300, 2, 64)])
def test_attention_forward(n_win, N, H, d):
    qkv, o, lse = _attention(n_win, N, H, d)
    ld, p = 3 * H * d, L.ptr
    _behind_a_failure(lambda status: (lambda: L.lib().aeris_attn_fwd(
        p(qkv), ld, 0, p(qkv), ld, H * d, p(qkv), ld, 2 * H * d, p(o), H * d, p(lse), n_win, N, H, d, ctypes.c_float(0.125),
        status, L.stream_ptr()), [o, lse]))


@pytest.mark.parametrize("n_win,N,H,d", [(8, 100, 2, 64), (8, 300, 2, 128)])
def test_attention_backward(n_win, N, H, d):
    qkv, o, lse = _attention(n_win, N, H, d)
    o.normal_(), lse.fill_(4.0)
    d_o, delta, g = torch.randn_like(o), torch.empty_like(lse), torch.empty_like(qkv)
    ld, p = 3 * H * d, L.ptr
    _behind_a_failure(lambda status: (lambda: L.lib().aeris_attn_bwd(
        p(qkv), ld, 0, H * d, 2 * H * d, p(o), p(d_o), H * d, p(lse), p(delta), p(g), ld, n_win, N, H, d, ctypes.c_float(0.125),
        status, L.stream_ptr()), [g]))         # delta is scratch
