"""Attention backward: two chains of tiles (96 rows for heads up to 64, 64 above), half of a tile's columns per warpgroup.
Windows that end at and around the edges of tiles, of halves and of steps of 16, with fewer tiles than chains, and several
items a CTA, whose tiles the chains take on without a break."""
import math

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("d", [64, 24, 128])
@pytest.mark.parametrize("nw,N,H", [(320, 1, 1), (160, 16, 2), (160, 47, 2), (160, 48, 2), (160, 49, 2), (150, 95, 2),
                                    (150, 96, 2), (150, 97, 2), (80, 143, 3), (80, 145, 3), (64, 191, 3), (64, 192, 3),
                                    (64, 193, 3), (30, 288, 3), (30, 289, 3), (6, 961, 4), (1, 96, 1), (1, 17, 1)])
def test_tile_edges(nw, N, H, d):
    from aeris_gb_b200.ops import attention as A
    from aeris_gb_b200.ops import lib as L
    torch.manual_seed(N + d)
    qkv = torch.randn(nw * N, 3 * H * d, device=DEV).bfloat16()
    do = torch.randn(nw * N, H * d, device=DEV).bfloat16()
    o, lse = A.attn_fwd(qkv, nw, N, H, d)
    got = A.attn_bwd(qkv, o, do, lse, nw, N, H, d)
    again = A.attn_bwd(qkv, o, do, lse, nw, N, H, d)
    L.check_status()
    assert torch.equal(got, again)                       # no atomics
    x = qkv.double().requires_grad_(True)
    q, k, v = x.view(nw, N, 3, H, d).permute(2, 0, 3, 1, 4)
    out = (q @ k.transpose(-1, -2) / math.sqrt(d)).softmax(-1) @ v
    out.permute(0, 2, 1, 3).reshape(nw * N, H * d).backward(do.double())
    # P, dS and the results are rounded to bf16, o too, which enters dS: 2^-9 each at most, about half of that in the 2-norm
    for s in range(3):
        mine, ref = got[:, s * H * d:(s + 1) * H * d], x.grad[:, s * H * d:(s + 1) * H * d]
        if s < 2 and N == 1:        # a single key: o = v, dS = 0 but for the order of two fp32 sums over the head's width
            assert float(mine.float().abs().max()) < d * 2 ** -16
        else:
            assert rel_err(mine, ref) < 6e-3
