"""Attention backward, heads wider than 64: gradient rows leave warp by warp as tiled stores from two buffers in turn.
Windows whose last tile has rows for one to three of its four warps, several items a CTA: copies and empty groups
alternate."""
import math

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("d", [128, 72])
@pytest.mark.parametrize("nw,N,H", [(160, 129, 3), (160, 160, 3), (120, 161, 3), (120, 225, 3), (300, 31, 3), (300, 33, 3),
                                    (40, 353, 5)])
def test_gradient_rows(nw, N, H, d):
    from aeris_gb_b200.ops import attention as A
    torch.manual_seed(N + d)
    qkv = torch.randn(nw * N, 3 * H * d, device=DEV).bfloat16()
    do = torch.randn(nw * N, H * d, device=DEV).bfloat16()
    o, lse = A.attn_fwd(qkv, nw, N, H, d)
    # the gradients are a column slice: nothing beside it may be written
    wide = torch.full((nw * N, 3 * H * d + 16), 7.0, device=DEV, dtype=torch.bfloat16)
    got = A.attn_bwd(qkv, o, do, lse, nw, N, H, d, dqkv=wide[:, 8:8 + 3 * H * d])
    x = qkv.double().requires_grad_(True)
    q, k, v = x.view(nw, N, 3, H, d).permute(2, 0, 3, 1, 4)
    out = (q @ k.transpose(-1, -2) / math.sqrt(d)).softmax(-1) @ v
    out.permute(0, 2, 1, 3).reshape(nw * N, H * d).backward(do.double())
    # P, dS and the results are rounded to bf16, o too, which enters dS: 2^-9 each at most, about half of that in the 2-norm
    for s in range(3):
        assert rel_err(got[:, s * H * d:(s + 1) * H * d], x.grad[:, s * H * d:(s + 1) * H * d]) < 6e-3
    assert float((wide[:, :8] - 7).abs().max()) == 0 and float((wide[:, 8 + 3 * H * d:] - 7).abs().max()) == 0
