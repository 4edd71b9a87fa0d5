"""Attention forward of windows longer than one query tile (two tiles at a time, K and V in tiles of 128 rows) at the sizes
where it can go wrong: one row or one 16-column step more or less than a tile, a second chain without rows, a last tile of a
few columns or of more than half, more items than CTAs."""
import math

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"
# P and the result are rounded to bf16 (2^-9 each at most, half of that in the 2-norm of many): 4e-3 bounds their sum
TOL = 4e-3


def _reference(qkv, nw, N, H, d, scale=None):
    q, k, v = qkv.double().view(nw, N, 3, H, d).permute(2, 0, 3, 1, 4)
    s = (q @ k.transpose(-1, -2)) * (scale if scale is not None else 1 / math.sqrt(d))
    return (s.softmax(-1) @ v).permute(0, 2, 1, 3).reshape(nw * N, H * d), torch.logsumexp(s, -1) / math.log(2)


@pytest.mark.parametrize("d", [64, 128, 40])
@pytest.mark.parametrize("nw,N,H", [(2, 128, 3), (2, 129, 3), (1, 144, 2), (2, 160, 3), (2, 192, 3), (2, 193, 3),
                                    (3, 225, 64), (2, 255, 3), (2, 256, 3), (2, 257, 3), (1, 352, 2), (1, 353, 2),
                                    (1, 384, 2), (1, 385, 2), (1, 513, 160), (1, 641, 2), (1, 900, 2)])
def test_forward_at_the_edges_of_its_tiles(nw, N, H, d):
    from aeris_gb_b200.ops import attention as A
    torch.manual_seed(N + d)
    qkv = torch.randn(nw * N, 3 * H * d, device=DEV)
    qkv[:, :H * d] *= 8 * torch.rand(nw * N, 1, device=DEV)          # flat and sharp rows: the reference maximum is raised
    qkv = qkv.bfloat16()
    # the output is a column slice: nothing beside it may be written
    wide = torch.full((nw * N, H * d + 16), 7.0, device=DEV, dtype=torch.bfloat16)
    o, lse = A.attn_fwd(qkv, nw, N, H, d, out=wide[:, 8:8 + H * d])
    ref, lref = _reference(qkv, nw, N, H, d)
    assert rel_err(o, ref) < TOL
    assert (lse - lref).abs().max().item() < 1e-3
    assert float((wide[:, :8] - 7).abs().max()) == 0 and float((wide[:, 8 + H * d:] - 7).abs().max()) == 0


@pytest.mark.parametrize("d", [64, 128, 40])
@pytest.mark.parametrize("N", [129, 132, 133, 160, 225, 255, 256, 320, 384, 448, 700, 900, 1025])
def test_forward_equals_the_kernel_that_sees_64_columns(N, d):
    """Two query tiles at a time over 128 columns give what the kernel of one query tile over 64 columns gives, bit for bit,
    as long as no row's maximum is raised in the second half of a tile (scores of N(0, 1) stay far below 2^8)."""
    from aeris_gb_b200.ops import attention as A, lib as L
    torch.manual_seed(N)
    nw, H = 3, 60
    qkv = torch.randn(nw * N, 3 * H * d, device=DEV).bfloat16()
    o, lse = A.attn_fwd(qkv, nw, N, H, d)
    assert L.lib().aeris_attn_set_fwd_variant(-1, 1) == 0        # the same arithmetic, one query tile at a time
    try:
        ref, lref = A.attn_fwd(qkv, nw, N, H, d)
        torch.cuda.synchronize()
    finally:
        L.lib().aeris_attn_set_fwd_variant(-1, 0)
    assert torch.equal(o, ref) and torch.equal(lse, lref)


@pytest.mark.parametrize("N", [100, 300])
@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_forward_with_a_scale_that_is_not_positive(N, scale):
    """Masked columns carry -inf, which only a positive scale turns into probability 0: other scales take the kernel for
    short windows."""
    from aeris_gb_b200.ops import attention as A
    qkv = torch.randn(2 * N, 3 * 2 * 64, device=DEV).bfloat16()
    o, _ = A.attn_fwd(qkv, 2, N, 2, 64, scale=scale)
    assert rel_err(o, _reference(qkv, 2, N, 2, 64, scale)[0]) < TOL


@pytest.mark.parametrize("N,d,keep", [(450, 64, True), (260, 128, False), (256, 64, False)])
def test_forward_pushes_the_rows_to_their_owners(N, d, keep):
    """The Ulysses push with both owners' buffers on this GPU: the same rows as without it, bit for bit."""
    import ctypes
    from aeris_gb_b200.ops import attention as A, lib as L
    nw, H, sp = 3, 2, 2
    n_loc, HD = N // sp, H * d
    qkv = torch.randn(nw * N, 3 * HD, device=DEV).bfloat16()
    ref, lref = A.attn_fwd(qkv, nw, N, H, d)
    bufs = [torch.zeros(nw * n_loc, 2 * HD, device=DEV, dtype=torch.bfloat16) for _ in range(sp)]
    o = torch.empty_like(ref) if keep else None
    lse = torch.empty_like(lref)
    arr = (ctypes.c_void_p * sp)(*[b.data_ptr() for b in bufs])
    rc = L.lib().aeris_attn_fwd_push(L.ptr(qkv), 3 * HD, H, L.ptr(o), HD, L.ptr(lse), nw, N, d,
                                     ctypes.c_float(1 / math.sqrt(d)), arr, sp, n_loc, 2 * HD, HD, L.ptr(L.status_word()),
                                     L.stream_ptr())
    assert rc == 0
    got = torch.stack([b.view(nw, n_loc, 2 * HD) for b in bufs], 1).reshape(nw * N, 2 * HD)
    assert torch.equal(got[:, HD:], ref) and float(got[:, :HD].abs().max()) == 0
    assert torch.equal(lse, lref) and (o is None or torch.equal(o, ref))
