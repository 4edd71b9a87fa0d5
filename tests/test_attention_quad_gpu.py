"""Attention forward, four query tiles at a time: windows of three, four, seven and eight tiles whose last tile, last 64
columns and last step of 16 are full, nearly full or nearly empty, groups with an idle chain, one and several items a CTA.
The output is that of the kernel of one query tile, bit for bit."""
import math

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _quad_ran(fn):
    from torch.profiler import ProfilerActivity, profile
    for _ in range(5):                  # a profile now and then comes back empty
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            out = fn()
            torch.cuda.synchronize()
        names = [e.name for e in prof.events() if "attn_fwd" in e.name]
        if names:
            return out, any("attn_fwd_quad_kernel" in n for n in names)
    raise AssertionError("no attention kernel in any profile")


# 96 (window, head) pairs of 3 or 4 tiles and 74 of 7 or 8 are one item a CTA, 296 and 222 several
@pytest.mark.parametrize("d", [64, 40])
@pytest.mark.parametrize("nw,N,H", [(3, 257, 32), (3, 272, 32), (3, 320, 32), (3, 321, 32), (3, 383, 32), (3, 384, 32),
                                    (3, 385, 32), (8, 450, 37), (3, 512, 32), (2, 769, 37), (6, 831, 37), (2, 895, 37),
                                    (2, 896, 37),
                                    (6, 900, 37), (2, 1024, 37)])
@pytest.mark.parametrize("sharp", [False, True])
def test_equals_the_kernel_of_one_query_tile(nw, N, H, d, sharp):
    from aeris_gb_b200.ops import attention as A, lib as L
    torch.manual_seed(N + d)
    qkv = torch.randn(nw * N, 3 * H * d, device=DEV)
    if sharp:                      # flat and sharp rows: the reference maximum is raised, in any tile
        qkv[:, :H * d] *= 8 * torch.rand(nw * N, 1, device=DEV)
    qkv = qkv.bfloat16()
    # the output is a column slice: nothing beside it may be written
    wide = torch.full((nw * N, H * d + 16), 7.0, device=DEV, dtype=torch.bfloat16)
    (o, lse), quad = _quad_ran(lambda: A.attn_fwd(qkv, nw, N, H, d, out=wide[:, 8:8 + H * d]))
    L.check_status()
    assert quad
    assert L.lib().aeris_attn_set_fwd_variant(-1, 1) == 0        # the same arithmetic, one query tile at a time
    try:
        ref, lref = A.attn_fwd(qkv, nw, N, H, d)
        torch.cuda.synchronize()
    finally:
        L.lib().aeris_attn_set_fwd_variant(-1, 0)
    assert torch.equal(o, ref) and torch.equal(lse, lref)
    assert float((wide[:, :8] - 7).abs().max()) == 0 and float((wide[:, 8 + H * d:] - 7).abs().max()) == 0
    # P and the result are rounded to bf16 (2^-9 each at most, half of that in the 2-norm of many): 4e-3 bounds their sum
    q, k, v = qkv[:N].double().view(N, 3, H, d).permute(1, 2, 0, 3)
    want = ((q @ k.transpose(-1, -2) / math.sqrt(d)).softmax(-1) @ v).permute(1, 0, 2).reshape(N, H * d)
    assert rel_err(o[:N], want) < 4e-3


@pytest.mark.parametrize("keep", [True, False])
def test_pushes_the_rows_to_their_owners(keep):
    """The Ulysses push with both owners' buffers on this GPU: the same rows as without it, bit for bit."""
    import ctypes
    from aeris_gb_b200.ops import attention as A, lib as L
    nw, N, H, d, sp = 3, 450, 32, 64, 2
    n_loc, HD = N // sp, H * d
    qkv = torch.randn(nw * N, 3 * HD, device=DEV).bfloat16()
    ref, lref = A.attn_fwd(qkv, nw, N, H, d)
    bufs = [torch.zeros(nw * n_loc, 2 * HD, device=DEV, dtype=torch.bfloat16) for _ in range(sp)]
    o = torch.empty_like(ref) if keep else None
    lse = torch.empty_like(lref)
    arr = (ctypes.c_void_p * sp)(*[b.data_ptr() for b in bufs])
    rc, quad = _quad_ran(lambda: L.lib().aeris_attn_fwd_push(
        L.ptr(qkv), 3 * HD, H, L.ptr(o), HD, L.ptr(lse), nw, N, d, ctypes.c_float(1 / math.sqrt(d)), arr, sp, n_loc, 2 * HD,
        HD, L.ptr(L.status_word()), L.stream_ptr()))
    assert rc == 0 and quad
    got = torch.stack([b.view(nw, n_loc, 2 * HD) for b in bufs], 1).reshape(nw * N, 2 * HD)
    assert torch.equal(got[:, HD:], ref) and float(got[:, :HD].abs().max()) == 0
    assert torch.equal(lse, lref) and (o is None or torch.equal(o, ref))
