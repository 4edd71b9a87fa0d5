"""Modulation vectors read in place: samples in one launch whose vectors are parts of one tensor."""
import pytest
import torch

from aeris_gb_b200.models import block as NB
from aeris_gb_b200.models import fused, fused_io
from aeris_gb_b200.ops import elementwise as E

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [8, 264, 1536, 5120, 5128])       # one to three vectors a thread, and sample by sample
@pytest.mark.parametrize("mode", [E.MODE_MOD_THEN_NORM, E.MODE_NORM_THEN_MOD])
def test_modnorm_rows_of_a_wider_tensor(D, mode):
    x = torch.randn(3 * 7, D, device=DEV).bfloat16()
    mod = torch.randn(3, 2 * D, device=DEV)
    w = torch.randn(D, device=DEV).bfloat16()
    shift, scale = mod.chunk(2, dim=1)
    kw = dict(mode=mode, eps=1e-6, batch=3)
    assert torch.equal(E.modnorm_fwd(x, scale, shift, w, **kw),
                       E.modnorm_fwd(x, scale.contiguous(), shift.contiguous(), w, **kw))


@pytest.mark.parametrize("D,heads,F", [(128, 2, 128), (256, 4, 256), (384, 6, 384)])     # both GEMM kernels' gates
@pytest.mark.parametrize("offset", [0, 1])                      # a modulation tensor off the 16-byte grid
def test_merged_samples_equal_single_ones(D, heads, F, offset):
    L, wins, B, d = 70, 2, 3, 64
    meta = fused.BlockMeta(wins, L, heads, d, E.MODE_MOD_THEN_NORM, 1e-6)
    rnd = lambda *s: (torch.randn(*s, device=DEV) * s[-1] ** -0.5).bfloat16()
    ws = (1 + rnd(D), rnd(3 * heads * d, D), rnd(D, heads * d), 1 + rnd(D), rnd(2 * F, D), rnd(D, F))
    x = torch.randn(B * wins * L, D, device=DEV).bfloat16()
    mod = torch.randn(B * 6 * D + offset, device=DEV)[offset:].view(B, 6 * D)
    assert NB.takes(meta, x, mod, ws)
    y = fused.block_forward(x, mod, meta, *ws)
    n = wins * L
    one = [fused.block_forward(x[b * n:(b + 1) * n], mod[b:b + 1].clone(), meta, *ws) for b in range(B)]
    assert torch.equal(y, torch.cat(one))


def test_head_rows_in_place_or_copied():
    mod = torch.randn(2, 2 * 64, device=DEV)
    shift, scale = mod.chunk(2, dim=1)
    assert fused_io._mod_rows(shift, scale)[1].data_ptr() == scale.data_ptr()
    for sh, sc in ((shift, scale.contiguous()), (mod[:, 1:65], mod[:, 63:127]), (shift.t().contiguous().t(), scale)):
        a, b = fused_io._mod_rows(sh, sc)
        assert a.is_contiguous() and b.is_contiguous() and torch.equal(a, sh) and torch.equal(b, sc)
