"""Weight gradients that ask for slices: the choice between the two GEMM kernels never makes a sum's slices longer than those of
the kernel with single CTAs, whose error they bound."""
import pytest
import torch

from aeris_gb_b200.ops.lib import lib

SMS = 148


def _cd(a, b):
    return -(-a // b)


def _slice(M, N, K, want, pairs):
    """Rows per slice, in blocks of 64."""
    kb, side = _cd(K, 64), 256 if pairs else 128
    s = lib().aeris_choose_k_splits(_cd(M, side) * _cd(N, side), kb, SMS // 2 if pairs else SMS, 64 if pairs else 4, want)
    return _cd(kb, s)


def test_pairs_never_lengthen_the_slices():
    taken = kept = 0
    for M in range(128, 4097, 128):
        for N in range(128, 2048, 256):                 # wider ones and whole tiles of 256 are the pairs' in any case
            for K in (1600, 4096, 12150, 20000, 28800, 53550, 64800):
                for want in (1, 4, 16, 60, 240):
                    shorter = _slice(M, N, K, want, True) <= _slice(M, N, K, want, False)
                    pays = lib().aeris_gemm_takes_pairs(M, N, K, 3, 1)
                    assert lib().aeris_wgrad_takes_pairs(M, N, K, -want, SMS) == (pays and shorter), (M, N, K, want)
                    taken += pays and shorter
                    kept += pays and not shorter
                assert lib().aeris_wgrad_takes_pairs(M, N, K, 0, SMS) == lib().aeris_gemm_takes_pairs(M, N, K, 3, 1)
    assert taken and kept


def test_whole_tiles_as_before():
    for M, N, K, want in ((384, 256, 53550, 240), (384, 2176, 28800, 60), (128, 2048, 1600, 4)):
        assert lib().aeris_wgrad_takes_pairs(M, N, K, -want, SMS) == 1
    assert lib().aeris_wgrad_takes_pairs(384, 192, 53550, -4, SMS) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,want", [(1152, 384, 53550, 60), (1152, 384, 20250, 16), (384, 384, 53550, 240),
                                        (384, 384, 28800, 60), (1792, 384, 28800, 240), (384, 896, 64800, 16)])
def test_error_against_64_bits(M, N, K, want):
    from aeris_gb_b200.ops import gemm as G
    torch.manual_seed(K)
    a, b = torch.randn(K, M, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    ref = a.double().t() @ b.double()

    def error(two_cta):
        w = torch.zeros(M, N, device="cuda")
        G.gemm(a, b, a_t=True, b_t=True, out=w, epi=G.EPI_ACC_F32, k_splits=-want, two_cta=two_cta)
        return ((w - ref).norm() / ref.norm()).item()
    # the same slices on the same kernel differ by the order of their fp32 additions, a small part of the error; slices of
    # two to twelve times the rows show as that factor
    assert error(None) < 1.25 * error(False)
