"""Extents that the attention backward kernels cannot count in 32 bits are refused before anything is launched."""
import pytest

from aeris_gb_b200.ops.lib import lib

SMS = 148


@pytest.mark.parametrize("d,bt", [(32, 96), (64, 96), (72, 64), (128, 64)])
def test_tiles_that_one_cta_streams(d, bt):
    """Rows of 128 per item, `bt` per streamed tile: a CTA's share of the products of both has to stay below 2^31."""
    taken = refused = 0
    for n_win in (1, 3, 64, 65535):
        for H in (1, 24, 65535):
            for N in (1, 64, 900, 3600, 1 << 16, 1 << 20, 1 << 24, (1 << 31) - 1):
                items = -(-N // 128) * H * n_win
                per_cta = -(-items // min(items, SMS)) * -(-N // bt)
                got = lib().aeris_attn_bwd_countable(n_win, N, H, d, SMS)
                if got:
                    assert items < 2 ** 31 and per_cta < 2 ** 31
                else:
                    assert items > 2 ** 29 or per_cta > 2 ** 29           # no more than what comes near is refused
                taken += got
                refused += not got
    assert taken and refused


def test_extents_in_use():
    for n_win, N, H, d in ((1152, 900, 24, 64), (288, 3600, 40, 128), (65535, 64, 64, 64), (1, 1 << 20, 24, 64)):
        assert lib().aeris_attn_bwd_countable(n_win, N, H, d, SMS)


def test_more_tiles_than_32_bits_count():
    """2,048 windows of 2^19 rows: 8,388,608 items of 5,462 tiles each, 309 million a CTA; of 2^22 rows, 20 billion."""
    assert lib().aeris_attn_bwd_countable(2048, 1 << 19, 1, 64, SMS)
    assert not lib().aeris_attn_bwd_countable(2048, 1 << 22, 1, 64, SMS)
