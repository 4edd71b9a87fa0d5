"""Attention entry points: operands that the 16-byte accesses of the kernels cannot take are refused or copied. Addresses are
made up and no launch is reached: the C entries check them before they touch the driver."""
import ctypes

import pytest
import torch

from aeris_gb_b200.ops import attention as A
from aeris_gb_b200.ops import lib as L

BASE = 1 << 20           # any 16-byte boundary
V = ctypes.c_void_p


def _fwd(d=32, o=BASE, ldo=None, n_win=2, N=10, H=2):
    ld = 3 * H * d
    return L.lib().aeris_attn_fwd(V(BASE), ld, 0, V(BASE), ld, H * d, V(BASE), ld, 2 * H * d, V(o), ldo or H * d, V(BASE),
                                  n_win, N, H, d, ctypes.c_float(1.0), V(0), V(0))


def _bwd(d=32, o=BASE, do=BASE, ldo=None, dqkv=BASE, ldg=None, H=2):
    ld = 3 * H * d
    return L.lib().aeris_attn_bwd(V(BASE), ld, 0, H * d, 2 * H * d, V(o), V(do), ldo or H * d, V(BASE), V(BASE), V(dqkv),
                                  ldg or ld, 2, 10, H, d, ctypes.c_float(1.0), V(0), V(0))


@pytest.mark.parametrize("d", [8, 32, 64, 96, 128])
@pytest.mark.parametrize("bad", [dict(o=BASE + 2), dict(o=BASE + 8), dict(ldo=2 * 128 + 4)])
def test_forward_entry_refuses_an_output_that_is_not_in_whole_vectors(d, bad):
    assert _fwd(d, **bad) == -4


@pytest.mark.parametrize("d", [8, 32, 64, 96, 128])
@pytest.mark.parametrize("bad", [dict(o=BASE + 2), dict(do=BASE + 8), dict(ldo=2 * 128 + 4), dict(dqkv=BASE + 4),
                                 dict(ldg=6 * 128 + 2)])
def test_backward_entry_refuses_operands_that_are_not_in_whole_vectors(d, bad):
    assert _bwd(d, **bad) == -4


class _Recorder:
    """Stands in for the library: records the head width and the addresses of every call."""

    def __init__(self):
        self.calls = []

    def aeris_attn_fwd(self, q, ldq, _q0, k, ldk, _k0, v, ldv, _v0, o, ldo, lse, n_win, N, H, d, *_):
        self.calls.append((d, [q.value, o.value], [ldq, ldo]))
        return 0

    def aeris_attn_bwd(self, qkv, ldq, _q0, _k0, _v0, o, d_o, ldo, lse, delta, dqkv, ldg, n_win, N, H, d, *_):
        self.calls.append((d, [qkv.value, o.value, d_o.value, dqkv.value], [ldq, ldo, ldg]))
        return 0


@pytest.fixture
def recorder(monkeypatch):
    r = _Recorder()
    monkeypatch.setattr(L, "lib", lambda: r)
    monkeypatch.setattr(L, "status_word", lambda: None)
    monkeypatch.setattr(L, "stream_ptr", lambda: V(0))
    return r


def _rows(T, C, ld=None, off=0, step=1):
    """[T, C] bf16 with row pitch ``ld``, ``off`` elements past a 16-byte boundary, columns ``step`` elements apart."""
    ld = ld or C * step
    buf = torch.zeros(T * ld + off + 64, dtype=torch.bfloat16)
    off += (-buf.data_ptr() % 16) // 2
    return buf.as_strided((T, C), (ld, step), off)


@pytest.mark.parametrize("d", [16, 32, 96])
@pytest.mark.parametrize("qkv_kw,out_kw", [({}, {}), (dict(off=1), {}), ({}, dict(off=4)), (dict(pad=4), {}),
                                           ({}, dict(pad=2)), ({}, dict(step=2))])
def test_narrow_heads_reach_the_kernels_in_whole_vectors_or_as_padded_copies(recorder, d, qkv_kw, out_kw):
    """Every form that the padded copies took is still taken, and only whole vectors go straight to the kernels."""
    n_win, N, H = 2, 5, 2
    T = n_win * N

    def make(C, pad=0, **kw):
        return _rows(T, C, ld=C * kw.get("step", 1) + pad, **kw)

    plain = not qkv_kw and not out_kw
    A.attn_fwd(make(3 * H * d, **qkv_kw), n_win, N, H, d, out=make(H * d, **out_kw))
    o = make(H * d, **qkv_kw)
    A.attn_bwd(make(3 * H * d, **qkv_kw), o, o, torch.zeros(n_win, H, N), n_win, N, H, d, dqkv=make(3 * H * d, **out_kw))
    assert len(recorder.calls) == 2
    for width, ptrs, pitches in recorder.calls:
        assert width == (d if plain else (64 if d < 64 else 128))
        assert all(p % 16 == 0 for p in ptrs) and all(ld % 8 == 0 for ld in pitches)


@pytest.mark.parametrize("d", [8, 32, 96, 120])
def test_push_entries_take_the_kernels_own_head_widths_only(d):
    peers = (V * 2)(BASE, BASE)
    H, ld, hd = 2, 6 * d, 2 * d
    rc = L.lib().aeris_attn_fwd_push(V(BASE), ld, H, V(BASE), hd, V(BASE), 2, 16, d, ctypes.c_float(1.0), peers, 2, 8,
                                     2 * hd, 0, V(0), V(0))
    assert rc == -1
    rc = L.lib().aeris_attn_bwd_push(V(BASE), ld, H, V(BASE), V(BASE), hd, V(BASE), V(BASE), 2, 16, d, ctypes.c_float(1.0),
                                     peers, 2, 8, 6 * hd, 2 * hd, 0, V(0), V(0))
    assert rc == -1
