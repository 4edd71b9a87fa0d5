"""Modulation vectors that do not start on a 16-byte boundary: the kernels of both directions read vectors of four."""
import pytest
import torch

from aeris_gb_b200.models import block as NB
from aeris_gb_b200.models import fused
from aeris_gb_b200.ops import elementwise as E

DEV = "cuda"


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("way", ["forward", "backward"])
def test_vectors_off_the_grid_are_moved_before_a_kernel_reads_them(way, native, monkeypatch):
    """Both directions, in one native call and launch by launch: the addresses handed on to a library that runs nothing."""
    from aeris_gb_b200.ops import lib
    seen = []

    class Library:
        def __getattr__(self, entry):
            def call(*a):
                if entry.startswith("aeris_block"):
                    seen.append(a[0]._obj.mod)
                elif entry.startswith("aeris_modnorm"):          # scale, shift
                    seen.extend(p.value for p in (a[5:7] if "fwd" in entry else a[3:5]))
                elif entry == "aeris_gemm_auto" and a[14].value:
                    seen.append(a[14].value)                     # gate
                return 0
            return call

    monkeypatch.setattr(lib, "lib", Library)
    monkeypatch.setattr(lib, "raw_stream", lambda: 0)
    monkeypatch.setattr(lib, "status_word", lambda: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(fused, "_WS", fused.Workspace())
    monkeypatch.setattr(NB, "takes", lambda *a: native)
    D, F, T = 32, 48, 64
    meta = fused.BlockMeta(2, 16, 2, 64, E.MODE_MOD_THEN_NORM, 1e-6)
    z = lambda *s: torch.zeros(s, dtype=torch.bfloat16)
    ws = dict(n1=z(D), to_qkv=z(384, D), wo=z(D, 128), n2=z(D), w1=z(2 * F, D), w2=z(D, F))
    base = torch.zeros(2 * 6 * D + 4)
    mod = base[(16 - base.data_ptr() % 16) // 4 % 4 + 1:][:2 * 6 * D].view(2, 6 * D)
    assert mod.data_ptr() % 16 == 4 and mod.is_contiguous()
    if way == "forward":
        fused.block_forward(z(T, D), mod, meta, *ws.values())
    else:
        fused.block_backward(z(T, D), mod, z(T, D), meta, *ws.values(), {k: torch.zeros(w.shape) for k, w in ws.items()})
    assert seen and all(p and p % 16 == 0 for p in seen)


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
def test_backward_off_the_grid_equals_an_aligned_copy(native, monkeypatch):
    D, heads, F, L, wins, B = 128, 2, 128, 70, 2, 2
    meta = fused.BlockMeta(wins, L, heads, 64, E.MODE_MOD_THEN_NORM, 1e-6)
    rnd = lambda *s: (torch.randn(*s, device=DEV) * s[-1] ** -0.5).bfloat16()
    ws = dict(n1=1 + rnd(D), to_qkv=rnd(3 * heads * 64, D), wo=rnd(D, heads * 64), n2=1 + rnd(D), w1=rnd(2 * F, D),
              w2=rnd(D, F))
    x, dy = torch.randn(2, B * wins * L, D, device=DEV).bfloat16()
    mod = torch.randn(B * 6 * D + 1, device=DEV)[1:].view(B, 6 * D)
    if not native:
        monkeypatch.setattr(NB, "takes", lambda *a: False)
    out = []
    for m in (mod, mod.clone()):
        grads = {k: torch.zeros(w.shape, device=DEV) for k, w in ws.items()}
        out.append((*fused.block_backward(x, m, dy, meta, *ws.values(), grads), *grads.values()))
    assert torch.equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1:], out[1][1:]):         # fp32 sums by atomics, in another order each time
        assert float((a - b).norm() / b.norm()) < 1e-5
