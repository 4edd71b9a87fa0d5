"""The native issue of a block's launches (``models/block.py``, ``csrc/block.cu``) against the same launches one by one."""
import re
from pathlib import Path

import pytest
import torch

from conftest import rel_err


def _struct(name):
    text = (Path(__file__).parent.parent / "aeris_gb_b200" / "csrc" / "api.h").read_text()
    body = re.search(r"typedef struct %s \{(.*?)\} %s;" % (name, name), text, re.S).group(1)
    fields = []
    for decl in re.sub(r"//[^\n]*", "", body).split(";"):
        m = re.match(r"\s*((?:const |long |unsigned )*\w+)\s+(.*)", decl.strip() + " ", re.S)
        base = re.match(r"\s*(const void\* const\*|const \w+|long long|unsigned|\w+)", decl)
        if not base:
            continue
        ptr = "*" in decl
        names = re.findall(r"\w+", decl[base.end():])
        kind = "p" if ptr else {"int": "i", "float": "f", "long long": "q"}[base.group(1).strip()]
        fields += [(n, kind) for n in names]
    return fields


@pytest.mark.parametrize("name", ["AerisBlock", "AerisBlockGrad"])
def test_argument_structs_mirror_the_header(name):
    import ctypes
    from aeris_gb_b200.models import block
    cls = {"AerisBlock": block.BlockArgs, "AerisBlockGrad": block.BlockGradArgs}[name]
    kinds = {ctypes.c_int: "i", ctypes.c_float: "f", ctypes.c_longlong: "q", ctypes.c_void_p: "p"}
    assert [(n, kinds[t]) for n, t in cls._fields_] == _struct(name)


def test_what_the_native_call_does_not_take_goes_one_by_one():
    """Exchanges of the parallel paths, other types, gaps, heads that are not whole vectors."""
    from aeris_gb_b200.models import block, fused
    from aeris_gb_b200.ops import elementwise as E

    class T:        # what takes() asks of a tensor
        def __init__(self, dtype=torch.bfloat16, cuda=True, whole=True):
            self.dtype, self.is_cuda, self.whole = dtype, cuda, whole

        def is_contiguous(self):
            return self.whole
    meta = lambda d=64, **k: fused.BlockMeta(2, 16, 2, d, E.MODE_MOD_THEN_NORM, 1e-6, 64, **k)
    mod, ok = T(torch.float32), [T()] * 6
    assert block.takes(meta(), T(), mod, ok, [mod]) and block.takes(meta(40), T(), mod, ok)
    for m, x, md, ws, gs in ((meta(sp=object()), T(), mod, ok, ()), (meta(tp=object()), T(), mod, ok, ()),
                             (meta(36), T(), mod, ok, ()), (meta(136), T(), mod, ok, ()),
                             (meta(), T(torch.float32), mod, ok, ()), (meta(), T(cuda=False), mod, ok, ()),
                             (meta(), T(whole=False), mod, ok, ()), (meta(), T(), T(), ok, ()),
                             (meta(), T(), mod, ok[:5] + [T(torch.float32)], ()),
                             (meta(), T(), mod, ok[:5] + [T(whole=False)], ()),
                             (meta(), T(), mod, ok, [T()]), (meta(), T(), mod, ok, [T(torch.float32, whole=False)])):
        assert not block.takes(m, x, md, ws, gs)


def _operands():
    """A block of two samples of two windows of 16 tokens, on the CPU: (meta, operands by name)."""
    from aeris_gb_b200.models import fused
    from aeris_gb_b200.ops import elementwise as E
    meta, T, D, HD, F = fused.BlockMeta(2, 16, 2, 64, E.MODE_MOD_THEN_NORM, 1e-6, 64), 64, 32, 128, 48
    z = lambda *s, dt=torch.bfloat16: torch.zeros(s, dtype=dt)
    f = lambda *s: z(*s, dt=torch.float32)
    shapes = {"n1": (D,), "to_qkv": (3 * HD, D), "wo": (D, HD), "n2": (D,), "w1": (2 * F, D), "w2": (D, F)}
    ops = {"x": z(T, D), "mod": f(2, 6 * D), "dy": z(T, D), "dx": z(T, D), "out": z(T, D), "table": torch.arange(T).int()}
    return meta, {**ops, **{k: z(*s) for k, s in shapes.items()}, **{"g_" + k: f(*s) for k, s in shapes.items()}}


MISFITS = {                         # operand -> one of another extent; which directions take it
    "n1": ((16,), "fb"), "n2": ((16,), "fb"), "to_qkv": ((320, 32), "fb"), "wo": ((32, 64), "fb"), "w1": ((64, 32), "fb"),
    "w2": ((16, 48), "fb"), "mod": ((2, 160), "fb"), "x": ((32, 32), "fb"), "out": ((32, 32), "f"), "table": ((32,), "f"),
    "dy": ((32, 32), "b"), "dx": ((32, 32), "b"), "g_n1": ((16,), "b"), "g_n2": ((16,), "b"), "g_wo": ((32, 64), "b"),
    "g_to_qkv": ((320, 32), "b"), "g_w1": ((64, 32), "b"), "g_w2": ((16, 48), "b")}


@pytest.mark.parametrize("name,way", [(n, w) for n, (_, ways) in MISFITS.items() for w in ways] + [(None, "f"), (None, "b")])
def test_operands_of_other_extents_are_refused(name, way, monkeypatch):
    """The native call derives every extent; what does not fit goes launch by launch and is refused there. The library is a
    stand-in that accepts every launch."""
    from aeris_gb_b200.models import block, fused
    from aeris_gb_b200.ops import lib

    class Library:
        def __getattr__(self, entry):
            return lambda *a: 0

    meta, ops = _operands()
    if name is not None:
        ops[name] = torch.zeros(MISFITS[name][0], dtype=ops[name].dtype)
    native = []
    monkeypatch.setattr(lib, "lib", Library)
    monkeypatch.setattr(lib, "raw_stream", lambda: 0)
    monkeypatch.setattr(lib, "status_word", lambda: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(fused, "_WS", fused.Workspace())
    monkeypatch.setattr(block, "takes", lambda *a: True)          # all but the extents is right
    monkeypatch.setattr(block, "forward", lambda *a: native.append("f"))
    monkeypatch.setattr(block, "backward", lambda *a: native.append("b"))
    ws = [ops[k] for k in block.WEIGHTS]

    def run():
        if way == "f":
            fused.block_forward(ops["x"], ops["mod"], meta, *ws, out=ops["out"], gather=(ops["table"], [0], ops["x"]))
        else:
            grads = {k: ops["g_" + k] for k in block.WEIGHTS}
            fused.block_backward(ops["x"], ops["mod"], ops["dy"], meta, *ws, grads, dx=ops["dx"])
    if name is None:
        run()
        assert native == [way]
    else:
        with pytest.raises((AssertionError, RuntimeError, ValueError)):
            run()
        assert not native


@pytest.mark.parametrize("step", [0, -1])
def test_chunks_of_no_windows_are_refused(step):
    """Before anything is launched: by the entry points, whose loop over chunks would not end, and by both directions."""
    import ctypes
    from aeris_gb_b200.models import block, fused
    from aeris_gb_b200.ops import lib
    a, g = block.BlockArgs(step=step, batch=1, n_win=2, L=16, D=32, F=48, heads=2, head_dim=64), block.BlockGradArgs()
    assert lib.lib().aeris_block_forward(ctypes.byref(a)) == -1
    assert lib.lib().aeris_block_backward(ctypes.byref(a), ctypes.byref(g)) == -1
    meta, ops = _operands()
    meta = fused.BlockMeta(2, 16, 2, 64, meta.mode, 1e-6, step, min_chunk_bytes=0)
    ws = [ops[k] for k in block.WEIGHTS]
    with pytest.raises(ValueError):
        fused.block_forward(ops["x"], ops["mod"], meta, *ws)
    with pytest.raises(ValueError):
        fused.block_backward(ops["x"], ops["mod"], ops["dy"], meta, *ws, {k: ops["g_" + k] for k in block.WEIGHTS})


@pytest.mark.gpu
@pytest.mark.parametrize("B,n_win,L,heads,d,F,chunk,floor,mode,rope", [
    (1, 3, 225, 4, 64, 512, 2, 0, 0, False),        # two chunks, the second one short
    (2, 3, 225, 4, 64, 512, 64, None, 1, False),    # both samples in one forward launch
    (2, 2, 64, 2, 128, 256, 1, 0, 0, True),         # rotary embedding, one window per chunk
    (3, 2, 30, 16, 40, 384, 64, None, 1, False)])    # narrow heads, widths for the one-CTA kernel
@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("gathered", [False, True])
def test_block_in_one_call_equals_its_launches(B, n_win, L, heads, d, F, chunk, floor, mode, rope, keep, gathered,
                                               monkeypatch):
    from aeris_gb_b200.models import block, fused
    from aeris_gb_b200.ops import lib
    torch.manual_seed(B * L)
    D = 256 if d != 40 else 128
    HD, T = heads * d, B * n_win * L
    r = None
    if rope:
        ang = torch.rand(L, d // 2, device="cuda")
        r = (ang.cos(), ang.sin())
    meta = fused.BlockMeta(n_win, L, heads, d, mode, 1e-3, chunk, rope=r, min_chunk_bytes=floor)
    g = lambda *s, k=1.0: torch.randn(*s, device="cuda") * k
    x, mod = g(T, D).bfloat16(), g(B, 6 * D)
    ws = [w.bfloat16() for w in (g(D), g(3 * HD, D, k=0.05), g(D, HD, k=0.05), g(D), g(2 * F, D, k=0.05), g(D, F, k=0.05))]
    dy = g(T, D).bfloat16()
    gather = None
    if gathered:
        gather = (torch.randperm(T, device="cuda").int(), [x.data_ptr()], x)
    out = []
    takes = block.takes
    for native in (True, False):
        monkeypatch.setattr(block, "takes", takes if native else (lambda *a: False))
        kept = {k: torch.empty(s, dtype=t, device="cuda") for k, (s, t) in
                fused._kept_shapes(T, D, HD, heads, F).items()} if keep else None
        xin = torch.empty_like(x) if gathered else x
        n0 = lib.launch_count()
        y = fused.block_forward(xin, mod, meta, *ws, gather=gather, kept=kept)
        n1 = lib.launch_count()
        grads = {k: torch.zeros(w.shape, device="cuda") for k, w in zip(("n1", "to_qkv", "wo", "n2", "w1", "w2"), ws)}
        dx, dmod = fused.block_backward(xin, mod, dy, meta, *ws, grads, kept=kept)
        out.append((y, dx, dmod, grads, (n1 - n0, lib.launch_count() - n1)))
    lib.check_status()
    (y0, dx0, dm0, g0, n0), (y1, dx1, dm1, g1, n1) = out
    assert torch.equal(y0, y1) and torch.equal(dx0, dx1)
    # the two gated matrices share a launch before and after each sample's products
    assert n0[0] == n1[0] and n0[1] == n1[1] - 2 * B
    # the column sums and split reductions are fp32 atomics in another order each time
    assert rel_err(dm0, dm1) < 1e-5
    for k in g0:
        assert rel_err(g0[k], g1[k]) < 1e-5, k
