"""Kernels that may start while the one before them still runs: blocks issued back to back, each reading what the one before
wrote and overwriting what the one before that read, against the same launches with a wait after each. Small windows (every
kernel leaves the GPU part empty, so the next one starts early), several chunks, and rows moved from block to block."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
N_BLOCKS = 12


def _case(L, heads, d, D, F, rope):
    from aeris_gb_b200.models import fused
    torch.manual_seed(L)
    n_win, HD = 3, heads * d
    r = None
    if rope:
        ang = torch.rand(L, d // 2, device="cuda")
        r = (ang.cos(), ang.sin())
    meta = fused.BlockMeta(n_win, L, heads, d, 1, 1e-3, 2, rope=r, min_chunk_bytes=0)
    g = lambda *s, k=1.0: torch.randn(*s, device="cuda") * k
    ws = [w.bfloat16() for w in (g(D), g(3 * HD, D, k=0.05), g(D, HD, k=0.05), g(D), g(2 * F, D, k=0.05), g(D, F, k=0.05))]
    return meta, g(n_win * L, D).bfloat16(), g(1, 6 * D), ws, torch.randperm(n_win * L, device="cuda").int()


def _forward(meta, x, mod, ws, table, bufs):
    """Blocks over three buffers that take turns; every second one gathers its rows."""
    from aeris_gb_b200.models import fused
    bufs[0].copy_(x)
    cur = 0
    for i in range(N_BLOCKS):
        src, gather = cur, None
        if i % 2:
            cur = (src + 1) % 3
            gather = (table, [bufs[src].data_ptr()], bufs[src])
        y = next(k for k in range(3) if k not in (src, cur))
        fused.block_forward(bufs[cur], mod, meta, *ws, out=bufs[y], gather=gather)
        cur = y
    return bufs[cur]


def _wait_after_each_launch(monkeypatch):
    from aeris_gb_b200.models import block
    from aeris_gb_b200.ops import lib
    check = lib.check
    monkeypatch.setattr(block, "takes", lambda *a: False)
    monkeypatch.setattr(lib, "check", lambda *a, **k: (check(*a, **k), torch.cuda.synchronize())[0])


@pytest.mark.parametrize("L,heads,d,D,F,rope", [(64, 2, 64, 128, 256, False), (225, 4, 64, 256, 512, True),
                                                (400, 2, 128, 256, 384, False), (30, 16, 40, 128, 128, False)])
def test_chained_launches_equal_waited_for_ones(L, heads, d, D, F, rope, monkeypatch):
    from aeris_gb_b200.models import fused
    from aeris_gb_b200.ops import lib
    meta, x, mod, ws, table = _case(L, heads, d, D, F, rope)
    bufs = [torch.empty_like(x) for _ in range(3)]

    def passes():
        y = _forward(meta, x, mod, ws, table, bufs).clone()
        grads = {k: torch.zeros(w.shape, device="cuda") for k, w in zip(("n1", "to_qkv", "wo", "n2", "w1", "w2"), ws)}
        g = [y, torch.empty_like(y)]
        for i in range(N_BLOCKS):       # the gradient of one block is the next one's
            fused.block_backward(x, mod, g[i % 2], meta, *ws, grads, dx=g[1 - i % 2])
        return _forward(meta, x, mod, ws, table, bufs).clone(), g[N_BLOCKS % 2], grads

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    runs = [passes() for _ in range(3)]
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        runs.append(passes())
    torch.cuda.synchronize()
    _wait_after_each_launch(monkeypatch)
    y, dx, grads = passes()
    lib.check_status()
    for y0, dx0, g0 in runs:
        assert torch.equal(y0, y) and torch.equal(dx0, dx)
        for k in grads:
            assert rel_err(g0[k], grads[k]) < 1e-5, k      # fp32 atomics in another order each time


def test_chained_launches_in_a_graph():
    from aeris_gb_b200.ops import lib
    meta, x, mod, ws, table = _case(225, 4, 64, 256, 512, False)
    bufs = [torch.empty_like(x) for _ in range(3)]
    want = _forward(meta, x, mod, ws, table, bufs).clone()       # and the workspaces are there
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _forward(meta, x, mod, ws, table, bufs)
    for b in bufs:
        b.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    lib.check_status()
    assert torch.equal(out, want)
