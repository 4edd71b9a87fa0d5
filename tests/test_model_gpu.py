"""The CUDA block path (hand-written forward and backward) against the PyTorch oracle on a small model."""
import os

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _small_cfg(after_mod_norm=True, head_dim=64, window=(16, 16)):
    from aeris_gb_b200.models.aeris import AerisConfig
    return AerisConfig(img=(32, 64), window=window, in_channels=20, out_channels=8, dim=128, heads=2,
                       head_dim=head_dim, mlp_dim=256, n_layers=2, sublayers=2, after_mod_norm=after_mod_norm,
                       norm_eps=1e-3, chunk_windows=3)


def _recompute_in_chunks(cfg, recompute):
    """Every block recomputes in chunks of three of its eight windows (two full ones and a remainder), or keeps its
    internals."""
    if recompute:
        cfg.recompute, cfg.min_chunk_bytes = True, 0
    return cfg


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("after_mod_norm", [True, False])
def test_fused_model_matches_oracle(after_mod_norm, recompute):
    from aeris_gb_b200.models.aeris import AerisModel
    torch.manual_seed(1)
    cfg = _recompute_in_chunks(_small_cfg(after_mod_norm), recompute)
    model = AerisModel(cfg).cuda()
    for n, p in model.named_parameters():
        if "modulation" in n and p.dim() == 2:
            torch.nn.init.normal_(p, std=0.05)
    x = torch.randn(2, 32, 64, cfg.in_channels, device="cuda")
    t = torch.tensor([0.3, 1.2], device="cuda")
    params = [p for p in model.parameters() if p.requires_grad]

    def run(force_oracle):
        os.environ["AERIS_FORCE_ORACLE"] = "1" if force_oracle else "0"
        for p in params:
            p.grad = None
        xin = x.clone().requires_grad_(True)
        y = model(xin, t)
        (y * torch.linspace(-1, 1, y.numel(), device="cuda").view_as(y)).sum().backward()
        return y.detach(), xin.grad, [p.grad.clone() if p.grad is not None else None for p in params]

    try:
        y0, gx0, g0 = run(True)
        y1, gx1, g1 = run(False)
    finally:
        os.environ.pop("AERIS_FORCE_ORACLE", None)
    assert rel_err(y1, y0) < 3e-2
    assert rel_err(gx1, gx0) < 5e-2
    names = [n for n, p in model.named_parameters() if p.requires_grad]
    for n, a, b in zip(names, g1, g0):
        if b is None or b.float().norm() == 0:
            continue
        assert a is not None, n
        assert rel_err(a, b) < 8e-2, (n, rel_err(a, b))


@pytest.mark.parametrize("recompute", [False, True])
def test_fused_model_with_rope_matches_oracle(recompute):
    """Optional 2-D rotary embedding: the CUDA path (rotation applied to the qkv chunks, inverse rotation of their
    gradients) against the PyTorch formulation."""
    from aeris_gb_b200.models.aeris import AerisModel
    torch.manual_seed(2)
    cfg = _recompute_in_chunks(_small_cfg(), recompute)
    cfg.use_rope = True
    model = AerisModel(cfg).cuda()
    for n, p in model.named_parameters():
        if "modulation" in n and p.dim() == 2:
            torch.nn.init.normal_(p, std=0.05)
    x = torch.randn(2, 32, 64, cfg.in_channels, device="cuda")
    t = torch.tensor([0.3, 1.2], device="cuda")
    params = [p for p in model.parameters() if p.requires_grad]

    def run(force_oracle):
        os.environ["AERIS_FORCE_ORACLE"] = "1" if force_oracle else "0"
        for p in params:
            p.grad = None
        y = model(x, t)
        (y * torch.linspace(-1, 1, y.numel(), device="cuda").view_as(y)).sum().backward()
        return y.detach(), [p.grad.clone() if p.grad is not None else None for p in params]

    try:
        y0, g0 = run(True)
        y1, g1 = run(False)
        cfg.use_rope = False
        y2, _ = run(True)
    finally:
        os.environ.pop("AERIS_FORCE_ORACLE", None)
    assert rel_err(y1, y0) < 3e-2
    assert rel_err(y2, y0) > 1e-3          # the embedding does change the result
    for a, b in zip(g1, g0):
        if b is None or b.float().norm() == 0:
            continue
        assert rel_err(a, b) < 8e-2


@pytest.mark.parametrize("recompute", [False, True])
def test_wide_block_dim5120_matches_oracle(recompute):
    """The block dimensions of the 13 B-class configuration (dim 5120, 40 heads x 128, 30 x 30 windows) on a small
    image: forward and input gradient of the CUDA path against the PyTorch formulation."""
    from aeris_gb_b200.models.aeris import AerisConfig, AerisModel
    torch.manual_seed(4)
    cfg = AerisConfig(img=(60, 120), window=(30, 30), in_channels=20, out_channels=8, dim=5120, heads=40, head_dim=128,
                      mlp_dim=13824, n_layers=2, sublayers=1, norm_eps=1e-3, chunk_windows=3)
    _recompute_in_chunks(cfg, recompute)
    model = AerisModel(cfg).cuda()
    for n, p in model.named_parameters():
        if "modulation" in n and p.dim() == 2:
            torch.nn.init.normal_(p, std=0.02)
    x = torch.randn(1, 60, 120, cfg.in_channels, device="cuda")
    t = torch.tensor([0.7], device="cuda")

    def run(force_oracle):
        os.environ["AERIS_FORCE_ORACLE"] = "1" if force_oracle else "0"
        model.zero_grad(set_to_none=True)
        xin = x.clone().requires_grad_(True)
        y = model(xin, t)
        (y * torch.linspace(-1, 1, y.numel(), device="cuda").view_as(y)).sum().backward()
        return y.detach(), xin.grad, model.layers[0].modulelist[0][3].w2.weight.grad.clone()

    try:
        y0, gx0, gw0 = run(True)
        y1, gx1, gw1 = run(False)
    finally:
        os.environ.pop("AERIS_FORCE_ORACLE", None)
    assert rel_err(y1, y0) < 3e-2
    assert rel_err(gx1, gx0) < 6e-2
    assert rel_err(gw1, gw0) < 8e-2


def test_train_step_raises_on_a_device_timeout_instead_of_stepping():
    """A bounded device wait that runs out (here: a wait on a flag that nothing sets, queued ahead of the step) must
    surface as KernelError from train_step before the optimizer touches the weights; the trainer stays usable."""
    import ctypes
    from aeris_gb_b200.engine.optim import OptimConfig
    from aeris_gb_b200.engine.trainer import DiffusionConfig, Trainer
    from aeris_gb_b200.ops import lib as L
    cfg = _small_cfg()
    tr = Trainer(cfg, OptimConfig(), DiffusionConfig(cond_channels=cfg.in_channels - cfg.out_channels), "cuda:0")
    x = torch.randn(1, 32, 64, cfg.out_channels).pin_memory()
    c = torch.randn(1, 32, 64, cfg.in_channels - cfg.out_channels).pin_memory()
    tr.train_step(x, c)
    before = [p.detach().clone() for p in tr.model.parameters()]
    steps = tr.opt.step_count
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = L.lib().aeris_wait_flag(L.ptr(flag), ctypes.c_uint(1), L.ptr(L.status_word()), ctypes.c_double(0.3),
                                 L.stream_ptr())
    assert rc == 0
    with pytest.raises(L.KernelError, match="peer signal"):
        tr.train_step(x, c)
    assert tr.opt.step_count == steps
    assert all(torch.equal(a, b.detach()) for a, b in zip(before, tr.model.parameters()))
    assert all(float(g.abs().max()) == 0.0 for g in tr.opt.grad_buffers())
    loss = tr.train_step(x, c)              # status cleared, gradients dropped: the next step runs normally
    assert loss == loss and tr.opt.step_count == steps + 1


@pytest.mark.parametrize("mod_first", [True, False])
def test_kept_internals_give_the_gradients_of_the_recompute(mod_first, monkeypatch):
    """A block that keeps its internals and one that recomputes them launch the same kernels on the same values: equal
    outputs, and gradients equal up to the order of the fp32 atomic sums. What is kept must survive a backward pass (the
    gated product is written beside it, not over it): a second one over the retained graph gives the same."""
    from aeris_gb_b200.models import fused
    from aeris_gb_b200.models.aeris import AerisConfig, AerisModel
    cfg = AerisConfig(img=(30, 60), window=(15, 15), in_channels=20, out_channels=8, dim=256, heads=4, head_dim=64,
                      mlp_dim=512, n_layers=2, sublayers=2, after_mod_norm=mod_first, chunk_windows=3)
    monkeypatch.setattr(fused, "MIN_CHUNK_BYTES", 1)          # three-window chunks: 8 windows leave a remainder
    torch.manual_seed(3)
    model = AerisModel(cfg).cuda()
    for p in model.parameters():
        torch.nn.init.normal_(p, std=0.05)
    x = torch.randn(2, 30, 60, 20, device="cuda")
    t = torch.tensor([0.4, 1.1], device="cuda")
    n_blocks, runs = 4, {}
    for keep in (0, 3, n_blocks):
        monkeypatch.setattr(fused, "plan_kept_blocks", lambda *a, keep=keep: keep)
        model.zero_grad(set_to_none=True)
        y = model(x, t)
        loss = (y * torch.linspace(-1, 1, y.numel(), device="cuda").view_as(y)).sum()
        loss.backward(retain_graph=True)
        first = {n: p.grad.float().clone() for n, p in model.named_parameters() if p.grad is not None}
        model.zero_grad(set_to_none=True)
        loss.backward()
        second = {n: p.grad.float().clone() for n, p in model.named_parameters() if p.grad is not None}
        runs[keep] = (y.detach(), first, second)
    for keep in (3, n_blocks):
        assert torch.equal(runs[keep][0], runs[0][0])
        for got in runs[keep][1:]:
            for n, g in runs[0][1].items():
                # bf16 gradients of bf16 weights: an atomic sum in another order may round to the neighbouring value
                assert rel_err(got[n], g) < 2.0 ** -9, n


@pytest.mark.parametrize("dim,heads", [(256, 4), (5376, 42)])
def test_samples_in_one_launch_equal_samples_one_by_one(dim, heads):
    """A batch whose samples are one chunk each runs every forward kernel once, with the modulation vectors picked by row:
    the same values as each sample alone, bit for bit (windows of 225 tokens: tiles straddle the sample boundary). 5376
    columns: no batched modulate + norm launch, one per sample."""
    from aeris_gb_b200.models import fused
    from aeris_gb_b200.ops import elementwise as E
    torch.manual_seed(1)
    L, n_win, B, F = 225, 3, 3, 512
    if dim > 5120:
        x = torch.randn(4, dim, device="cuda").bfloat16()
        w, sc = torch.ones(dim, device="cuda").bfloat16(), torch.randn(2, dim, device="cuda")
        one = [E.modnorm_fwd(x[2 * b:2 * b + 2], sc[b], sc[b], w, mode=0, eps=1e-3) for b in range(2)]
        assert torch.equal(E.modnorm_fwd(x, sc, sc, w, mode=0, eps=1e-3, batch=2), torch.cat(one))
        return
    meta = fused.BlockMeta(n_win, L, heads, dim // heads, E.MODE_MOD_THEN_NORM, 1e-3, 64)
    T = B * n_win * L
    x = torch.randn(T, dim, device="cuda").bfloat16()
    mod = torch.randn(B, 6 * dim, device="cuda")
    ws = [torch.ones(dim), torch.randn(3 * dim, dim) * 0.05, torch.randn(dim, dim) * 0.05, torch.ones(dim),
          torch.randn(2 * F, dim) * 0.05, torch.randn(dim, F) * 0.05]
    ws = [w.cuda().bfloat16() for w in ws]
    assert len(fused._forward_spans(meta, B, n_win, dim, F, False)) == 1
    y = fused.block_forward(x, mod, meta, *ws)
    n = n_win * L
    for b in range(B):
        assert torch.equal(y[b * n:(b + 1) * n], fused.block_forward(x[b * n:(b + 1) * n], mod[b:b + 1], meta, *ws))


@pytest.mark.parametrize("L,n_win,chunk,dims", [(64, 32, 8, (512, 128)), (64, 32, 8, (128, 256)), (900, 8, 4, (1024, 256)),
                                                (64, 288, 4, (256, 256))])
def test_weight_gradients_of_merged_chunks_are_as_accurate_as_those_of_the_chunks(L, n_win, chunk, dims):
    """Small weights, where finer slices cost nothing: one product over all windows, with the slices that
    ``block_backward`` asks for, against one per ``chunk_windows`` with four slices each. The error against 64 bits is the
    tensor core's truncation, proportional to the rows of a slice, and may not grow beyond the rounding of the fp32
    additions between slices (2^-24 each)."""
    from aeris_gb_b200.ops import gemm as G
    torch.manual_seed(L)
    a, b = (torch.randn(n_win * L, k, device="cuda").bfloat16() for k in dims)
    ref = a.double().t() @ b.double()
    err = []
    for step in (chunk, n_win):
        out = torch.zeros(dims, device="cuda")
        for w in range(0, n_win, step):
            n = min(step, n_win - w)
            sl = slice(w * L, (w + n) * L)
            G.gemm(a[sl], b[sl], a_t=True, b_t=True, out=out, epi=G.EPI_ACC_F32,
                   k_splits=4 if step == chunk else -4 * -(-n // chunk))
        err.append(((out.double() - ref).norm() / ref.norm()).item())
    assert err[1] < err[0] + 2.0 ** -24, err
