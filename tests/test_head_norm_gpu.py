"""The output stage of the objectives without a fused loss on the fp32 modulate + norm kernels, against float64."""
import pytest
import torch

from aeris_gb_b200.models import aeris as A

pytestmark = pytest.mark.gpu
U = 2.0 ** -24                       # rounding unit of fp32


def _problem(B, rows, D, out, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    cfg = A.AerisConfig(dim=64, heads=2, head_dim=32, out_channels=4)
    stage = A.OutputStage(cfg).cuda()
    stage.head = torch.nn.Linear(D, out, bias=False).cuda()
    stage.norm = torch.nn.RMSNorm(D).cuda()
    with torch.no_grad():
        stage.norm.weight.copy_(1 + 0.2 * rnd(D))
    x = (rnd(B * rows, D) * 2).bfloat16()
    mod = 0.3 * rnd(B, 2 * D)
    return stage, x, mod, rnd(B * rows, out)


def _run(stage, x, mod, dout):
    x = x.clone().requires_grad_(True)
    mod = mod.clone().requires_grad_(True)
    shift, scale = mod.chunk(2, dim=1)
    y = A._HeadFn.apply(x, shift, scale, stage.norm.weight, stage.head.weight, stage)
    grads = torch.autograd.grad(y, [x, mod, stage.norm.weight, stage.head.weight], dout)
    return [y.detach(), *grads]


def _exact(stage, x, mod, dout, B):
    """Results in float64 and, for each, the sum of the magnitudes of the terms that it adds up."""
    x64 = x.double()
    rows, D = x.shape[0] // B, x.shape[1]
    shift, scale = (t.repeat_interleave(rows, 0) for t in mod.double().chunk(2, dim=1))
    w, W, do = stage.norm.weight.detach().double(), stage.head.weight.detach().double(), dout.double()
    r = (x64.pow(2).mean(1, keepdim=True) + stage.cfg.eps(torch.float32)).rsqrt()
    n = x64 * r
    y = n * w * (1 + scale) + shift
    ya = (n * w * (1 + scale)).abs() + shift.abs()
    dy, dya = do @ W, do.abs() @ W.abs()
    gn, gna = dy * w * (1 + scale), dya * (w * (1 + scale)).abs()
    dx = r * (gn - n * (gn * n).mean(1, keepdim=True))
    dxa = r * (gna + n.abs() * (gna * n.abs()).mean(1, keepdim=True))
    per = lambda t: t.view(B, rows, D).sum(1)
    res = [y @ W.t(), dx, torch.cat([per(dy), per(dy * n * w)], 1), (dy * (1 + scale) * n).sum(0), do.t() @ y]
    mag = [ya @ W.abs().t(), dxa, torch.cat([per(dya), per(dya * (n * w).abs())], 1),
           (dya * ((1 + scale) * n).abs()).sum(0), do.abs().t() @ ya]
    return res, mag


@pytest.mark.parametrize("B,rows,D,out,step", [
    (1, 1, 8, 1, 64), (2, 37, 384, 16, 1 << 16), (3, 65, 512, 70, 64), (1, 130, 1536, 70, 128), (2, 41, 1544, 7, 1 << 16),
    (1, 33, 2560, 5, 16), (2, 19, 5120, 70, 1 << 16), (1, 1200, 264, 70, 1 << 16)])
def test_head_norm_kernels(B, rows, D, out, step, monkeypatch):
    monkeypatch.setattr(A._HeadFn, "STEP", step)
    stage, x, mod, dout = _problem(B, rows, D, out)
    got = _run(stage, x, mod, dout)
    want, mag = _exact(stage, x, mod, dout, B)
    # Each result is a sum (or a sum of sums) of n products of a few rounded factors: its error is at most (n + 32) units
    # of the terms' magnitudes, in any order of summation. Two nested sums over a row enter dx, and the sum over the
    # output channels every gradient; dx is rounded to bf16 at the end.
    n_terms = [2 * D, 2 * D + out, rows + D + out, B * rows + D + out, B * rows + D]
    for i, (g, w_, m, n) in enumerate(zip(got, want, mag, n_terms)):
        tol = (n + 32) * U * m + (2.0 ** -8 * w_.abs() if i == 1 else 0)
        assert ((g.double() - w_).abs() <= tol + 1e-30).all(), i


@pytest.mark.parametrize("change", ["odd width", "offset stream", "strided stream", "wide rows", "no rows"])
def test_head_norm_other_forms(change, monkeypatch):
    """Forms outside the kernels' rule take the PyTorch route, whose result they equal."""
    D = {"odd width": 36, "wide rows": 5128}.get(change, 64)
    stage, x, mod, dout = _problem(2, 24, D, 6)
    if change == "offset stream":
        x = torch.cat([x.flatten()[:4], x.flatten()])[4:].view_as(x)
    elif change == "strided stream":
        x = torch.cat([x, x], 1)[:, :D]
    elif change == "no rows":
        x, dout = x[:0], dout[:0]
    shift, scale = mod.chunk(2, dim=1)
    assert not A._HeadFn._kernels(x, shift, scale, stage.norm.weight, stage.head.weight)
    y = A._HeadFn.apply(x, shift, scale, stage.norm.weight, stage.head.weight, stage)
    ref = torch.cat([stage.forward_rows(xb, shift[b:b + 1], scale[b:b + 1]) for b, xb in enumerate(x.chunk(2))]) \
        if x.numel() else y
    assert torch.equal(y, ref)


def test_head_norm_saved_hooks_and_graph():
    """Saved tensors that come back with other strides, and a backward pass that is itself recorded."""
    stage, x, mod, dout = _problem(2, 40, 128, 6)
    want = _run(stage, x, mod, dout)

    def other_strides(t):
        return t.t().contiguous().t() if t.dim() == 2 and t.shape[0] != 6 else t      # not the head: another product

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, other_strides):
        got = _run(stage, x, mod, dout)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    xr = x.clone().requires_grad_(True)
    shift, scale = mod.chunk(2, dim=1)
    y = A._HeadFn.apply(xr, shift, scale, stage.norm.weight, stage.head.weight, stage)
    assert torch.equal(torch.autograd.grad(y, xr, dout, create_graph=True)[0], want[1])
