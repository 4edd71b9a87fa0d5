"""Kernels around the conditioning vector and the packed weights of the two ends, against plain PyTorch."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,K", [(1, 4), (70, 100), (257, 256), (1536, 1536), (130, 2052), (64, 1001), (20000, 1536)])
@pytest.mark.parametrize("B", [1, 2, 3, 8])
@pytest.mark.parametrize("silu_in", [False, True])
def test_gemv_forward_and_gradients(N, K, B, silu_in):
    """Row counts around the kernel's templates, widths that are no multiple of a vector (K = 1001: scalar loads, and no
    backward kernel) or of a CTA's columns, bf16 and fp32 operands; fp32 sums of K (or N) terms, fast exp in the SiLU."""
    _gemv_case(N, K, B, silu_in)


@pytest.mark.parametrize("B,K", [(1, 8192), (3, 3076), (3, 4096), (3, 5120), (5, 2456), (8, 1540), (8, 5120), (8, 6400)])
def test_gemv_rows_beyond_the_default_shared_memory(B, K):
    """Rows of x that need more than 48 KB, up to the kernel's limit of 200 KB."""
    _gemv_case(300, K, B, True)


def _gemv_case(N, K, B, silu_in):
    from aeris_gb_b200.ops import diffusion as DF
    torch.manual_seed(N + K + B)
    for wt, xt in ((torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.bfloat16, torch.float32)):
        W, b = torch.randn(N, K, device=DEV).to(wt), torch.randn(N, device=DEV).to(wt)
        x = torch.randn(B, K, device=DEV).to(xt)
        dy = torch.randn(B, N, device=DEV)
        Wd, bd, xd = (v.double().requires_grad_(True) for v in (W, b, x))
        ref = (torch.nn.functional.silu(xd) if silu_in else xd) @ Wd.t() + bd
        ref.backward(dy.double())
        assert rel_err(DF.gemv_bias_act(W, b, x, silu_in=silu_in), ref) < 4e-6
        dW, db, dx = torch.ones(N, K, device=DEV), torch.ones(N, device=DEV), torch.zeros(B, K, device=DEV)
        if not DF.gemv_bwd_ok(W, dW):
            assert K % 4
            continue
        DF.gemv_bwd(W, x, dy, dW, db, dx, silu_in)
        assert rel_err(dW, Wd.grad + 1) < 4e-6 and rel_err(db, bd.grad + 1) < 4e-6 and rel_err(dx, xd.grad) < 4e-6
        dW2 = torch.ones(N, K, device=DEV)
        DF.gemv_bwd(W, x, dy, dW2, None, None, silu_in)        # without the bias and without the gradient of x
        assert torch.equal(dW, dW2)


def test_modulation_of_three_samples_at_dim_5120():
    """The widest model with several samples per step: both layers on the kernel, against the stock operators."""
    from aeris_gb_b200.models.aeris import ModulationLinear
    from aeris_gb_b200.models.fused import modulation
    from aeris_gb_b200.ops import diffusion as DF
    assert DF.gemv_ok(3, 5120)
    seq = ModulationLinear(5120, 640, True).cuda().modulation
    for p in seq.parameters():
        torch.nn.init.normal_(p, std=0.02)
    emb = torch.randn(3, 5120, device=DEV)
    assert rel_err(modulation(seq, emb), seq.double()(emb.double())) < 4e-6


def test_modulation_gradients_without_the_kernel():
    """A width that is no multiple of four runs the PyTorch formulas."""
    from aeris_gb_b200.models.fused import GemvLinearFn
    W, b, x = (torch.randn(*s, device=DEV, requires_grad=True) for s in ((6, 101), (6,), (2, 101)))
    GemvLinearFn.apply(x, W, b, True).sum().backward()
    got = [v.grad.clone() for v in (W, b, x)]
    for v in (W, b, x):
        v.grad = None
    (torch.nn.functional.silu(x) @ W.t() + b).sum().backward()
    for g, v in zip(got, (W, b, x)):
        assert rel_err(g, v.grad) < 1e-5


def test_noise_embedding_matches_the_oracle():
    from aeris_gb_b200.models import oracle as O
    from aeris_gb_b200.ops import diffusion as DF
    t = torch.tensor([0.0, 0.3, 1.5707963], device=DEV)
    ref = O.timestep_embedding(t.double(), 256, 10_000.0)
    assert rel_err(DF.noise_embedding(t, 256, 10_000.0, torch.float32), ref) < 1e-7
    assert rel_err(DF.noise_embedding(t, 256, 10_000.0, torch.bfloat16), ref) < 2.0 ** -9


def test_packed_weights_of_the_ends():
    from aeris_gb_b200.ops import diffusion as DF
    W, b = torch.randn(130, 20, device=DEV), torch.randn(130, device=DEV)
    p = DF.pack_embed_weights(W, b, 128)
    hi, lo = W.bfloat16(), (W - W.bfloat16().float()).bfloat16()
    bh, bl = b.bfloat16(), (b - b.bfloat16().float()).bfloat16()
    assert torch.equal(p, torch.cat([hi, hi, lo, bh[:, None], bl[:, None], torch.zeros(130, 66, device=DEV).bfloat16()], 1))
    G, dW, db = torch.randn(130, 128, device=DEV), torch.ones(130, 20, device=DEV), torch.ones(130, device=DEV)
    DF.fold_embed_grad(G, dW, db)
    assert torch.equal(dW, 1 + (G[:, :20] + G[:, 20:40])) and torch.equal(db, 1 + G[:, 60])
    w3 = DF.pack_head_weights(W, 256)
    assert torch.equal(w3[:130], torch.cat([hi, lo, hi], 1)) and not w3[130:].any()


@pytest.mark.parametrize("n,rows,D", [(1, 1, 64), (130, 200, 128), (1000, 1000, 384), (257, 300, 1536)])
def test_head_product_of_split_operands(n, rows, D):
    """hi and lo rows in two blocks (rows that are no multiple of a tile, a block longer than the rows in use), against
    fp64: what is dropped is lo x lo, 2^-17 of a term at most, and the tensor core's fp32 sums."""
    from aeris_gb_b200.ops import diffusion as DF
    v, W = torch.randn(n, D, device=DEV), torch.randn(70, D, device=DEV)
    y = torch.full((2, rows, D), float("nan"), dtype=torch.bfloat16, device=DEV)
    y[0, :n] = v.bfloat16()
    y[1, :n] = (v - y[0, :n].float()).bfloat16()
    out = torch.full((n + 1, 128), 7.0, device=DEV)
    DF.head_gemm(y, n, DF.pack_head_weights(W, 128), out)
    assert rel_err(out[:n, :70], v.double() @ W.double().t()) < 2.0 ** -16 and not out[:n, 70:].any()
    assert (out[n:] == 7).all()
