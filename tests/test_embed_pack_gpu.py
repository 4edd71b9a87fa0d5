"""Packed rows of the input projection against PyTorch: one and two channels a lane, rows that begin and end inside a warp's
share, inside a window and inside a row of a window, windows cut between sequence ranks, no conditioning, no encoding, rows
wider than needed, outputs that do not start on 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ws_y,ws_x,nwy,nwx,sp,B,cx,cc,row0,ape,pad,shift", [
    (30, 30, 4, 8, 1, 1, 70, 74, 0, True, 0, 0),        # 28,800 rows: five a warp
    (30, 30, 4, 8, 1, 1, 69, 70, 7, True, 8, 0),
    (15, 9, 3, 40, 1, 2, 70, 75, 131, True, 0, 0),
    (8, 8, 2, 3, 4, 2, 16, 18, 0, True, 0, 2),          # sequence ranks: rows start inside a window's row
    (6, 10, 7, 90, 4, 1, 16, 0, 3, True, 0, 0),
    (1, 1, 5, 7, 1, 3, 1, 2, 0, False, 0, 0),
    (12, 20, 5, 12, 1, 1, 128, 128, 0, True, 200, 4)])
def test_packed_rows(ws_y, ws_x, nwy, nwx, sp, B, cx, cc, row0, ape, pad, shift):
    from aeris_gb_b200.ops import diffusion as DF
    torch.manual_seed(cx + cc)
    H, W, C, n_local = ws_y * nwy, ws_x * nwx, cx + cc, ws_y * ws_x // sp
    x, cond = torch.randn(B, H, W, cx, device="cuda"), torch.randn(B, H, W, cc, device="cuda")
    cs = torch.rand(B, 2, device="cuda") + 0.1
    ch = C // 2
    ay, ax = (torch.randn(H, ch, device="cuda"), torch.randn(W, ch, device="cuda")) if ape else (None, None)
    KP = (3 * C + 2 + 7) // 8 * 8 + pad
    sd = 0.7
    for rank in range(sp):
        g = DF.TokGeom(B, nwy, nwx, ws_y, ws_x, n_local, rank, 0, 0, H, W, 0)
        rows = g.rows - row0
        buf = torch.full((rows * KP + 16,), 9.0, device="cuda", dtype=torch.bfloat16)
        out = buf[shift:shift + rows * KP].view(rows, KP)
        DF.embed_pack(x, cond if cc else None, cs, g, ay, ax, 0, sd, False, out, row0=row0)
        v = x * cs[:, 0].view(B, 1, 1, 1) * (torch.ones((), device="cuda") / torch.tensor(sd, device="cuda"))
        v = torch.cat([v, cond], -1)
        if ape:
            v[..., :ch] += ay.view(1, H, 1, ch)
            v[..., ch:2 * ch] += ax.view(1, 1, W, ch)
        tok = v.view(B, nwy, ws_y, nwx, ws_x, C).transpose(2, 3).reshape(B, nwy * nwx, ws_y * ws_x, C)
        tok = tok[:, :, rank * n_local:(rank + 1) * n_local].reshape(-1, C)[row0:]
        hi = tok.bfloat16()
        # the reciprocal of sd and the product with it may be rounded the other way: 2^-22 of a value, 2^-13 of its rest
        got = out[:, :C].double() + out[:, C:2 * C].double()
        assert (got - tok.double()).abs().max() <= 2.0 ** -16 * tok.abs().max()
        assert torch.equal(out[:, :C], out[:, 2 * C:3 * C]) and (out[:, :C] != hi).float().mean() < 1e-3
        assert bool((out[:, 3 * C:3 * C + 2] == 1).all()) and not out[:, 3 * C + 2:].any()
        assert bool((buf[:shift] == 9).all()) and bool((buf[shift + rows * KP:] == 9).all())
