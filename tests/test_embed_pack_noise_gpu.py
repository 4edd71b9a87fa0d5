"""Packed rows of the noised input against PyTorch with the generator's own noise: one and two channels a lane, last groups of
four that are not full, rows that begin inside a warp's share and inside a window, sequence ranks, blocks of a larger image,
outputs that do not start on 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ws_y,ws_x,nwy,nwx,sp,B,cx,cc,row0,y0,x0,shift", [
    (30, 30, 4, 8, 1, 1, 69, 71, 0, 0, 0, 0),
    (30, 30, 4, 8, 1, 1, 69, 70, 7, 0, 0, 0),
    (15, 9, 3, 40, 1, 2, 70, 74, 131, 15, 36, 0),
    (8, 8, 2, 3, 4, 2, 17, 18, 5, 0, 0, 2),
    (6, 10, 7, 90, 4, 1, 18, 0, 3, 12, 0, 0),
    (1, 1, 5, 7, 1, 3, 1, 2, 0, 0, 0, 0),
    (12, 20, 5, 12, 1, 1, 127, 129, 1000, 0, 20, 4)])
def test_packed_rows_with_noise(ws_y, ws_x, nwy, nwx, sp, B, cx, cc, row0, y0, x0, shift):
    from aeris_gb_b200.ops import diffusion as DF
    torch.manual_seed(cx + cc)
    H, W, C, n_local = ws_y * nwy, ws_x * nwx, cx + cc, ws_y * ws_x // sp
    x, cond = torch.randn(B, H, W, cx, device="cuda"), torch.randn(B, H, W, cc, device="cuda")
    cs = torch.rand(B, 2, device="cuda") + 0.1
    ch = C // 2 - C // 2 % 2 if cx % 2 == 0 else C // 2
    full_h, full_w, seed, sd = H + y0, W + x0, (3 << 32) + 5, 0.7
    ay, ax = torch.randn(full_h, ch, device="cuda"), torch.randn(full_w, ch, device="cuda")
    KP = (3 * C + 2 + 7) // 8 * 8
    for rank in range(sp):
        g = DF.TokGeom(B, nwy, nwx, ws_y, ws_x, n_local, rank, y0, x0, full_h, full_w, 2)
        z = DF.noise_mix(torch.empty_like(x), 0.0, 1.0, seed, g)
        rows = g.rows - row0
        buf = torch.full((rows * KP + 16,), 9.0, device="cuda", dtype=torch.bfloat16)
        out = buf[shift:shift + rows * KP].view(rows, KP)
        DF.embed_pack(x, cond if cc else None, cs, g, ay, ax, seed, sd, True, out, row0=row0)
        v = (x.double() * cs[:, 0].view(B, 1, 1, 1) + z.double() * sd * cs[:, 1].view(B, 1, 1, 1)) / sd
        v = torch.cat([v, cond.double()], -1)
        v[..., :ch] += ay[y0:].view(1, H, 1, ch)
        v[..., ch:2 * ch] += ax[x0:].view(1, 1, W, ch)
        tok = v.view(B, nwy, ws_y, nwx, ws_x, C).transpose(2, 3).reshape(B, nwy * nwx, ws_y * ws_x, C)
        tok = tok[:, :, rank * n_local:(rank + 1) * n_local].reshape(-1, C)[row0:]
        # eight bits in each part: 2^-17 of a value; half a dozen roundings of 2^-24 of the largest addend before
        got = out[:, :C].double() + out[:, C:2 * C].double()
        assert (got - tok).abs().max() <= 2.0 ** -16 * tok.abs().max()
        assert torch.equal(out[:, :C], out[:, 2 * C:3 * C])
        assert bool((out[:, 3 * C:3 * C + 2] == 1).all()) and not out[:, 3 * C + 2:].any()
        assert bool((buf[:shift] == 9).all()) and bool((buf[shift + rows * KP:] == 9).all())
