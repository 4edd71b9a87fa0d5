"""A kernel that cannot be launched: the entry point says so. The launches go to a stream whose capture has been invalidated,
where the runtime refuses every one of them and nothing runs."""
import ctypes

import pytest
import torch

from aeris_gb_b200.ops import lib as L

gpu = pytest.mark.gpu
V = ctypes.c_void_p
LAUNCH_FAILED = -21


@pytest.fixture
def refusing():
    """A stream that takes no more launches."""
    from cuda.bindings import runtime as R
    torch.zeros(1, device="cuda")                      # the context is there
    err, stream = R.cudaStreamCreateWithFlags(R.cudaStreamNonBlocking)
    assert err == R.cudaError_t.cudaSuccess
    assert R.cudaStreamBeginCapture(stream, R.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)[0] == R.cudaError_t.cudaSuccess
    assert R.cudaStreamSynchronize(stream)[0] != R.cudaError_t.cudaSuccess           # not allowed: ends the capture
    yield V(int(stream))
    assert R.cudaStreamEndCapture(stream)[0] != R.cudaError_t.cudaSuccess
    R.cudaGetLastError()
    assert R.cudaStreamDestroy(stream)[0] == R.cudaError_t.cudaSuccess


@gpu
@pytest.mark.parametrize("D", [64, 256, 2048, 5120, 6144])
def test_modnorm_backward(refusing, D):
    rows, dev = 16, "cuda"
    x, dh, dx = (torch.zeros(rows, D, dtype=torch.bfloat16, device=dev) for _ in range(3))
    w = torch.ones(D, dtype=torch.bfloat16, device=dev)
    s, t, ds, dt, dw, sums = (torch.zeros(4, 3, D, device=dev) for _ in range(6))
    dh32, w32 = dh.float(), w.float()
    p, eps = L.ptr, ctypes.c_float(1e-6)
    rc = L.lib().aeris_modnorm_bwd(p(x), p(dh), V(0), p(s), p(t), p(w), p(dx), p(ds), p(dt), p(dw), rows, D, 0, eps, V(0),
                                   refusing)
    assert rc == LAUNCH_FAILED
    if D <= 5120:
        rc = L.lib().aeris_modnorm_bwd_f32(p(x), p(dh32), p(s), p(t), p(w32), p(dx), p(ds), p(dt), p(dw), p(sums), 4, rows, D,
                                           0, eps, refusing)
        assert rc == LAUNCH_FAILED


@gpu
def test_chained_launches(refusing):
    """The launches around it, a few of every kind."""
    rows, D, dev = 128, 256, "cuda"
    a, b, c = (torch.zeros(rows, D, dtype=torch.bfloat16, device=dev) for _ in range(3))
    f = torch.zeros(rows, D, device=dev)
    p, eps, lib = L.ptr, ctypes.c_float(1e-6), L.lib()
    rcs = [lib.aeris_modnorm_fwd(p(a), V(0), V(0), 0, V(0), p(f), p(f), p(b), p(c), rows, D, 0, eps, V(0), V(0), refusing),
           lib.aeris_rope_qk(p(a), p(f), p(f), ctypes.c_longlong(32), 32, 1, 64, 0, refusing)]
    for two_cta in (0, 2):
        rcs.append(lib.aeris_gemm_auto(p(a), p(b), p(c), rows, rows, D, D, D, D, 0, 0, 0, V(0), 0, V(0), 0, 0, V(0), 0, 0, 1, 0,
                                       two_cta, V(0), refusing))
    assert rcs == [LAUNCH_FAILED] * 4
