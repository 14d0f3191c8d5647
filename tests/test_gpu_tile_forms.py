"""Tile kernels compiled for one prologue and epilogue: a zero-padded transform
equals the plain transform of the same input with its zeros written out, each
side a form of its own.  (The kernels that decide prologue and epilogue at run
time: test_column_twiddle_forms, and test_gpu_runtime_forms.py.)

Both sides round independently, each with a relative L2 error of at most
about eps/2 * log2(N) (eps = 2^-23), so they may differ by eps * log2(N)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_l2
from mufft_gb300 import capi as K
from mufft_gb300 import signals

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import mufft_gb300
    return mufft_gb300.load()


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available()
    return t


def _run(gpu, torch, kind, N, direction, flags, x, out_shape, opts=None):
    import ctypes
    B = x.shape[0]
    dx = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    dy = torch.zeros(out_shape, dtype=torch.complex64, device="cuda")
    plan = gpu.gb_create_plan_1d(kind, N, direction, flags, B, 0, 0, ctypes.byref(opts) if opts else None)
    assert plan, gpu.gb_last_error_string()
    assert gpu.gb_execute_plan_1d_async(plan, dy.data_ptr(), dx.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    gpu.free_plan_1d(plan)
    return dy.cpu().numpy()


@pytest.mark.parametrize("lg,B", [(1, 300), (4, 257), (5, 129), (6, 65), (9, 9), (10, 3), (12, 5), (13, 3), (14, 3),
                                  (15, 3), (17, 3), (21, 2), (22, 2), (24, 1)])
@pytest.mark.parametrize("direction", [K.FORWARD, K.INVERSE])
def test_c2c_forms(gpu, torch, lg, B, direction):
    N = 1 << lg
    xh = signals.complex_uniform(81000 + lg, B * N // 2).reshape(B, N // 2)
    x = np.concatenate([xh, np.zeros_like(xh)], axis=1)
    a = _run(gpu, torch, 0, N, direction, 0, x, (B, N))
    b = _run(gpu, torch, 0, N, direction, K.FLAG_ZERO_PAD_UPPER_HALF, xh, (B, N))
    assert rel_l2(a, b) <= 2.0 ** -23 * lg


@pytest.mark.parametrize("lg,B", [(2, 300), (5, 129), (6, 65), (10, 9), (11, 3), (13, 3), (14, 3), (15, 3), (18, 3)])
def test_r2c_forms(gpu, torch, lg, B):
    N = 1 << lg
    xh = signals.uniform(82000 + lg, B * N // 2).reshape(B, N // 2).astype(np.float32)
    x = np.concatenate([xh, np.zeros_like(xh)], axis=1)
    a = _run(gpu, torch, 1, N, K.FORWARD, 0, x, (B, N // 2 + 1))
    b = _run(gpu, torch, 1, N, K.FORWARD, K.FLAG_ZERO_PAD_UPPER_HALF, xh, (B, N // 2 + 1))
    assert rel_l2(a, b) <= 2.0 ** -23 * lg


@pytest.mark.parametrize("mode", [1, 2])
def test_column_twiddle_forms(gpu, torch, mode):
    """Four-step columns by table (the run-time form) and by column powers."""
    N, B = 1 << 17, 3
    x = signals.complex_uniform(83000, B * N).reshape(B, N)
    ref = np.fft.fft(x.astype(np.complex128), axis=1)
    got = _run(gpu, torch, 0, N, K.FORWARD, 0, x, (B, N), gpu.options(twiddle_table=mode))
    assert rel_l2(got, ref) <= 2.0 ** -23 * 17


@pytest.mark.parametrize("tile", [(512, 0, 0, 2, 32, 1), (512, 0, 0, 8, 16, 1), (1024, 0, 0, 1, 32, 1), (8192, 0, 0, 1, 32, 1),
                                  (8192, 0, 0, 1, 16, 1), (16384, 0, 0, 1, 32, 1), (16384, 0, 0, 1, 16, 1)])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_wide_radix_rows(gpu, torch, tile, kind):
    """Row tiles of 16 and of 32 elements a thread (radix-32 stages), every kind."""
    L, B = tile[0], 17
    N = L if kind == 0 else 2 * L
    lg = N.bit_length() - 1
    opts = gpu.options(tiles=[tile])
    x = signals.complex_uniform(84000 + N + kind, B * N).reshape(B, N)
    if kind == 0:
        got = _run(gpu, torch, 0, N, K.INVERSE, 0, x, (B, N), opts)
        assert rel_l2(got, np.fft.ifft(x.astype(np.complex128), axis=1) * N) <= 2.0 ** -23 * lg
        return
    xr = np.ascontiguousarray(x.real)
    X = np.fft.rfft(xr.astype(np.float64), axis=1)
    if kind == 1:
        assert rel_l2(_run(gpu, torch, 1, N, K.FORWARD, 0, xr, (B, N // 2 + 1), opts), X) <= 2.0 ** -23 * lg
        return
    Xs = X.astype(np.complex64)
    back = _run(gpu, torch, 2, N, K.INVERSE, 0, Xs, (B, N // 2), opts).view(np.float32)
    assert rel_l2(back, np.fft.irfft(Xs.astype(np.complex128), axis=1) * N) <= 2.0 ** -23 * lg
