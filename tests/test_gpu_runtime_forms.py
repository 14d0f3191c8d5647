"""The tile kernels that decide prologue and epilogue at run time, each against
FP64: full-spectrum r2c rows, and multi-pass transforms and convolutions whose
column twiddles are not column powers (twiddle_table 0 and 1; 2, the compiled
forms, beside them).

Bound per transform: eps * log2(N), eps = 2^-23 (each side's own error is about
half of it); a convolution is three of them."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import rel_l2
from mufft_gb300 import capi as K
from mufft_gb300 import signals

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -23


@pytest.fixture(scope="module")
def gpu():
    import mufft_gb300
    return mufft_gb300.load()


def _run(gpu, kind, N, direction, flags, x, out_shape, out_dtype, opts=None):
    import torch
    dx = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    dy = torch.zeros(out_shape, dtype=out_dtype, device="cuda")
    plan = gpu.gb_create_plan_1d(kind, N, direction, flags, x.shape[0], 0, 0, ctypes.byref(opts) if opts else None)
    assert plan, gpu.gb_last_error_string()
    st = torch.cuda.current_stream().cuda_stream
    assert gpu.gb_execute_plan_1d_async(plan, dy.data_ptr(), dx.data_ptr(), st) == 0
    torch.cuda.synchronize()
    gpu.free_plan_1d(plan)
    return dy.cpu().numpy()


@pytest.mark.parametrize("lg", range(2, 16))
@pytest.mark.parametrize("pad", [0, K.FLAG_ZERO_PAD_UPPER_HALF])
def test_full_spectrum_rows(gpu, lg, pad):
    import torch
    N, B = 1 << lg, 5
    m = N // 2 if pad else N
    x = signals.uniform(91000 + lg, B * m).reshape(B, m).astype(np.float32)
    want = np.fft.fft(x.astype(np.float64), n=N, axis=1)
    full = _run(gpu, 1, N, K.FORWARD, pad | K.FLAG_FULL_R2C, x, (B, N), torch.complex64)
    half = _run(gpu, 1, N, K.FORWARD, pad, x, (B, N // 2 + 1), torch.complex64)
    assert rel_l2(full, want) <= EPS * lg
    assert rel_l2(half, want[:, : N // 2 + 1]) <= EPS * lg


@pytest.mark.parametrize("lg, B", [(15, 3), (17, 2), (18, 3), (20, 2), (22, 1)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_multi_pass(gpu, lg, B, mode):
    import torch
    o = gpu.options(twiddle_table=mode)
    N = 1 << lg
    z = signals.complex_uniform(92000 + lg, B * N).reshape(B, N)
    w = z.astype(np.complex128)
    for d, ref in ((K.FORWARD, np.fft.fft(w, axis=1)), (K.INVERSE, np.fft.ifft(w, axis=1) * N)):
        assert rel_l2(_run(gpu, 0, N, d, 0, z, (B, N), torch.complex64, o), ref) <= EPS * lg
    h = np.ascontiguousarray(z[:, : N // 2])
    got = _run(gpu, 0, N, K.FORWARD, K.FLAG_ZERO_PAD_UPPER_HALF, h, (B, N), torch.complex64, o)
    assert rel_l2(got, np.fft.fft(h.astype(np.complex128), n=N, axis=1)) <= EPS * lg
    # real transforms of twice the points: the same column passes
    R = 2 * N
    x = signals.uniform(93000 + lg, B * R).reshape(B, R).astype(np.float32)
    X = np.fft.rfft(x.astype(np.float64), axis=1)
    assert rel_l2(_run(gpu, 1, R, K.FORWARD, 0, x, (B, N + 1), torch.complex64, o), X) <= EPS * (lg + 1)
    xh = np.ascontiguousarray(x[:, :N])
    got = _run(gpu, 1, R, K.FORWARD, K.FLAG_ZERO_PAD_UPPER_HALF, xh, (B, N + 1), torch.complex64, o)
    assert rel_l2(got, np.fft.rfft(xh.astype(np.float64), n=R, axis=1)) <= EPS * (lg + 1)
    Xs = X.astype(np.complex64)
    back = _run(gpu, 2, R, K.INVERSE, 0, Xs, (B, R), torch.float32, o)
    assert rel_l2(back, np.fft.irfft(Xs.astype(np.complex128), n=R, axis=1) * R) <= EPS * (lg + 1)


@pytest.mark.parametrize("lg", [16, 18, 20])
@pytest.mark.parametrize("stereo", [0, 1])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_convolution(gpu, lg, stereo, mode):
    import torch
    o = gpu.options(twiddle_table=mode)
    N = 1 << lg
    plan = gpu.gb_create_plan_conv(N, 0, stereo, ctypes.byref(o))
    assert plan, gpu.gb_last_error_string()
    bins = gpu.conv_get_transformed_block_size(plan) // 8
    a = signals.complex_uniform(94000 + lg, N) if stereo else signals.uniform(94000 + lg, N).astype(np.float32)
    b = signals.uniform(95000 + lg, N).astype(np.float32)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    sa, sb = (torch.empty(bins, dtype=torch.complex64, device="cuda") for _ in range(2))
    out = torch.empty_like(da)
    st = torch.cuda.current_stream().cuda_stream
    assert gpu.gb_execute_conv_input_async(plan, 0, sa.data_ptr(), da.data_ptr(), st) == 0
    assert gpu.gb_execute_conv_input_async(plan, 1, sb.data_ptr(), db.data_ptr(), st) == 0
    assert gpu.gb_execute_conv_output_async(plan, out.data_ptr(), sa.data_ptr(), sb.data_ptr(), st) == 0
    torch.cuda.synchronize()
    gpu.free_plan_conv(plan)
    want = np.fft.ifft(np.fft.fft(a.astype(np.complex128)) * np.fft.fft(b.astype(np.float64)))
    assert rel_l2(out.cpu().numpy(), want if stereo else want.real) <= 3 * EPS * lg


# 4096 rows: the automatic choice goes through two column passes below 400
# columns, and one pass was asked for beside it
@pytest.mark.parametrize("nx", [2, 4, 64, 256, 512])
def test_narrow_grids_of_4096_rows(gpu, nx):
    ny = 4096
    lg = (nx * ny).bit_length() - 1
    z = signals.complex_uniform(96000 + nx, nx * ny).reshape(ny, nx)
    w = z.astype(np.complex128)
    one = gpu.options(columns_2d=1)
    for d, ref in ((K.FORWARD, np.fft.fft2(w)), (K.INVERSE, np.fft.ifft2(w) * (nx * ny))):
        assert rel_l2(gpu.fft2_c2c(z, d), ref) <= EPS * lg
        assert rel_l2(gpu.fft2_c2c(z, d, opts=one), ref) <= EPS * lg


def test_persistent_columns_with_few_tiles(gpu):
    """64 columns of 4096 points in one pass: a persistent grid of fewer tiles
    than SMs, the same bits as one launch per tile, for every kind."""
    nx, ny = 64, 4096
    lg = (nx * ny).bit_length() - 1
    on, off = (gpu.options(columns_2d=1, persistent_tiles=v) for v in (1, 0))
    text = ctypes.create_string_buffer(4096)
    assert gpu.gb_describe_schedule_2d(0, nx, ny, K.FORWARD, 0, ctypes.byref(on), text, 4096) == 0
    assert b"persistent" in text.value
    same = lambda u, v: np.array_equal(u.view(np.uint32), v.view(np.uint32))  # noqa: E731
    x = signals.uniform(97000, nx * ny).reshape(ny, nx)
    a, b = gpu.fft2_r2c(x, opts=on), gpu.fft2_r2c(x, opts=off)
    assert same(a, b)
    assert rel_l2(a[:, : nx // 2 + 1], np.fft.rfft2(x.astype(np.float64))) <= EPS * lg
    back, back0 = gpu.fft2_c2r(a, opts=on), gpu.fft2_c2r(a, opts=off)
    assert same(back, back0)
    assert rel_l2(back / (nx * ny), x) <= 2 * EPS * lg
    z = signals.complex_uniform(98000, nx * ny).reshape(ny, nx)
    for d, ref in ((K.FORWARD, np.fft.fft2(z.astype(np.complex128))),
                   (K.INVERSE, np.fft.ifft2(z.astype(np.complex128)) * (nx * ny))):
        a, b = gpu.fft2_c2c(z, d, opts=on), gpu.fft2_c2c(z, d, opts=off)
        assert same(a, b)
        assert rel_l2(a, ref) <= EPS * lg
