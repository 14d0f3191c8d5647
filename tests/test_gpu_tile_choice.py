"""Tiles chosen by the size of a pass: transforms and batches on both sides of
every line the choice draws, against FP64 (bound: eps * log2 of the points,
eps = 2^-23, each side's own error being about half of it)."""
from __future__ import annotations

import ctypes

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


# (points, batch): one tile with ragged last tiles; four-step columns and rows of
# 256 .. 2048 points with few and many CTAs; three-level 128-point columns
@pytest.mark.parametrize("lg,batch", [(4, 131), (5, 131), (6, 35), (7, 19), (8, 9), (9, 5), (10, 3), (15, 1), (15, 70),
                                      (16, 1), (16, 20), (17, 40), (18, 1), (18, 19), (19, 1), (19, 11), (20, 1),
                                      (20, 3), (21, 1), (22, 1)])
def test_1d(gpu, lg, batch):
    import torch
    n = 1 << lg
    st = torch.cuda.current_stream().cuda_stream
    x = signals.complex_uniform(85000 + lg, n * batch).reshape(batch, n)
    dx = torch.from_numpy(x).cuda()
    dy, dz = torch.empty_like(dx), torch.empty_like(dx)
    plans = [gpu.gb_create_plan_1d(0, n, d, 0, batch, 0, 0, None) for d in (K.FORWARD, K.INVERSE)]
    assert all(plans)
    assert gpu.gb_execute_plan_1d_async(plans[0], dy.data_ptr(), dx.data_ptr(), st) == 0
    assert gpu.gb_execute_plan_1d_async(plans[1], dz.data_ptr(), dy.data_ptr(), st) == 0
    torch.cuda.synchronize()
    rows = sorted({0, batch // 2, batch - 1})
    got = dy[rows].cpu().numpy()
    assert rel_l2(got, np.fft.fft(x[rows].astype(np.complex128), axis=1)) <= 2.0 ** -23 * lg
    assert rel_l2(dz.cpu().numpy() / n, x) <= 2 * 2.0 ** -23 * lg
    for p in plans:
        gpu.free_plan_1d(p)


@pytest.mark.parametrize("batch", [1023, 1024])
def test_real_rows_of_1024(gpu, batch):
    import torch
    n = 2048
    st = torch.cuda.current_stream().cuda_stream
    x = signals.uniform(86000, n * batch).reshape(batch, n).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    dX = torch.empty((batch, n // 2 + 1), dtype=torch.complex64, device="cuda")
    back = torch.empty_like(dx)
    plans = [gpu.gb_create_plan_1d(k, n, 0, 0, batch, 0, 0, None) for k in (1, 2)]
    assert gpu.gb_execute_plan_1d_async(plans[0], dX.data_ptr(), dx.data_ptr(), st) == 0
    assert gpu.gb_execute_plan_1d_async(plans[1], back.data_ptr(), dX.data_ptr(), st) == 0
    torch.cuda.synchronize()
    assert rel_l2(dX.cpu().numpy(), np.fft.rfft(x.astype(np.float64), axis=1)) <= 2.0 ** -23 * 11
    assert rel_l2(back.cpu().numpy() / n, x) <= 2 * 2.0 ** -23 * 11
    for p in plans:
        gpu.free_plan_1d(p)


# column tiles of 64 .. 2048 points, one and two column passes of 4096, widths with a ragged last tile (r2c, c2r)
@pytest.mark.parametrize("nx,ny", [(32, 64), (128, 128), (1024, 256), (8192, 256), (256, 512), (16384, 512), (64, 1024),
                                   (1024, 2048), (2048, 2048), (512, 4096), (1024, 4096)])
def test_2d(gpu, nx, ny):
    lg = (nx * ny).bit_length() - 1
    x = signals.uniform(87000 + nx + ny, nx * ny).reshape(ny, nx)
    want = np.fft.rfft2(x.astype(np.float64))
    X = gpu.fft2_r2c(x)
    assert rel_l2(X[:, : nx // 2 + 1], want) <= 2.0 ** -23 * lg
    assert rel_l2(gpu.fft2_c2r(X) / (nx * ny), x) <= 2 * 2.0 ** -23 * lg
    z = signals.complex_uniform(87500 + nx + ny, nx * ny).reshape(ny, nx)
    assert rel_l2(gpu.fft2_c2c(z, K.INVERSE), np.fft.ifft2(z.astype(np.complex128)) * (nx * ny)) <= 2.0 ** -23 * lg


def test_caller_choice_wins(gpu):
    """A tile the caller prefers is used at any size."""
    buf = ctypes.create_string_buffer(4096)
    opts = gpu.options(tiles=[(512, 0, 0, 8, 16, 1)])
    assert gpu.gb_describe_schedule_1d(512, 0, K.FORWARD, 0, 5000, ctypes.byref(opts), buf, 4096) == 0
    assert b"L=512 R=16 C=8" in buf.value
    assert gpu.gb_describe_schedule_1d(512, 0, K.FORWARD, 0, 5000, None, buf, 4096) == 0
    assert b"L=512 R=32 C=2" in buf.value
