"""Blocking executes on page-locked host memory: the same bits as the same
plan's asynchronous execute on device buffers, whether the kernel takes the
host memory itself (small, aligned, apart) or it is staged (in place,
misaligned, partly device, large, several passes)."""
from __future__ import annotations

import numpy as np
import pytest

from mufft_gb300 import capi as K

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import mufft_gb300
    return mufft_gb300.load()


class Pinned:
    def __init__(self, gpu, nbytes):
        self.gpu, self.addr = gpu, gpu.alloc(nbytes)
        self.__array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (self.addr, False), "version": 3}

    def __del__(self):
        self.gpu.free(self.addr)


def _view(p, offset, count, dtype):
    return np.asarray(p)[offset: offset + count * np.dtype(dtype).itemsize].view(dtype)


@pytest.mark.parametrize("kind,n", [(0, 2), (0, 64), (0, 1024), (0, 16384), (0, 1 << 17), (1, 4), (1, 2048),
                                    (1, 1 << 16), (2, 4), (2, 2048), (2, 32768)])
@pytest.mark.parametrize("how", ["apart", "in_place", "misaligned", "device_out"])
def test_pinned(gpu, kind, n, how):
    import torch
    rng = np.random.default_rng(n + kind)
    nin = (2 * n, n, n + 2)[kind]  # floats
    nout = (2 * n, n + 2, n)[kind]
    x = rng.uniform(-1, 1, nin).astype(np.float32)
    if kind == 2:
        x[1] = x[-1] = 0
    plan = gpu.gb_create_plan_1d(kind, n, K.FORWARD, 0, 1, 0, 0, None)
    assert plan
    dx = torch.from_numpy(x).cuda()
    dy = torch.empty(nout, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert gpu.gb_execute_plan_1d_async(plan, dy.data_ptr(), dx.data_ptr(), st) == 0
    want = dy.cpu().numpy()
    off = 4 if how == "misaligned" else 0
    src = Pinned(gpu, 4 * max(nin, nout) + 64)
    dst = src if how == "in_place" else Pinned(gpu, 4 * max(nin, nout) + 64)
    _view(src, off, nin, np.float32)[...] = x
    for _ in range(1 if how == "in_place" else 2):
        if how == "device_out":
            out = torch.zeros(nout, device="cuda")
            gpu.execute_plan_1d(plan, out.data_ptr(), src.addr)
            got = out.cpu().numpy()
        else:
            gpu.execute_plan_1d(plan, dst.addr + off, src.addr + off)
            got = _view(dst, off, nout, np.float32)
        gpu.check("execute_plan_1d")
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    gpu.free_plan_1d(plan)


@pytest.mark.parametrize("stereo", [False, True])
@pytest.mark.parametrize("same", [False, True])
def test_conv_output_over_its_spectra(gpu, stereo, same):
    """The output buffer on top of the first spectrum (staged) and apart from it."""
    n = 512
    rng = np.random.default_rng(5)
    plan = gpu.create_plan_conv(n, 0, 1 if stereo else 0)
    nblk = gpu.conv_get_transformed_block_size(plan)
    m = 2 * n if stereo else n
    bufs = [Pinned(gpu, 4 * m), Pinned(gpu, 4 * n), Pinned(gpu, max(nblk, 4 * m)), Pinned(gpu, nblk), Pinned(gpu, 4 * m)]
    x, h = rng.uniform(-1, 1, m).astype(np.float32), rng.uniform(-1, 1, n).astype(np.float32)
    _view(bufs[0], 0, m, np.float32)[...] = x
    _view(bufs[1], 0, n, np.float32)[...] = h
    gpu.execute_conv_input(plan, 0, bufs[2].addr, bufs[0].addr)
    gpu.execute_conv_input(plan, 1, bufs[3].addr, bufs[1].addr)
    out = bufs[2] if same else bufs[4]
    gpu.execute_conv_output(plan, out.addr, bufs[2].addr, bufs[3].addr)
    gpu.check("conv")
    xs = x.view(np.complex64) if stereo else x
    want = np.fft.ifft(np.fft.fft(xs.astype(np.complex128)) * np.fft.fft(h.astype(np.float64)))
    got = _view(out, 0, m, np.float32).view(np.complex64) if stereo else _view(out, 0, m, np.float32)
    want = want if stereo else want.real
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 3 * 2.0 ** -23 * 9
    gpu.free_plan_conv(plan)
