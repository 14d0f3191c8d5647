"""Class pipelines of the ragged convolution batch (column pass, rows with the
multiply, column pass): every size and method they take, zero-padded and
whole inputs, one and several requests a class, against FP64.

Bound: each of the two transforms errs by about eps/2 * log2(N) (eps = 2^-23),
as does the filter's spectrum: 1.5 eps log2(N) in all, doubled for the noise of
a bound on relative L2."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_l2
from mufft_gb300 import capi as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,stereo", [(1 << 14, True), (1 << 15, True), (1 << 16, True), (1 << 15, False),
                                      (1 << 16, False)])
@pytest.mark.parametrize("pad", [False, True])
@pytest.mark.parametrize("count", [1, 3])
def test_class(n, stereo, pad, count):
    import torch

    import mufft_gb300
    gpu = mufft_gb300.load()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(n + count)
    m = n // 2 if pad else n
    method = (1 if stereo else 0) | ((K.CONV_METHOD_FLAG_ZERO_PAD_UPPER_HALF_FIRST |
                                      K.CONV_METHOD_FLAG_ZERO_PAD_UPPER_HALF_SECOND) if pad else 0)
    shape = (count, m, 2) if stereo else (count, m)
    x = torch.rand(shape, device="cuda", generator=g) * 2 - 1
    x = torch.view_as_complex(x) if stereo else x
    h = torch.randn((count, m), device="cuda", generator=g)
    plan = gpu.create_plan_conv(n, 0, method)
    bins = gpu.conv_get_transformed_block_size(plan) // 8
    H = torch.zeros((count, bins), dtype=torch.complex64, device="cuda")
    out = torch.zeros((count, n), dtype=x.dtype, device="cuda")
    reqs = (K.ConvRequest * count)()
    for i in range(count):
        assert gpu.gb_execute_conv_input_async(plan, 1, H[i].data_ptr(), h[i].data_ptr(), st) == 0
        reqs[i] = K.ConvRequest(n, method, x[i].data_ptr(), H[i].data_ptr(), out[i].data_ptr())
    batch = gpu.gb_create_conv_batch(reqs, count, 0, None)
    assert batch, gpu.gb_last_error_string()
    assert gpu.gb_conv_batch_class_size(batch) == 16384
    for _ in range(2):
        out.zero_()
        assert gpu.gb_execute_conv_batch(batch, st) == 0
        torch.cuda.synchronize()
        want = np.fft.ifft(np.fft.fft(x.cpu().numpy().astype(np.complex128), n, axis=1) *
                           np.fft.fft(h.cpu().numpy().astype(np.complex128), n, axis=1), axis=1)
        want = want if stereo else want.real
        assert rel_l2(out.cpu().numpy(), want) <= 3 * 2.0 ** -23 * np.log2(n)
    gpu.gb_free_conv_batch(batch)
    gpu.free_plan_conv(plan)
