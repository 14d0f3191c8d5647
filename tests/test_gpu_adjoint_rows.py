"""The filter adjoint's reduction over signals: one row of signals, several
rows with uneven shares, more rows than fill one chunk -- against FP64.

Bound: every spectrum carries a relative error of about eps/2 * log2(N)
(eps = 2^-23) and the FP32 sum of `batch` terms at most eps/2 * log2-ish
growth by rows and in-row chains of at most batch / rows terms, whose rounding
errors are independent: eps * (log2(N) + sqrt(batch)) covers both."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,stereo", [(32, 700, True), (32, 15, False), (64, 513, False), (1024, 9, True),
                                            (1024, 8, False), (8192, 131, True), (8192, 131, False),
                                            (1 << 16, 17, True)])
def test_filter_adjoint_rows(n, batch, stereo):
    import torch

    import mufft_gb300
    gpu = mufft_gb300.load()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(n * 7 + batch)

    def draw(*shape):
        if stereo:
            return torch.view_as_complex(torch.rand((*shape, 2), device="cuda", generator=g) * 2 - 1)
        return torch.rand(shape, device="cuda", generator=g) * 2 - 1
    plan = gpu.create_plan_conv(n, 0, 1 if stereo else 0)
    bins = gpu.conv_get_transformed_block_size(plan) // 8
    x, r = draw(batch, n), draw(batch, n)
    A = torch.zeros((batch, bins), dtype=torch.complex64, device="cuda")
    for b in range(batch):
        assert gpu.gb_execute_conv_input_async(plan, 0, A[b].data_ptr(), x[b].data_ptr(), st) == 0
    got = [torch.empty(n, device="cuda") for _ in range(2)]
    assert gpu.gb_conv_adjoint_filter(plan, got[0].data_ptr(), r.data_ptr(), n, A.data_ptr(), bins, batch, st) == 0
    assert gpu.gb_conv_adjoint(plan, got[1].data_ptr(), None, 0, r.data_ptr(), n, A.data_ptr(), bins, None, batch,
                               st) == 0
    torch.cuda.synchronize()
    gpu.free_plan_conv(plan)
    X = np.fft.fft(x.cpu().numpy().astype(np.complex128), axis=1)
    R = np.fft.fft(r.cpu().numpy().astype(np.complex128), axis=1)
    want = np.fft.ifft((R * X.conj()).sum(axis=0)).real
    bound = 2.0 ** -23 * (np.log2(n) + np.sqrt(batch))
    for v in got:
        assert rel_l2(v.cpu().numpy(), want) <= bound
