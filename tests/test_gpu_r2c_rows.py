"""Four-step r2c whose row pass resolves the bins: every split it takes, few
and many transforms (narrow and wide tiles), packed and full outputs, zero
padding, padded distances -- against FP64 (bound: eps * log2(N), eps = 2^-23)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from helpers import rel_l2
from mufft_gb300 import capi as K
from mufft_gb300 import signals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg,batch", [(16, 1), (16, 60), (17, 2), (17, 41), (18, 1), (18, 21), (19, 3), (19, 20)])
@pytest.mark.parametrize("flags", [0, K.FLAG_FULL_R2C, K.FLAG_ZERO_PAD_UPPER_HALF])
def test_r2c_rows(lg, batch, flags):
    import torch

    import mufft_gb300
    gpu = mufft_gb300.load()
    n = 1 << lg
    m = n // 2 if flags & K.FLAG_ZERO_PAD_UPPER_HALF else n
    nout = n if flags & K.FLAG_FULL_R2C else n // 2 + 1
    x = signals.uniform(88000 + lg, m * batch).reshape(batch, m).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    dist = nout + 5
    dX = torch.zeros((batch, dist), dtype=torch.complex64, device="cuda")
    plan = gpu.gb_create_plan_1d_r2c_batched(n, flags, batch, 0, dist)
    assert plan, gpu.gb_last_error_string()
    buf = ctypes.create_string_buffer(4096)
    gpu.gb_plan_1d_describe(plan, buf, 4096)
    assert b"r2c_rows" in buf.value and b"fixup" not in buf.value
    st = torch.cuda.current_stream().cuda_stream
    for _ in range(2):
        assert gpu.gb_execute_plan_1d_async(plan, dX.data_ptr(), dx.data_ptr(), st) == 0
    torch.cuda.synchronize()
    gpu.free_plan_1d(plan)
    got = dX.cpu().numpy()
    assert np.all(got[:, nout:] == 0)  # nothing past a transform's bins
    rows = sorted({0, batch // 2, batch - 1})
    want = np.fft.fft(x[rows].astype(np.float64), n, axis=1)[:, :nout]
    assert rel_l2(got[rows, :nout], want) <= 2.0 ** -23 * lg
