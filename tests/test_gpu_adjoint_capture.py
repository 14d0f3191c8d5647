"""Filter gradients in a captured graph that is replayed after the plan has
served more signals: the graph's partial sums are still the plan's."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


def test_replay_after_more_signals():
    import torch

    import mufft_gb300
    gpu = mufft_gb300.load()
    n, few, many = 256, 16, 700  # 2 and 64 rows of signals
    g = torch.Generator(device="cuda").manual_seed(11)
    draw = lambda *shape: torch.view_as_complex(torch.rand((*shape, 2), device="cuda", generator=g) * 2 - 1)
    plan = gpu.create_plan_conv(n, 0, 1)
    bins = gpu.conv_get_transformed_block_size(plan) // 8
    x, r, H = draw(many, n), draw(many, n), draw(bins)
    A = torch.fft.fft(x).contiguous()
    gx = torch.empty((many, n), dtype=torch.complex64, device="cuda")
    gh = [torch.empty(n, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        st = stream.cuda_stream
        # the spectra's scratch at its largest, then the filter gradient of a few signals
        assert gpu.gb_conv_adjoint(plan, None, gx.data_ptr(), n, r.data_ptr(), n, None, 0, H.data_ptr(), many, st) == 0
        few_args = (plan, gh[0].data_ptr(), r.data_ptr(), n, A.data_ptr(), bins, few)
        assert gpu.gb_conv_adjoint_filter(*few_args, st) == 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rc = gpu.gb_conv_adjoint_filter(*few_args, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    with torch.cuda.stream(stream):
        assert gpu.gb_conv_adjoint_filter(plan, gh[1].data_ptr(), r.data_ptr(), n, A.data_ptr(), bins, many, st) == 0
    torch.cuda.synchronize()
    other = torch.full((1 << 18,), 7.0, device="cuda")  # memory given back would be handed out again
    gh[0].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert bool((other == 7).all())
    X, R = (np.fft.fft(t.cpu().numpy().astype(np.complex128), axis=1) for t in (x, r))
    for k, v in ((few, gh[0]), (many, gh[1])):
        want = np.fft.ifft((R[:k] * X[:k].conj()).sum(axis=0)).real
        # eps * (log2 n + sqrt(signals)), as for the reduction by rows
        assert rel_l2(v.cpu().numpy(), want) <= 2.0 ** -23 * (8 + np.sqrt(k))
    gpu.free_plan_conv(plan)
