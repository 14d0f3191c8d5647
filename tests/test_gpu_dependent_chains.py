"""Dependently launched kernels beside the default 1D and 2D schedules: the
split-precision engines (tables loaded before the wait), TMA-staged, streaming
and persistent tiles, the no-allocation execute and its shared scratch, the
filter adjoint's chunks over one workspace, streaming blocks.  Chains queued
without synchronising, between producer and consumer kernels and in a captured
graph, give bit for bit what they give with a synchronisation after each step."""
from __future__ import annotations

import ctypes

import pytest

from mufft_gb300 import capi as K

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


def _noise(torch, seed, *shape, complex_=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if not complex_:
        return torch.rand(shape, device="cuda", generator=g) - 0.5
    return torch.view_as_complex(torch.rand((*shape, 2), device="cuda", generator=g) - 0.5)


def _check(torch, steps, results, capture=True):
    """`steps`: functions that return 0 or None; `results`: what they leave."""
    def clear():
        for r in results:
            r.zero_()

    def run(sync):
        for s in steps:
            assert not s()
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
    clear()
    run(True)
    want = [r.clone() for r in results]
    assert all(bool(w.abs().max() > 0) for w in want)
    for _ in range(4):
        clear()
        run(False)
        assert all(torch.equal(r, w) for r, w in zip(results, want))
    if not capture:
        return
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        codes = [s() for s in steps]
    assert not any(codes)
    for _ in range(3):
        clear()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(r, w) for r, w in zip(results, want))


def _stream(torch):
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("n, batch", [(256, 300), (4096, 700)])
@pytest.mark.parametrize("flag", [K.FLAG_SPLIT_BF16X3, K.FLAG_SPLIT_BF16X2])
@pytest.mark.parametrize("engine", [0, 1])
def test_split(gpu, torch, n, batch, flag, engine):
    o = gpu.options(split_engine=engine)
    plans = [gpu.gb_create_plan_1d(0, n, d, flag, batch, 0, 0, ctypes.byref(o)) for d in (K.FORWARD, K.INVERSE)]
    assert all(plans), gpu.gb_last_error_string()
    x = _noise(torch, n, batch, n)
    a, b = torch.empty_like(x), torch.empty_like(x)

    def ex(p, dst, src):
        return lambda: gpu.gb_execute_plan_1d_async(p, dst.data_ptr(), src.data_ptr(), _stream(torch))
    steps = [lambda: a.copy_(x) is None]
    for _ in range(3):  # producer kernel, forward, inverse, consumer kernel
        steps += [lambda: a.mul_(0.5) is None, ex(plans[0], b, a), ex(plans[1], a, b), lambda: a.mul_(2.0 / n) is None]
    _check(torch, steps, [a, b])
    for p in plans:
        gpu.free_plan_1d(p)


@pytest.mark.parametrize("n, batch, fields", [
    (1 << 22, 1, dict(tma=1)), (1 << 22, 1, dict(tma=2)), (1 << 18, 5, dict(tma=1)),
    (1024, 2000, dict(stream_tiles=1)), (256, 5000, dict(stream_tiles=1)),
    (1 << 24, 1, dict(multipass_levels=2, persistent_tiles=1)), (1 << 24, 1, dict(multipass_levels=3, fused_passes=1)),
    (1 << 20, 2, dict(twiddle_table=1)), (16384, 20, dict(tile_occupancy=1))],
    ids=lambda v: "-".join(f"{k}{w}" for k, w in v.items()) if isinstance(v, dict) else str(v))
def test_optional_tiles(gpu, torch, n, batch, fields):
    o = gpu.options(**fields)
    plans = [gpu.gb_create_plan_1d(0, n, d, 0, batch, 0, 0, ctypes.byref(o)) for d in (K.FORWARD, K.INVERSE)]
    assert all(plans), gpu.gb_last_error_string()
    x = _noise(torch, n + batch, batch, n)
    a, b = torch.empty_like(x), torch.empty_like(x)

    def ex(p, dst, src):
        return lambda: gpu.gb_execute_plan_1d_async(p, dst.data_ptr(), src.data_ptr(), _stream(torch))
    steps = [lambda: a.copy_(x) is None]
    for _ in range(2):
        steps += [ex(plans[0], b, a), ex(plans[1], a, b), lambda: a.mul_(1.0 / n) is None, ex(plans[0], b, a)]
    _check(torch, steps, [a, b])
    for p in plans:
        gpu.free_plan_1d(p)


@pytest.mark.parametrize("nx", [64, 2048])
def test_persistent_columns(gpu, torch, nx):
    ny = 4096
    o = gpu.options(columns_2d=1, persistent_tiles=1)
    plans = [gpu.gb_create_plan_2d(0, nx, ny, d, 0, ctypes.byref(o)) for d in (K.FORWARD, K.INVERSE)]
    assert all(plans), gpu.gb_last_error_string()
    x = _noise(torch, nx, ny, nx)
    a, b = torch.empty_like(x), torch.empty_like(x)

    def ex(p, dst, src):
        return lambda: gpu.gb_execute_plan_2d_async(p, dst.data_ptr(), src.data_ptr(), _stream(torch))
    steps = [lambda: a.copy_(x) is None]
    for _ in range(2):
        steps += [ex(plans[0], b, a), ex(plans[1], a, b), lambda: a.mul_(1.0 / (nx * ny)) is None]
    _check(torch, steps, [a, b])
    for p in plans:
        gpu.free_plan_2d(p)


@pytest.mark.parametrize("n", [1 << 10, 1 << 14, 1 << 15, 1 << 18])
def test_no_allocation(gpu, torch, n):
    """Consecutive calls share one scratch array."""
    x = _noise(torch, n, 3, n)
    a, b, c = (torch.empty_like(x) for _ in range(3))

    def ex(dst, src, d):
        return lambda: gpu.gb_execute_c2c_noalloc(n, d, dst.data_ptr(), src.data_ptr(), _stream(torch))
    steps = []
    for i in range(3):
        steps += [ex(a[i], x[i], K.FORWARD)]
    for i in range(3):
        steps += [ex(b[i], a[i], K.INVERSE), lambda i=i: b[i].mul_(1.0 / n) is None, ex(c[i], b[i], K.FORWARD)]
    assert gpu.gb_execute_c2c_noalloc(n, K.FORWARD, a.data_ptr(), x.data_ptr(), _stream(torch)) == 0  # set up
    _check(torch, steps, [a, b, c])


@pytest.mark.parametrize("n, batch, stereo", [(8192, 700, True), (256, 40, False), (1 << 21, 35, True), (1 << 20, 70, False)])
def test_adjoint_steps(gpu, torch, n, batch, stereo):
    """Gradient steps back to back: chunks of signals (2^21: 16 and 3 of them a
    chunk, mono 2^20: 63 and 7) over one spectrum scratch, one set of partial sums."""
    plan = gpu.create_plan_conv(n, 0, 1 if stereo else 0)
    bins = gpu.conv_get_transformed_block_size(plan) // 8
    A = _noise(torch, n, batch, bins)
    r = _noise(torch, n + 1, batch, n, complex_=stereo)
    h = _noise(torch, n + 2, n, complex_=False)
    filt = torch.empty(bins, dtype=torch.complex64, device="cuda")
    y, gx = torch.empty_like(r), torch.empty_like(r)
    gh = [torch.empty(n, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()

    def adjoint(out):
        return lambda: gpu.gb_conv_adjoint(plan, out.data_ptr(), gx.data_ptr(), n, r.data_ptr(), n, A.data_ptr(), bins,
                                           filt.data_ptr(), batch, _stream(torch))
    steps = [lambda: gpu.gb_execute_conv_input_async(plan, 1, filt.data_ptr(), h.data_ptr(), _stream(torch)),
             lambda: gpu.gb_execute_conv_output_batched(plan, y.data_ptr(), n, A.data_ptr(), bins, filt.data_ptr(), batch,
                                                        _stream(torch)),
             adjoint(gh[0]),
             # the gradient steps the filter: a producer kernel before the next step
             lambda: gpu.gb_execute_conv_input_async(plan, 1, filt.data_ptr(), gh[0].data_ptr(), _stream(torch)),
             adjoint(gh[1])]
    _check(torch, steps, [y, gx, *gh], capture=batch * n <= 1 << 23)
    gpu.free_plan_conv(plan)


@pytest.mark.parametrize("block, taps, stereo", [(64, 5000, 0), (256, 40000, 1), (1024, 100000, 1), (2048, 30000, 0)])
def test_stream_blocks(gpu, torch, block, taps, stereo):
    h = _noise(torch, taps, taps, complex_=False)
    torch.cuda.synchronize()
    conv = gpu.gb_create_stream_conv(block, stereo, h.data_ptr(), taps, 0, None)
    assert conv, gpu.gb_last_error_string()
    assert gpu.gb_stream_conv_fused(conv) == 1
    nb = 24
    floats = block * (2 if stereo else 1)
    x = _noise(torch, block, nb, floats, complex_=False)
    out = torch.empty_like(x)

    class View:
        def __init__(self, addr):
            self.__cuda_array_interface__ = {"shape": (floats,), "typestr": "<f4", "data": (addr, False), "version": 3}
    src = torch.as_tensor(View(gpu.gb_stream_conv_input(conv)), device="cuda")
    dst = torch.as_tensor(View(gpu.gb_stream_conv_output(conv)), device="cuda")
    steps = [lambda: gpu.gb_stream_conv_reset(conv, _stream(torch))]
    for k in range(nb):
        # kernels either side of the block, not only copies
        steps += [lambda k=k: torch.mul(x[k], 0.5, out=src) is None,
                  lambda: gpu.gb_stream_conv_process(conv, _stream(torch)),
                  lambda k=k: torch.mul(dst, 2.0, out=out[k]) is None]
    _check(torch, steps, [out])
    assert gpu.gb_stream_conv_status(conv) == 0
    gpu.gb_free_stream_conv(conv)
