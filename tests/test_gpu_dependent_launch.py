"""Executes queued without synchronising -- back to back, between other
kernels and copies, and inside a captured graph -- give bit for bit what the
same executes give with a synchronisation after each: a launch never reads
what the previous one has not finished writing."""
from __future__ import annotations

import pytest

from mufft_gb300 import capi as K

pytestmark = pytest.mark.gpu

# (n, batch) of 1D plans -- one tile, tiles of many CTAs, four-step, three-level -- and 2D sides
SHAPES_1D = [(64, 5), (1024, 300), (16384, 40), (1 << 15, 3), (1 << 18, 7), (1 << 22, 1)]


@pytest.fixture(scope="module")
def gpu():
    import mufft_gb300
    return mufft_gb300.load()


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available()
    return t


def _steps(gpu, torch, n, batch):
    """A chain of executes, each on the previous one's output, with a scaling
    kernel and a copy in it; returns (steps, result)."""
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    x = torch.view_as_complex(torch.rand((batch, n, 2), device="cuda", generator=g) - 0.5)
    a, b = torch.empty_like(x), torch.empty_like(x)
    r = torch.empty((batch, n // 2 + 1), dtype=torch.complex64, device="cuda")
    out = torch.empty((batch, n), device="cuda")
    plans = [gpu.gb_create_plan_1d(0, n, K.FORWARD, 0, batch, 0, 0, None),
             gpu.gb_create_plan_1d(0, n, K.INVERSE, 0, batch, 0, 0, None),
             gpu.gb_create_plan_1d(1, n, 0, 0, batch, 0, 0, None),
             gpu.gb_create_plan_1d(2, n, 0, 0, batch, 0, 0, None)]
    assert all(plans), gpu.gb_last_error_string()

    def ex(p, dst, src):
        return lambda: gpu.gb_execute_plan_1d_async(p, dst.data_ptr(), src.data_ptr(),
                                                    torch.cuda.current_stream().cuda_stream)
    steps = [lambda: a.copy_(x) is None]
    for _ in range(3):
        steps += [ex(plans[0], b, a), ex(plans[1], a, b), lambda: a.mul_(1.0 / n) is None]
    steps += [lambda: out.copy_(a.real) is None, ex(plans[2], r, out), ex(plans[3], out, r), ex(plans[2], r, out),
              ex(plans[3], out, r)]
    return steps, out, plans


@pytest.mark.parametrize("n,batch", SHAPES_1D)
def test_chains(gpu, torch, n, batch):
    steps, out, plans = _steps(gpu, torch, n, batch)
    for s in steps:
        assert not s()
        torch.cuda.synchronize()
    want = out.clone()
    for _ in range(3):
        out.zero_()
        for s in steps:
            assert not s()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for s in steps:
            s()
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    for p in plans:
        gpu.free_plan_1d(p)


@pytest.mark.parametrize("nx,ny", [(32, 16), (512, 1024), (4096, 256), (256, 4096), (4096, 4096)])
def test_2d_there_and_back(gpu, torch, nx, ny):
    g = torch.Generator(device="cuda").manual_seed(nx * ny)
    x = torch.rand((ny, nx), device="cuda", generator=g) - 0.5
    spec = torch.zeros((ny, nx), dtype=torch.complex64, device="cuda")
    back = torch.empty(2 * ny * nx, device="cuda")
    plans = [gpu.create_plan_2d_r2c(nx, ny, 0), gpu.create_plan_2d_c2r(nx, ny, 0)]
    assert all(plans)

    def there(sync):
        st = torch.cuda.current_stream().cuda_stream
        for _ in range(2):
            assert gpu.gb_execute_plan_2d_async(plans[0], spec.data_ptr(), x.data_ptr(), st) == 0
            if sync:
                torch.cuda.synchronize()
            assert gpu.gb_execute_plan_2d_async(plans[1], back.data_ptr(), spec.data_ptr(), st) == 0
            if sync:
                torch.cuda.synchronize()
    there(True)
    want = back[: nx * ny].clone()
    for _ in range(5):
        back.zero_()
        there(False)
        torch.cuda.synchronize()
        assert torch.equal(back[: nx * ny], want)
    for p in plans:
        gpu.free_plan_2d(p)
