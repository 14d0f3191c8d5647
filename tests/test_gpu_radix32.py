"""Radix-32 stages against the radix-16 ones they replace: error against FP64.

Tiles of 32 elements a thread transform 512, 1024, 8192 and 16384 points with
one stage fewer than those of 16.  On the same inputs their error may not be
larger (float emulation of both: 0.96, 0.97, 0.96 and 0.97 of it).
"""
from __future__ import annotations

import ctypes

import pytest

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


ROW, COL, ROWT = (0, 0), (1, 1), (0, 1)


def _error(lib, torch, N, batch, tiles, x, exact):
    o = lib.options(tiles=tiles)
    p = lib.gb_create_plan_1d(0, N, K.FORWARD, 0, batch, 0, 0, ctypes.byref(o))
    assert p, lib.gb_last_error_string()
    y = torch.empty_like(x)
    assert lib.gb_execute_plan_1d_async(p, y.data_ptr(), x.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    text = ctypes.create_string_buffer(4096)
    lib.gb_plan_1d_describe(p, text, 4096)
    lib.free_plan_1d(p)
    for L, la, sa, c, r, q in tiles:
        assert f"L={L} R={r} C={c} Q={q} {'across' if la else 'along'}/{'across' if sa else 'along'}" in text.value.decode()
    return float((y.to(torch.complex128) - exact).norm() / exact.norm())


@pytest.mark.parametrize("N, batch, wide, narrow", [
    (512, 4096, [(512, *ROW, 2, 32, 1)], [(512, *ROW, 8, 16, 1)]),
    (1024, 2048, [(1024, *ROW, 1, 32, 1)], [(1024, *ROW, 1, 16, 1)]),
    (8192, 256, [(8192, *ROW, 1, 32, 1)], [(8192, *ROW, 1, 16, 1)]),
    (16384, 128, [(16384, *ROW, 1, 32, 1)], [(16384, *ROW, 1, 16, 1)]),
    # four-step: column tiles with the twiddle's base in the last stage, rows stored transposed
    (1 << 18, 8, [(512, *COL, 8, 32, 1), (512, *ROWT, 8, 32, 1)], [(512, *COL, 8, 16, 1), (512, *ROWT, 8, 16, 1)]),
    (1 << 20, 2, [(1024, *COL, 8, 32, 1), (1024, *ROWT, 8, 32, 1)],
     [(1024, *COL, 8, 16, 1), (1024, *ROWT, 8, 16, 1)]),
], ids=lambda v: str(v) if isinstance(v, int) else "")
def test_error_no_larger_than_radix_16(gpu, torch, N, batch, wide, narrow):
    x = torch.from_numpy(signals.complex_uniform(83000 + batch, batch * N).reshape(batch, N)).cuda()
    exact = torch.fft.fft(x.to(torch.complex128))
    assert _error(gpu, torch, N, batch, wide, x, exact) <= _error(gpu, torch, N, batch, narrow, x, exact)


@pytest.mark.parametrize("ctas", [2887, 2888, 2889])
@pytest.mark.parametrize("direction", [K.FORWARD, K.INVERSE])
def test_rows_of_512_in_many_ctas(gpu, torch, ctas, direction):
    """Both sides of the line between the two register budgets, ragged last tile."""
    N, batch = 512, 2 * ctas - 1
    x = torch.from_numpy(signals.complex_uniform(84000 + ctas, batch * N).reshape(batch, N)).cuda()
    w = x.to(torch.complex128)
    exact = torch.fft.fft(w) if direction == K.FORWARD else torch.fft.ifft(w) * N
    p = gpu.gb_create_plan_1d(0, N, direction, 0, batch, 0, 0, None)
    y = torch.empty_like(x)
    assert gpu.gb_execute_plan_1d_async(p, y.data_ptr(), x.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    gpu.free_plan_1d(p)
    err = (y.to(torch.complex128) - exact).norm(dim=1) / exact.norm(dim=1)
    assert float(err.max()) <= 2.0 ** -23 * 9  # eps * log2(N), every row
