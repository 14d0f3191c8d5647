"""Blocking executes on host buffers of which only a part is page-locked: no
kernel may take them directly.  The copies that stage them either work -- then
the result is that of the device buffers, bit for bit -- or report an error."""
from __future__ import annotations

import mmap

import numpy as np
import pytest

from mufft_gb300 import capi as K
from mufft_gb300 import signals

pytestmark = pytest.mark.gpu

PAGE = 1 << 16
SIZE = 4 * PAGE  # 16 transforms of 2048 points


class Buffer:
    """SIZE bytes of mapped memory; `pinned`: the page ranges registered with CUDA."""

    def __init__(self, torch, pinned):
        self.rt = torch.cuda.cudart()
        self.map = mmap.mmap(-1, SIZE + PAGE)
        raw = np.frombuffer(self.map, np.uint8)
        self.bytes = raw[(-raw.ctypes.data) % PAGE:][:SIZE]
        self.bytes[...] = 0
        self.done = []
        for first, last in pinned:
            at = self.bytes.ctypes.data + first * PAGE
            assert int(self.rt.cudaHostRegister(at, (last - first) * PAGE, 0)) == 0
            self.done.append(at)

    def close(self):
        for at in self.done:
            assert int(self.rt.cudaHostUnregister(at)) == 0


WHOLE = [(0, 4)]
PARTS = {"whole": WHOLE, "front": [(0, 1)], "back": [(3, 4)], "halves": [(0, 2), (2, 4)], "ends": [(0, 1), (3, 4)],
         "none": []}


@pytest.mark.parametrize("part", sorted(PARTS))
@pytest.mark.parametrize("which", ["in", "out"])
def test_partly_page_locked(part, which):
    import torch

    import mufft_gb300
    gpu = mufft_gb300.load()
    n, batch = 2048, SIZE // (8 * 2048)
    x = signals.complex_uniform(84000, n * batch)
    dx = torch.from_numpy(x).cuda()
    dy = torch.empty_like(dx)
    plan = gpu.gb_create_plan_1d(0, n, K.FORWARD, 0, batch, 0, 0, None)
    assert plan
    assert gpu.gb_execute_plan_1d_async(plan, dy.data_ptr(), dx.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    want = dy.cpu().numpy()
    src = Buffer(torch, PARTS[part] if which == "in" else WHOLE)
    dst = Buffer(torch, PARTS[part] if which == "out" else WHOLE)
    src.bytes[...] = x.view(np.uint8)
    gpu.gb_clear_error()
    gpu.execute_plan_1d(plan, dst.bytes.ctypes.data, src.bytes.ctypes.data)
    failed = gpu.gb_last_error()
    gpu.gb_clear_error()
    if part in ("whole", "none"):
        assert failed == 0
    if failed == 0:
        assert np.array_equal(dst.bytes.view(np.uint64), want.view(np.uint64))
    torch.cuda.synchronize()  # the context stays usable
    gpu.free_plan_1d(plan)
    src.close()
    dst.close()


@pytest.mark.parametrize("kind, n, limit", [(0, 16, 1 << 18), (0, 32, 1 << 19), (1, 16, 1 << 18), (2, 32, 1 << 18),
                                            (2, 64, 1 << 19), (0, 64, 1 << 20)])
def test_limits_of_direct_access(kind, n, limit):
    """The last batch the kernel takes itself and the first one that is staged: the same bits."""
    import torch

    import mufft_gb300
    gpu = mufft_gb300.load()
    fin, fout = (2 * n, n, n + 2)[kind], (2 * n, n + 2, n)[kind]  # floats per transform
    most = limit // (4 * max(fin, fout))
    for batch in (most, most + 1):
        x = signals.uniform(85000 + n, fin * batch).astype(np.float32)
        dx = torch.from_numpy(x).cuda()
        dy = torch.empty(fout * batch, device="cuda")
        plan = gpu.gb_create_plan_1d(kind, n, K.FORWARD, 0, batch, 0, 0, None)
        assert plan
        assert gpu.gb_execute_plan_1d_async(plan, dy.data_ptr(), dx.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        want = dy.cpu().numpy()
        src, dst = gpu.alloc(x.nbytes), gpu.alloc(want.nbytes)
        assert gpu.gb_memcpy(src, dx.data_ptr(), x.nbytes) == 0
        gpu.execute_plan_1d(plan, dst, src)
        gpu.check("execute_plan_1d")
        got = torch.empty(fout * batch, device="cuda")
        assert gpu.gb_memcpy(got.data_ptr(), dst, want.nbytes) == 0
        assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
        gpu.free_plan_1d(plan)
        gpu.free(src)
        gpu.free(dst)
