"""Performance cases of the framework: what its users run, through its public entry points.

A case is a dict of plain values.  `listed()` are the fixed ones, `draw(rng)`
one more of the same ranges, `prepare(case, seed)` the inputs and the plan or
handle a program keeps, `run(state)` one pass and its outputs, `work(case)` the
bytes and operations the pass cannot do without, `exact(case, seed)` its
outputs in 64-bit arithmetic by torch.

Families ("kind"):
  fft1d        batched 1D transforms on device buffers (c2c, r2c, c2r)
  fft2d        one 2D transform on device buffers (c2c, r2c, c2r)
  image        2D r2c followed by 2D c2r: the two halves of an image filter
  host_conv    fft.h as a muFFT program calls it: block convolution on mufft_alloc memory
  conv_batch   ragged convolution requests as one batch
  fft_batch    ragged transform requests as one batch
  adjoint      the library calls of one filter-fitting gradient step
  stream       a stream of blocks through a long filter
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import mufft_gb300
from mufft_gb300 import capi as K

DEV = "cuda"


# ------------------------------------------------------------------ cases

def listed() -> list[dict]:
    return [
        # a real-time effect built on muFFT: 1024-frame stereo blocks through a
        # 1024-tap filter, host memory in and out, latency counts
        dict(name="host_block_conv_2048", kind="host_conv", n=2048, stereo=True, pad=True),
        # spectra of many short frames (spectrogram, channeliser)
        dict(name="c2c_1024_x4096", kind="fft1d", form="c2c", n=1024, batch=4096, inverse=False, pad=False,
             full=False, split=0),
        # one very long transform (chirp or correlation over a whole recording)
        dict(name="c2c_2e24", kind="fft1d", form="c2c", n=1 << 24, batch=1, inverse=False, pad=False, full=False,
             split=0),
        # long real signals, an odd number of them: audio files into spectra
        dict(name="r2c_2e18_x61", kind="fft1d", form="r2c", n=1 << 18, batch=61, inverse=False, pad=False,
             full=False, split=0),
        # spectra back to real frames of 16384 samples (overlap-add synthesis)
        dict(name="c2r_16384_x3001", kind="fft1d", form="c2r", n=16384, batch=3001, inverse=True, pad=False,
             full=False, split=0),
        # the same short-frame work at tensor-core split precision
        dict(name="split_4096_x16384", kind="fft1d", form="c2c", n=4096, batch=16384, inverse=False, pad=False,
             full=False, split=3),
        # filtering one large image: to its spectrum and back
        dict(name="image_4096_r2c_c2r", kind="image", nx=4096, ny=4096),
        # a small complex field back to space (phase retrieval, optics)
        dict(name="c2c_2d_1024x512_inverse", kind="fft2d", form="c2c", nx=1024, ny=512, inverse=True, full=False),
        # a server's queue of convolution requests of mixed sizes
        dict(name="conv_requests_512", kind="conv_batch", count=512, mix=4, lo=8, hi=16),
        # a server's queue of transform requests of mixed kinds and sizes
        dict(name="fft_requests_512", kind="fft_batch", count=512, mix=6, lo=4, hi=16),
        # fitting a 2^16-tap filter to 64 stereo signals of 2^20 frames
        dict(name="adjoint_step_64x2e20", kind="adjoint", n=1 << 21, batch=64, taps=1 << 16, stereo=True),
        # convolution reverb: 1024-frame stereo blocks through 2^20 taps
        dict(name="stream_2e20_taps", kind="stream", block=1024, taps=1 << 20, stereo=True, blocks=32),
    ]


def _pow2(rng: random.Random, lo: int, hi: int) -> int:
    return 1 << rng.randint(lo, hi)


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    """An integer in lo..hi, spread over its logarithm (odd ones among them)."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["fft1d"] * 6 + ["split"] * 2 + ["fft2d"] * 3 + ["image", "host_conv", "host_conv", "conv_batch",
                                                                      "fft_batch", "adjoint", "adjoint", "stream"])
    if kind == "fft1d":
        form = rng.choice(["c2c", "c2c", "r2c", "c2r"])
        lg = rng.randint(1, 24) if form == "c2c" else rng.randint(2, 23)
        batch = _log_int(rng, 1, max(1, min(65535, (1 << 26) >> lg)))
        return dict(kind="fft1d", form=form, n=1 << lg, batch=batch,
                    inverse=form == "c2r" or (form == "c2c" and rng.random() < 0.5),
                    pad=form != "c2r" and rng.random() < 0.25, full=form == "r2c" and rng.random() < 0.25, split=0)
    if kind == "split":
        n = rng.choice([256, 4096])
        return dict(kind="fft1d", form="c2c", n=n, batch=_log_int(rng, 1, (1 << 26) // n), inverse=rng.random() < 0.5,
                    pad=False, full=False, split=rng.choice([3, 3, 2]))
    if kind == "fft2d":
        form = rng.choice(["c2c", "r2c", "c2r"])
        lx = rng.randint(2, 13)
        ly = rng.randint(1, min(13, 25 - lx))
        return dict(kind="fft2d", form=form, nx=1 << lx, ny=1 << ly,
                    inverse=form == "c2r" or (form == "c2c" and rng.random() < 0.5),
                    full=form == "r2c" and rng.random() < 0.25)
    if kind == "image":
        lx = rng.randint(6, 13)
        return dict(kind="image", nx=1 << lx, ny=_pow2(rng, 6, min(13, 25 - lx)))
    if kind == "host_conv":
        return dict(kind="host_conv", n=_pow2(rng, 6, 18), stereo=rng.random() < 0.5, pad=rng.random() < 0.75)
    if kind == "conv_batch":
        lo = rng.randint(6, 12)
        return dict(kind="conv_batch", count=_log_int(rng, 16, 600), mix=rng.randrange(1 << 20), lo=lo,
                    hi=rng.randint(lo, 16))
    if kind == "fft_batch":
        lo = rng.randint(3, 12)
        return dict(kind="fft_batch", count=_log_int(rng, 16, 900), mix=rng.randrange(1 << 20), lo=lo,
                    hi=rng.randint(lo, 16))
    if kind == "adjoint":
        lg = rng.randint(10, 21)
        n = 1 << lg
        return dict(kind="adjoint", n=n, batch=_log_int(rng, 1, min(2000, (1 << 26) // n)),
                    taps=_log_int(rng, 16, n // 2), stereo=rng.random() < 0.5)
    block = _pow2(rng, 6, 12)
    return dict(kind="stream", block=block, taps=_log_int(rng, block, 1 << 20), stereo=rng.random() < 0.5, blocks=32)


# ---------------------------------------------------------------- helpers

class Handle:
    """A library handle that is given back when the state goes."""

    def __init__(self, lib, p, free):
        if not p:
            raise RuntimeError(lib.gb_last_error_string().decode())
        self.p, self._free = p, free

    def __del__(self):
        self._free(self.p)


class PinnedArray:
    """Page-locked host memory from mufft_alloc as a numpy array's owner."""

    def __init__(self, lib, count: int, dtype):
        dt = np.dtype(dtype)
        self._lib, self.addr = lib, lib.alloc(max(1, count) * dt.itemsize)
        if not self.addr:
            raise MemoryError("mufft_alloc")
        self.__array_interface__ = {"shape": (count,), "typestr": dt.str, "data": (self.addr, False), "version": 3}

    def __del__(self):
        self._lib.free(self.addr)


class DeviceView:
    """Device memory owned by a handle, for torch (zero copy)."""

    def __init__(self, owner, addr: int, shape: tuple, dtype):
        self._owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": np.dtype(dtype).str, "data": (addr, False),
                                         "version": 3}


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(shape, complex_: bool, g) -> torch.Tensor:
    """Uniform [-1, 1) samples, float32 or complex64."""
    if not complex_:
        return torch.rand(shape, device=DEV, generator=g) * 2 - 1
    return torch.view_as_complex(torch.rand((*shape, 2), device=DEV, generator=g) * 2 - 1)


def _half_spectrum(shape, g) -> torch.Tensor:
    """N/2 + 1 bins of real signals: the first and the last bin are real."""
    x = _uniform(shape, True, g)
    x[..., 0].imag.zero_()
    x[..., -1].imag.zero_()
    return x


def _half_spectrum_2d(ny: int, nx: int, g) -> torch.Tensor:
    """Spectrum of a real ny x nx image in rows of nx complex, nx/2 + 1 of them used."""
    x = torch.zeros((ny, nx), dtype=torch.complex64, device=DEV)
    m = nx // 2
    x[:, : m + 1] = _uniform((ny, m + 1), True, g)
    for c in (0, m):  # these columns are conjugate-symmetric in y
        col = x[:, c].clone()
        x[:, c] = 0.5 * (col + col.flip(0).roll(1).conj())
    return x


def _decaying(n: int, tau: float, g) -> torch.Tensor:
    """Filter taps: Gaussian noise under an exponential decay."""
    t = torch.arange(n, device=DEV, dtype=torch.float32)
    return torch.randn(n, device=DEV, generator=g) * torch.exp(-t / tau)


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _ok(rc: int) -> None:
    if rc:
        raise RuntimeError(mufft_gb300.load().gb_last_error_string().decode())


def _log2(n: int) -> int:
    return n.bit_length() - 1


# ----------------------------------------------------------------- inputs
#
# Each family's inputs, the same for prepare() and exact().

def _in_fft1d(c, g):
    n, b = c["n"], c["batch"]
    if c["form"] == "c2r":
        return _half_spectrum((b, n // 2 + 1), g)
    return _uniform((b, n // 2 if c["pad"] else n), c["form"] == "c2c", g)


def _in_fft2d(c, g):
    if c["form"] == "c2r":
        return _half_spectrum_2d(c["ny"], c["nx"], g)
    return _uniform((c["ny"], c["nx"]), c["form"] == "c2c", g)


def _in_image(c, g):
    return torch.randn((c["ny"], c["nx"]), device=DEV, generator=g)


def _in_host_conv(c, g):
    n = c["n"]
    m = n // 2 if c["pad"] else n
    return _uniform((m,), c["stereo"], g), _decaying(m, n / 8, g)


def _requests(c) -> list[dict]:
    """The sizes, kinds and buffer places of a batch's requests (offsets in floats, 256-byte aligned)."""
    rng = random.Random(c["mix"])
    reqs, at_in, at_out = [], 0, 0
    for i in range(c["count"]):
        n = 1 << rng.randint(c["lo"], c["hi"])
        if c["kind"] == "conv_batch":
            r = dict(n=n, stereo=i % 2 == 0, fin=n if i % 2 == 0 else n // 2, fout=2 * n if i % 2 == 0 else n)
        else:
            t = rng.randrange(4)  # c2c forward, c2c inverse, r2c, c2r
            pad = t < 3 and rng.random() < 0.25
            full = t == 2 and rng.random() < 0.5
            half = n // 2 if pad else n
            r = dict(n=n, form=t, pad=pad, full=full, fin=(2 * half, 2 * half, half, n + 2)[t],
                     fout=(2 * n, 2 * n, 2 * n if full else n + 2, n)[t])
        r["at_in"], r["at_out"] = at_in, at_out
        at_in += -(-r["fin"] // 64) * 64
        at_out += -(-r["fout"] // 64) * 64
        reqs.append(r)
    return reqs


def _in_batch(c, reqs, g):
    """All requests' inputs in one float buffer; convolutions: their filters too."""
    last = reqs[-1]
    x = torch.rand(last["at_in"] + last["fin"], device=DEV, generator=g) * 2 - 1
    if c["kind"] == "fft_batch":
        for r in reqs:
            if r["form"] == 3:  # half spectra: the first and the last bin are real
                x[r["at_in"] + 1] = 0
                x[r["at_in"] + r["n"] + 1] = 0
        return x, None
    taps = [_decaying(r["n"] // 2, r["n"] / 8, g) for r in reqs]
    return x, taps


def _in_adjoint(c, g):
    n, b = c["n"], c["batch"]
    return _uniform((b, n // 2), c["stereo"], g), _uniform((b, n), c["stereo"], g), _decaying(c["taps"], c["taps"] / 8, g)


def _in_stream(c, g):
    return (_uniform((c["blocks"], c["block"]), c["stereo"], g), _decaying(c["taps"], max(1.0, c["taps"] / 8), g))


# ---------------------------------------------------------------- prepare

def _prep_fft1d(c, g, lib):
    n, b = c["n"], c["batch"]
    x = _in_fft1d(c, g)
    flags = (K.FLAG_ZERO_PAD_UPPER_HALF if c["pad"] else 0) | (K.FLAG_FULL_R2C if c["full"] else 0)
    flags |= {0: 0, 2: K.FLAG_SPLIT_BF16X2, 3: K.FLAG_SPLIT_BF16X3}[c["split"]]
    if c["form"] == "c2c":
        p = lib.gb_create_plan_1d_c2c_batched(n, K.INVERSE if c["inverse"] else K.FORWARD, flags, b, 0, 0)
        out = torch.empty((b, n), dtype=torch.complex64, device=DEV)
    elif c["form"] == "r2c":
        p = lib.gb_create_plan_1d_r2c_batched(n, flags, b, 0, 0)
        out = torch.empty((b, n if c["full"] else n // 2 + 1), dtype=torch.complex64, device=DEV)
    else:
        p = lib.gb_create_plan_1d_c2r_batched(n, flags, b, 0, 0)
        out = torch.empty((b, n), dtype=torch.float32, device=DEV)
    plan = Handle(lib, p, lib.free_plan_1d)

    def run():
        _ok(lib.gb_execute_plan_1d_async(plan.p, out.data_ptr(), x.data_ptr(), _stream()))
        return out
    return run


def _prep_fft2d(c, g, lib):
    nx, ny = c["nx"], c["ny"]
    x = _in_fft2d(c, g)
    if c["form"] == "c2c":
        p = lib.create_plan_2d_c2c(nx, ny, K.INVERSE if c["inverse"] else K.FORWARD, 0)
        out = torch.empty((ny, nx), dtype=torch.complex64, device=DEV)
        seen = out
    elif c["form"] == "r2c":
        p = lib.create_plan_2d_r2c(nx, ny, K.FLAG_FULL_R2C if c["full"] else 0)
        out = torch.empty((ny, nx), dtype=torch.complex64, device=DEV)
        seen = out if c["full"] else out[:, : nx // 2 + 1]  # the columns a 2D r2c defines
    else:
        p = lib.create_plan_2d_c2r(nx, ny, 0)
        out = torch.empty(2 * ny * nx, dtype=torch.float32, device=DEV)  # the API's buffer size
        seen = out[: ny * nx].view(ny, nx)  # what it defines
    plan = Handle(lib, p, lib.free_plan_2d)

    def run():
        _ok(lib.gb_execute_plan_2d_async(plan.p, out.data_ptr(), x.data_ptr(), _stream()))
        return seen
    return run


def _prep_image(c, g, lib):
    nx, ny = c["nx"], c["ny"]
    x = _in_image(c, g)
    fwd = Handle(lib, lib.create_plan_2d_r2c(nx, ny, 0), lib.free_plan_2d)
    inv = Handle(lib, lib.create_plan_2d_c2r(nx, ny, 0), lib.free_plan_2d)
    spec = torch.empty((ny, nx), dtype=torch.complex64, device=DEV)
    back = torch.empty(2 * ny * nx, dtype=torch.float32, device=DEV)
    seen = (spec[:, : nx // 2 + 1], back[: ny * nx].view(ny, nx))

    def run():
        st = _stream()
        _ok(lib.gb_execute_plan_2d_async(fwd.p, spec.data_ptr(), x.data_ptr(), st))
        _ok(lib.gb_execute_plan_2d_async(inv.p, back.data_ptr(), spec.data_ptr(), st))
        return seen
    return run


_PADS = K.CONV_METHOD_FLAG_ZERO_PAD_UPPER_HALF_FIRST | K.CONV_METHOD_FLAG_ZERO_PAD_UPPER_HALF_SECOND


def _prep_host_conv(c, g, lib):
    n, stereo = c["n"], c["stereo"]
    x, h = _in_host_conv(c, g)
    plan = Handle(lib, lib.create_plan_conv(n, 0, (_PADS if c["pad"] else 0) | (1 if stereo else 0)),
                  lib.free_plan_conv)
    nblk = lib.conv_get_transformed_block_size(plan.p) // 8
    sample = np.complex64 if stereo else np.float32
    px, ph = PinnedArray(lib, x.numel(), sample), PinnedArray(lib, h.numel(), np.float32)
    pa, pb = PinnedArray(lib, nblk, np.complex64), PinnedArray(lib, nblk, np.complex64)
    po = PinnedArray(lib, n, sample)
    np.asarray(px)[...] = x.cpu().numpy()
    np.asarray(ph)[...] = h.cpu().numpy()
    lib.execute_conv_input(plan.p, K.CONV_BLOCK_SECOND, pb.addr, ph.addr)
    seen = np.asarray(po)

    def run():
        lib.execute_conv_input(plan.p, K.CONV_BLOCK_FIRST, pa.addr, px.addr)
        lib.execute_conv_output(plan.p, po.addr, pa.addr, pb.addr)
        return seen
    return run


def _prep_conv_batch(c, g, lib):
    reqs = _requests(c)
    x, taps = _in_batch(c, reqs, g)
    out = torch.zeros(reqs[-1]["at_out"] + reqs[-1]["fout"], device=DEV)
    plans, spectra = {}, []
    creq = (K.ConvRequest * len(reqs))()
    for i, (r, h) in enumerate(zip(reqs, taps)):
        n, m = r["n"], _PADS | (1 if r["stereo"] else 0)
        if (n, m) not in plans:
            plans[n, m] = Handle(lib, lib.create_plan_conv(n, 0, m), lib.free_plan_conv)
        p = plans[n, m].p
        spec = torch.empty(lib.conv_get_transformed_block_size(p) // 8, dtype=torch.complex64, device=DEV)
        _ok(lib.gb_execute_conv_input_async(p, K.CONV_BLOCK_SECOND, spec.data_ptr(), h.data_ptr(), _stream()))
        spectra.append(spec)
        creq[i] = K.ConvRequest(n, m, x.data_ptr() + 4 * r["at_in"], spec.data_ptr(), out.data_ptr() + 4 * r["at_out"])
    batch = Handle(lib, lib.gb_create_conv_batch(creq, len(reqs), 0, None), lib.gb_free_conv_batch)
    torch.cuda.synchronize()  # the plans below go when this returns
    keep = (x, spectra)

    def run():
        _ok(lib.gb_execute_conv_batch(batch.p, _stream()))
        return out
    run.keep = keep
    return run


def _prep_fft_batch(c, g, lib):
    reqs = _requests(c)
    x, _ = _in_batch(c, reqs, g)
    out = torch.zeros(reqs[-1]["at_out"] + reqs[-1]["fout"], device=DEV)
    creq = (K.FftRequest * len(reqs))()
    for i, r in enumerate(reqs):
        flags = (K.FLAG_ZERO_PAD_UPPER_HALF if r["pad"] else 0) | (K.FLAG_FULL_R2C if r["full"] else 0)
        creq[i] = K.FftRequest(r["n"], (0, 0, 1, 2)[r["form"]],
                               (K.FORWARD, K.INVERSE, K.FORWARD, K.INVERSE)[r["form"]], flags,
                               x.data_ptr() + 4 * r["at_in"], out.data_ptr() + 4 * r["at_out"])
    batch = Handle(lib, lib.gb_create_fft_batch(creq, len(reqs), 0, None), lib.gb_free_fft_batch)

    def run():
        _ok(lib.gb_execute_fft_batch(batch.p, _stream()))
        return out
    run.keep = x
    return run


def _prep_adjoint(c, g, lib):
    n, b, stereo = c["n"], c["batch"], c["stereo"]
    x, r, taps = _in_adjoint(c, g)
    h = torch.zeros(n // 2, device=DEV)
    h[: taps.numel()] = taps
    plan = Handle(lib, lib.create_plan_conv(n, 0, _PADS | (1 if stereo else 0)), lib.free_plan_conv)
    nblk = lib.conv_get_transformed_block_size(plan.p) // 8
    spec = torch.empty((b, nblk), dtype=torch.complex64, device=DEV)  # the signals' spectra, kept across steps
    for i in range(b):
        _ok(lib.gb_execute_conv_input_async(plan.p, K.CONV_BLOCK_FIRST, spec[i].data_ptr(), x[i].data_ptr(), _stream()))
    filt = torch.empty(nblk, dtype=torch.complex64, device=DEV)
    dt = torch.complex64 if stereo else torch.float32
    y, gx = torch.empty((b, n), dtype=dt, device=DEV), torch.empty((b, n), dtype=dt, device=DEV)
    gh = torch.empty(n, device=DEV)
    torch.cuda.synchronize()

    # the residual between the two halves is the program's own work: here `r`
    # stands for it
    def run():
        st = _stream()
        _ok(lib.gb_execute_conv_input_async(plan.p, K.CONV_BLOCK_SECOND, filt.data_ptr(), h.data_ptr(), st))
        _ok(lib.gb_execute_conv_output_batched(plan.p, y.data_ptr(), n, spec.data_ptr(), nblk, filt.data_ptr(), b, st))
        _ok(lib.gb_conv_adjoint(plan.p, gh.data_ptr(), gx.data_ptr(), n, r.data_ptr(), n, spec.data_ptr(), nblk,
                                filt.data_ptr(), b, st))
        return y, gh, gx
    return run


def _prep_stream(c, g, lib):
    x, taps = _in_stream(c, g)
    torch.cuda.synchronize()
    conv = Handle(lib, lib.gb_create_stream_conv(c["block"], 1 if c["stereo"] else 0, taps.data_ptr(), c["taps"], 0, None),
                  lib.gb_free_stream_conv)
    dt = np.complex64 if c["stereo"] else np.float32
    shape = (c["block"],)
    src = torch.as_tensor(DeviceView(conv, lib.gb_stream_conv_input(conv.p), shape, dt), device=DEV)
    dst = torch.as_tensor(DeviceView(conv, lib.gb_stream_conv_output(conv.p), shape, dt), device=DEV)
    out = torch.empty_like(x)

    # a piece of a stream from its start, blocks in and blocks out, captured
    # once and replayed: the blocks of a renderer that runs ahead of real time
    def session():
        st = _stream()
        _ok(lib.gb_stream_conv_reset(conv.p, st))
        for k in range(x.shape[0]):
            src.copy_(x[k])
            _ok(lib.gb_stream_conv_process(conv.p, st))
            out[k].copy_(dst)

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        session()  # everything is loaded before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        session()

    def run():
        graph.replay()
        return out
    run.keep = (conv, src, dst, x)
    return run


_PREPARE = dict(fft1d=_prep_fft1d, fft2d=_prep_fft2d, image=_prep_image, host_conv=_prep_host_conv,
                conv_batch=_prep_conv_batch, fft_batch=_prep_fft_batch, adjoint=_prep_adjoint, stream=_prep_stream)


def prepare(case: dict, seed: int):
    return _PREPARE[case["kind"]](case, _gen(seed), mufft_gb300.load())


def run(state):
    return state()


# ------------------------------------------------------------------- work

def _fft_flops(n: int, real: bool) -> float:
    return (2.5 if real else 5.0) * n * max(1, _log2(n))


def work(case: dict) -> dict:
    c, k = case, case["kind"]
    if k == "fft1d":
        n, half = c["n"], c["n"] // 2 if c["pad"] else c["n"]
        spec = 8 * (n if c["full"] else n // 2 + 1)
        nb = {"c2c": 8 * half + 8 * n, "r2c": 4 * half + spec, "c2r": 8 * (n // 2 + 1) + 4 * n}[c["form"]]
        return dict(bytes=c["batch"] * nb, flops=c["batch"] * _fft_flops(n, c["form"] != "c2c"))
    if k in ("fft2d", "image"):
        nx, ny = c["nx"], c["ny"]
        spec = 8 * ny * (nx // 2 + 1)
        if k == "image":
            return dict(bytes=2 * (4 * nx * ny + spec), flops=2 * _fft_flops(nx * ny, True))
        nb = {"c2c": 16 * nx * ny, "r2c": 4 * nx * ny + (8 * nx * ny if c["full"] else spec),
              "c2r": spec + 4 * nx * ny}[c["form"]]
        return dict(bytes=nb, flops=_fft_flops(nx * ny, c["form"] != "c2c"))
    if k == "host_conv":
        n, s = c["n"], c["stereo"]
        half = n // 2 if c["pad"] else n
        nb = half * (8 if s else 4) + 8 * (n if s else n // 2 + 1) + n * (8 if s else 4)
        return dict(bytes=nb, flops=2 * _fft_flops(n, not s))
    if k in ("conv_batch", "fft_batch"):
        nb, fl = 0.0, 0.0
        for r in _requests(c):
            nb += 4 * (r["fin"] + r["fout"])
            if k == "conv_batch":
                nb += 8 * (r["n"] if r["stereo"] else r["n"] // 2 + 1)
                fl += 2 * _fft_flops(r["n"], not r["stereo"])
            else:
                fl += _fft_flops(r["n"], r["form"] >= 2)
        return dict(bytes=nb, flops=fl)
    if k == "adjoint":
        n, b, s = c["n"], c["batch"], c["stereo"]
        sig, spec = n * (8 if s else 4), 8 * (n if s else n // 2 + 1)
        # spectra and residuals in, outputs and input gradients out, the filter and its gradient
        return dict(bytes=b * (spec + 3 * sig) + 2 * n + 4 * n, flops=b * 3 * _fft_flops(n, not s))
    # stream: every filter spectrum and every kept window spectrum once a block
    nblk, parts = c["blocks"], -(-c["taps"] // c["block"])
    bins = 2 * c["block"] if c["stereo"] else c["block"] + 1
    return dict(bytes=nblk * (2 * parts * bins * 8 + 2 * c["block"] * (8 if c["stereo"] else 4)),
                flops=nblk * (8.0 * parts * bins + 2 * _fft_flops(2 * c["block"], not c["stereo"])))


# ------------------------------------------------------------------ exact

def _wide(x: torch.Tensor) -> torch.Tensor:
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _exact_fft1d(c, g):
    n = c["n"]
    x = _in_fft1d(c, g)
    if c["form"] == "c2r":
        return torch.fft.irfft(_wide(x), n=n) * n
    if c["form"] == "r2c" and not c["full"]:
        return torch.fft.rfft(_wide(x), n=n)
    return torch.fft.ifft(_wide(x), n=n) * n if c["inverse"] else torch.fft.fft(_wide(x), n=n)


def _exact_fft2d(c, g):
    nx, ny = c["nx"], c["ny"]
    x = _in_fft2d(c, g)
    if c["form"] == "c2r":
        return torch.fft.irfft2(_wide(x[:, : nx // 2 + 1]), s=(ny, nx)) * (nx * ny)
    if c["form"] == "r2c" and not c["full"]:
        return torch.fft.rfft2(_wide(x))
    return torch.fft.ifft2(_wide(x)) * (nx * ny) if c["inverse"] else torch.fft.fft2(_wide(x))


def _exact_image(c, g):
    x = _wide(_in_image(c, g))
    return torch.fft.rfft2(x), x * (c["nx"] * c["ny"])


def _convolve(x: torch.Tensor, h: torch.Tensor, n: int) -> torch.Tensor:
    """Circular convolution of length n in 64 bits; h is real."""
    if x.is_complex():
        return torch.fft.ifft(torch.fft.fft(_wide(x), n=n) * torch.fft.fft(_wide(h), n=n))
    return torch.fft.irfft(torch.fft.rfft(_wide(x), n=n) * torch.fft.rfft(_wide(h), n=n), n=n)


def _exact_host_conv(c, g):
    x, h = _in_host_conv(c, g)
    return _convolve(x, h, c["n"]).cpu().numpy()


def _exact_batch(c, g):
    reqs = _requests(c)
    x, taps = _in_batch(c, reqs, g)
    out = torch.zeros(reqs[-1]["at_out"] + reqs[-1]["fout"], dtype=torch.float64, device=DEV)
    for i, r in enumerate(reqs):
        n = r["n"]
        v = x[r["at_in"]: r["at_in"] + r["fin"]]
        if c["kind"] == "conv_batch":
            y = _convolve(torch.view_as_complex(v.view(-1, 2)) if r["stereo"] else v, taps[i], n)
        elif r["form"] == 3:
            y = torch.fft.irfft(_wide(torch.view_as_complex(v.view(-1, 2))), n=n) * n
        elif r["form"] == 2:
            y = torch.fft.fft(_wide(v), n=n)[: r["fout"] // 2]
        else:
            v = _wide(torch.view_as_complex(v.view(-1, 2)))
            y = torch.fft.fft(v, n=n) if r["form"] == 0 else torch.fft.ifft(v, n=n) * n
        y = torch.view_as_real(y).reshape(-1) if y.is_complex() else y
        out[r["at_out"]: r["at_out"] + r["fout"]] = y
    return out


def _exact_adjoint(c, g):
    n = c["n"]
    x, r, h = _in_adjoint(c, g)
    hf = torch.fft.fft(_wide(h), n=n)
    ys, gxs, acc = [], [], torch.zeros(n, dtype=torch.complex128, device=DEV)
    step = max(1, (1 << 24) // n)
    for b0 in range(0, c["batch"], step):
        xf = torch.fft.fft(_wide(x[b0: b0 + step]), n=n)
        rf = torch.fft.fft(_wide(r[b0: b0 + step]))
        y, gx = torch.fft.ifft(xf * hf), torch.fft.ifft(rf * hf.conj())
        ys.append(y if c["stereo"] else y.real)
        gxs.append(gx if c["stereo"] else gx.real)
        acc += (rf * xf.conj()).sum(dim=0)
    return torch.cat(ys), torch.fft.ifft(acc).real, torch.cat(gxs)


def _exact_stream(c, g):
    x, h = _in_stream(c, g)
    total = x.numel()
    y = _convolve(x.reshape(-1), h[:total], 2 * total)[:total]
    return y.reshape(x.shape)


_EXACT = dict(fft1d=_exact_fft1d, fft2d=_exact_fft2d, image=_exact_image, host_conv=_exact_host_conv,
              conv_batch=_exact_batch, fft_batch=_exact_batch, adjoint=_exact_adjoint, stream=_exact_stream)


def exact(case: dict, seed: int):
    return _EXACT[case["kind"]](case, _gen(seed))
