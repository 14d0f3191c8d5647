"""The extent check and the size limits behind direct host access
(csrc/host_range.h), compiled for the host."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mufft_gb300" / "csrc"

# (start, size, p, bytes): held
CASES = [
    (4096, 4096, 4096, 4096, 1),   # the whole range
    (4096, 4096, 4096, 4097, 0),   # its first byte page-locked, its last one not
    (4096, 4096, 6144, 2048, 1),
    (4096, 4096, 6144, 2049, 0),
    (4096, 4096, 8191, 1, 1),
    (4096, 4096, 8192, 0, 1),
    (4096, 4096, 8192, 1, 0),      # starts past the range
    (4096, 4096, 4095, 1, 0),      # starts before it
    (4096, 4096, 4096, 2 ** 64 - 1, 0),
    (2 ** 64 - 4096, 4096, 2 ** 64 - 8, 8, 1),
    (2 ** 64 - 4096, 4096, 2 ** 64 - 8, 9, 0),
    (0, 0, 4096, 8, 0),            # no range known
]

# (complex points, r2c or c2r, bytes): direct, where both ways were measured
LIMITS = [
    (2, 0, 1 << 20, 1), (8, 0, 1 << 20, 1), (64, 0, 1 << 20, 1), (16384, 0, 1 << 20, 1),
    (16, 0, 1 << 18, 1), (16, 0, 1 << 19, 0),  # 16 points: slower than staged from 512 KiB
    (32, 0, 1 << 19, 1), (32, 0, 1 << 20, 0),
    (4, 1, 1 << 20, 1), (8, 1, 1 << 18, 1), (8, 1, 1 << 19, 0), (16, 1, 1 << 19, 0),
    (32, 1, 1 << 19, 1), (32, 1, 1 << 20, 0), (128, 1, 1 << 20, 1),
    (1024, 0, (1 << 20) + 1, 0),
]


def _run(tmp_path, lines):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text('#include <cstdio>\n#include "host_range.h"\nint main() {\n' + "".join(
        f'    std::printf("%d\\n", (int)({line}));\n' for line in lines) + "}\n")
    subprocess.run([cxx, "-std=c++17", f"-I{CSRC}", str(src), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    return [int(v) for v in out.split()]


def test_range_holds(tmp_path):
    got = _run(tmp_path, [f"mgb::range_holds({a}ull, {b}ull, {c}ull, {d}ull)" for a, b, c, d, _ in CASES])
    assert got == [c[-1] for c in CASES]


def test_direct_host_bytes(tmp_path):
    got = _run(tmp_path, [f"{n}ull <= mgb::direct_host_bytes({m}u, {r})" for m, r, n, _ in LIMITS])
    assert got == [c[-1] for c in LIMITS]
