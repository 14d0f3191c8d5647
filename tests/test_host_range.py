"""The extent check behind direct host access (csrc/host_range.h), compiled for the host."""
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


def test_range_holds(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text('#include <cstdio>\n#include "host_range.h"\nint main() {\n' + "".join(
        f'    std::printf("%d\\n", mgb::range_holds({a}ull, {b}ull, {c}ull, {d}ull));\n' for a, b, c, d, _ in CASES) + "}\n")
    subprocess.run([cxx, "-std=c++17", f"-I{CSRC}", str(src), "-o", str(tmp_path / "t")], check=True)
    got = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    assert [int(g) for g in got] == [c[-1] for c in CASES]
