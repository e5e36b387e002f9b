"""The row windows that the MSA stages its words with: no word outside a row is
read, at any length, shift and orientation, and the codes inside it arrive. The
kernel discards what comes from outside a row, so a stray read shows in no
result. Runs without a GPU."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "harness", "windows.cu")
OUT = os.path.join(ROOT, "tests", "_build", "libwindows.so")
DEPS = [SRC, os.path.join(ROOT, "care_b200", "csrc", "device.cuh")]


@pytest.fixture(scope="module")
def lib():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        tmp = f"{OUT}.{os.getpid()}.tmp"
        subprocess.run(["nvcc", "-shared", "-Xcompiler", "-fPIC", "-O2", "-std=c++17", "-o", tmp, SRC],
                       check=True, capture_output=True)
        os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


# span: the codes a turned row is read back from (its length for bases, the
# storage's longest read for qualities)
@pytest.mark.parametrize("bits", [1, 2, 8])
@pytest.mark.parametrize("extra", [0, 1, 40])
def test_windows_stay_inside_the_row(lib, bits, extra):
    for L in range(1, 257):
        span = min(L + extra, 256)
        r = (ctypes.c_int * 2)(1 << 30, -(1 << 30))
        wrong = lib.hd_windows(bits, span, L, 0 if L % 2 else 16, r)
        words = -(-span * bits // 32)
        assert 0 <= r[0] and r[1] < words, f"length {L}: words {r[0]} .. {r[1]} of {words}"
        assert wrong == 0, f"length {L}"
