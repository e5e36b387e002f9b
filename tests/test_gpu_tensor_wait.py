"""The completion wait of the tensor-core alignment running out: the kernel
ends with its status set, writes no result of the product it gave up on, and
leaves the GPU as a later launch needs it; the MSA behind it leaves at once
(the alignments are unwritten). The limit of the wait is set to
zero polls; the products themselves complete."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "harness", "tensor_wait.cu")
OUT = os.path.join(ROOT, "tests", "_build", "libtensor_wait.so")
CSRC = os.path.join(ROOT, "care_b200", "csrc")
DEPS = [SRC] + [os.path.join(CSRC, f) for f in ("device.cuh", "tc_math.cuh", "tc05.cuh", "kernels.cuh", "align_tc.cuh")]
TENSOR_WAIT = 16 | 32                                # kStatusTensorWait | kStatusIncomplete
LIMIT = 1 << 22                                      # kTcWaitLimit


def build():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        tmp = f"{OUT}.{os.getpid()}.tmp"
        subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-O3", "-shared",
                        "-Xcompiler", "-fPIC", "-std=c++17", "-o", tmp, SRC], check=True, capture_output=True)
        os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


def _run(lib, rows, n, L, limit, grid, queue):
    res = np.zeros((n * (n - 1), 8), np.uint8)
    corrected = np.zeros(n, np.uint8)
    status = ctypes.c_int(-1)
    assert lib.gpu_align_with_limit(rows.ctypes.data_as(ctypes.c_void_p), n, L, ctypes.c_uint32(limit), grid, queue,
                                    res.ctypes.data_as(ctypes.c_void_p), corrected.ctypes.data_as(ctypes.c_void_p),
                                    ctypes.byref(status)) == 0
    return status.value, res, corrected


# reads of 256 bases take several products per list of candidates, those of 60 one
@pytest.mark.gpu
@pytest.mark.parametrize("L,n,queue", [(60, 9, 0), (256, 40, 0), (256, 40, 1)])
def test_wait_that_runs_out(L, n, queue):
    lib = build()
    rng = np.random.default_rng(L)
    rows = rng.integers(0, 1 << 32, (n, (L + 15) // 16), dtype=np.uint32)
    rows[1::2] = rows[0::2][: n // 2]                 # copies: pairs that align
    status, res, corrected = _run(lib, rows, n, L, 0, 3, queue)
    assert status == TENSOR_WAIT
    assert (res == 0x5A).all()                        # no result
    assert (corrected == 0x5A).all()                  # the MSA looked at no anchor
    status, res, corrected = _run(lib, rows, n, L, LIMIT, 3, queue)
    assert status == 0 and (corrected != 0x5A).all()
    assert res[0, 6] == 1 and not res[0, :2].any()    # read 1 is a copy of read 0: forward, shift 0
