"""The tensor-core alignment's operands, thresholds and exact counts
(care_b200/csrc/tc_math.cuh), emulated on the host with the addresses its
matrix descriptors form, against the CPU oracle's shifted Hamming alignment.
Integers throughout: compared exactly. Runs without a GPU."""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

import _oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "harness", "align_tc.cu")
OUT = os.path.join(ROOT, "tests", "_build", "libalign_tc.so")
DEPS = [SRC] + [os.path.join(ROOT, "care_b200", "csrc", f) for f in ("device.cuh", "tc_math.cuh")]


@pytest.fixture(scope="module")
def lib():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        tmp = f"{OUT}.{os.getpid()}.tmp"
        subprocess.run(["nvcc", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-O2", "-std=c++17",
                        "-o", tmp, SRC], check=True, capture_output=True)
        os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


def _enc(s, words):
    out = (ctypes.c_uint32 * words)()
    _oracle.lib().co_encode_2bit(s.encode(), len(s), out)
    return np.frombuffer(out, np.uint32).copy()


def _rc(s):
    return s[::-1].translate(str.maketrans("ACGT", "TGCA"))


def _rand(rng, n, letters="ACGT"):
    return "".join(rng.choice(letters) for _ in range(n))


def _mutate(rng, s, k):
    s = list(s)
    for _ in range(k if s else 0):
        s[rng.randrange(len(s))] = rng.choice("ACGT")
    return "".join(s)


def _oracle_one(a, c, mo, rate, ratio):
    r = _oracle.CoAlign()
    _oracle.lib().co_shd(_enc(a, 17).ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), len(a),
                         _enc(c, 17).ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), len(c), mo,
                         ctypes.c_float(rate), ctypes.c_float(ratio), ctypes.byref(r))
    return r


FIXED = [16, 17, 31, 32, 33, 64, 100, 150, 151, 255, 256]


@pytest.mark.parametrize("seed", range(90))
def test_operands_and_results_match_the_oracle(lib, seed):
    rng = random.Random(300 + seed)
    uniform = seed % 2 == 0
    La = FIXED[seed % len(FIXED)] if seed % 3 else rng.randint(1, 256)
    n = rng.choice([1, 7, 8, 9, 17, 32])
    lens = [La] * n if uniform else [rng.randint(1, 256) for _ in range(n)]
    mo = rng.choice([30, 30, 1, 20, 45])
    rate = rng.choice([0.2, 0.2, 0.05, 0.3, 0.0])
    ratio = rng.choice([0.3, 0.3, 0.0, 1.0, 0.5])
    letters = "ACGT" if seed % 5 else rng.choice(["A", "AC", "AG"])          # ties and possible shifts everywhere
    g = _rand(rng, 900, letters)
    at = 300
    a = _mutate(rng, g[at:at + La], rng.randint(0, 3))
    cands = []
    for L in lens:
        c0 = at + rng.randint(-L + 5, La - 5) if La > 5 and L > 5 else at
        c = _mutate(rng, g[max(c0, 0):max(c0, 0) + L], rng.randint(0, 8))
        c = (c + _rand(rng, L))[:L]
        cands.append(_rc(c) if rng.random() < 0.5 else c if rng.random() < 0.8 else _rand(rng, L))
    max_len = max([La] + lens)
    pitch = (max_len + 15) // 16
    rows = np.stack([_enc(c, pitch) for c in cands])
    rows[:, -1] |= np.uint32(0x1)        # storage past a read's end need not be zero
    rows = np.where((np.arange(pitch)[None, :] * 16 + 16 <= np.array(lens)[:, None]) |
                    (np.array(lens)[:, None] % 16 == 0), np.stack([_enc(c, pitch) for c in cands]), rows)
    ln = np.array(lens, np.int32)
    aw = _enc(a, 17)
    got = []
    for per_column in ([0, 1] if uniform else [1]):
        out = np.zeros((n, 22), np.int32)
        rc = lib.hd_tc(aw.ctypes.data_as(ctypes.c_void_p), La, rows.ctypes.data_as(ctypes.c_void_p), pitch,
                       ln.ctypes.data_as(ctypes.c_void_p), n, max_len, mo, ctypes.c_float(rate), ctypes.c_float(ratio),
                       ctypes.c_float(0.06), per_column, out.ctypes.data_as(ctypes.c_void_p))
        assert rc >= 0
        got.append(out)
    for out in got[1:]:
        assert np.array_equal(got[0], out)
    minov = max(mo, int(np.float32(La) * np.float32(ratio)))
    for i, c in enumerate(cands):
        o = got[0][i]

        def check(x, y, at, orient):
            """(x, y) with x as anchor: results from o[at], the orientation."""
            f, r = _oracle_one(x, y, mo, rate, ratio), _oracle_one(x, _rc(y), mo, rate, ratio)
            want = _oracle.lib().co_orientation(ctypes.byref(f), ctypes.byref(r), len(x), len(y), ctypes.c_float(ratio),
                                                mo, ctypes.c_float(0.06))
            assert orient == want
            if want in (1, 2):
                b = f if want == 1 else r
                at += 5 * (want - 1)
                assert list(o[at:at + 5]) == [b.score, b.overlap, b.shift, b.nops, b.valid]
            return f, r

        f, r = check(a, c, 0, o[20])
        if lens[i] >= La:                                # the mirrored pair
            m, mr = check(c, a, 10, o[21])
            if lens[i] == La and La >= minov:            # every alignment in full
                for k, x in enumerate((f, r, m, mr)):
                    assert list(o[5 * k:5 * k + 5]) == [x.score, x.overlap, x.shift, x.nops, x.valid]


@pytest.mark.parametrize("seed", range(60))
def test_counts_of_an_overflowing_list(lib, seed):
    """The form that counts a column's possible shifts from their bits and
    stops at what no longer improves, against the count of every possible
    shift: tandem repeats with ties, errors and unique ends."""
    rng = random.Random(900 + seed)
    La = FIXED[seed % len(FIXED)]
    n = rng.choice([1, 5, 8])
    lens = [La if seed % 2 else rng.randint(16, 256) for _ in range(n)]
    mo, ratio, rate = rng.choice([30, 1, 12]), rng.choice([0.3, 0.0]), rng.choice([0.2, 0.3, 0.05])
    unit = _rand(rng, 1 + seed % 7)
    reads = []
    for L in [La] + lens:
        at = rng.randrange(len(unit))
        r = (unit * 300)[at:at + L]
        if rng.random() < 0.5:                           # an end outside the repeat
            k = rng.randint(0, L)
            r = r[:k] + _rand(rng, L - k)
        r = _mutate(rng, r, rng.choice([0, 0, 2, L // 12]))
        reads.append(_rc(r) if rng.random() < 0.3 else r)
    max_len = max([La] + lens)
    pitch = (max_len + 15) // 16
    rows = np.stack([_enc(c, pitch) for c in reads[1:]])
    ln = np.array(lens, np.int32)
    out = []
    for form in (1, 2):
        o = np.zeros((n, 22), np.int32)
        hits = lib.hd_tc(_enc(reads[0], 17).ctypes.data_as(ctypes.c_void_p), La, rows.ctypes.data_as(ctypes.c_void_p),
                         pitch, ln.ctypes.data_as(ctypes.c_void_p), n, max_len, mo, ctypes.c_float(rate),
                         ctypes.c_float(ratio), ctypes.c_float(0.06), form, o.ctypes.data_as(ctypes.c_void_p))
        assert hits >= 0
        out.append(o)
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("L,coverage,ratio,anchors,mirror,tensor", [
    (36, 40, 0.3, 200_000, 0, 0), (50, 20, 0.3, 200_000, 0, 0), (50, 40, 0.3, 200_000, 0, 0),
    (50, 30, 0.3, 200_000, 1, 0), (60, 20, 0.3, 200_000, 0, 0), (85, 10, 0.3, 200_000, 0, 0),
    (85, 20, 0.3, 200_000, 0, 1), (100, 5, 0.3, 200_000, 0, 0), (100, 20, 0.3, 200_000, 0, 1),
    (150, 5, 0.3, 200_000, 0, 0), (150, 10, 0.3, 200_000, 0, 1), (150, 30, 0.3, 200_000, 1, 1),
    (100, 30, 0.8, 200_000, 0, 0), (150, 30, 0.9, 200_000, 0, 0), (150, 30, 0.6, 200_000, 0, 1),
    (250, 5, 0.3, 200_000, 0, 1), (250, 30, 0.8, 200_000, 0, 1), (250, 30, 0.9, 200_000, 0, 1),
    (50, 30, 0.3, 1000, 0, 0), (50, 5, 0.3, 4000, 0, 0), (70, 5, 0.3, 1000, 0, 1), (100, 5, 0.3, 128, 0, 1),
    (150, 30, 0.3, 128, 0, 1)])
def test_route_of_a_call(lib, L, coverage, ratio, anchors, mirror, tensor):
    """The rule between the thread scan and the tensor cores at sizes where one
    of them was measured to be 15 % or more ahead."""
    assert lib.hd_tc_faster(L, 30, ctypes.c_float(ratio), ctypes.c_float(coverage), anchors, mirror) == tensor


def test_random_pairs_rarely_stay_possible(lib):
    """The one-bit sums rule out nearly every shift of unrelated reads: that
    is what makes the exact counts few."""
    rng = random.Random(1)
    L, n = 150, 32
    a = _rand(rng, L)
    rows = np.stack([_enc(_rand(rng, L), 10) for _ in range(n)])
    ln = np.full(n, L, np.int32)
    out = np.zeros((n, 22), np.int32)
    hits = lib.hd_tc(_enc(a, 17).ctypes.data_as(ctypes.c_void_p), L, rows.ctypes.data_as(ctypes.c_void_p), 10,
                     ln.ctypes.data_as(ctypes.c_void_p), n, L, 30, ctypes.c_float(0.2), ctypes.c_float(0.3),
                     ctypes.c_float(0.06), 0, out.ctypes.data_as(ctypes.c_void_p))
    assert 0 <= hits <= 4
