"""Two host threads, a context each, on reads of very different lengths: no
call may meet a launch limit that the other thread's call has set (the
kernels' shared memory grows with the longest read and the number of
candidates per map)."""
import threading

import numpy as np
import pytest

import care_b200
from care_b200 import datagen

pytestmark = pytest.mark.gpu


def _corrector(L, n, coverage, seed):
    rng = np.random.default_rng(seed)
    genome = rng.integers(0, 4, n * L // 30 + 2 * L)
    start = rng.integers(0, genome.shape[0] - L, n)
    code = genome[start[:, None] + np.arange(L)[None, :]]
    err = rng.random(code.shape) < 0.01
    code = np.where(err, (code + rng.integers(1, 4, code.shape)) & 3, code)
    lengths = np.full(n, L, np.int32)
    c = care_b200.Corrector(care_b200.default_options(kmerlength=16, num_maps=24, estimated_coverage=coverage))
    c.upload_reads(care_b200.encode_reads(datagen.ASCII[code], lengths), lengths)
    c.build_tables()
    return c


def test_contexts_of_two_threads():
    calls, errors = 400, []
    sets = [_corrector(40, 600, 10.0, 1), _corrector(256, 600, 150.0, 2)]
    want = [c.correct_range(0, 64).sequences.copy() for c in sets]
    start = threading.Barrier(2)

    def work(i):
        try:
            start.wait()
            for _ in range(calls):
                if not np.array_equal(sets[i].correct_range(0, 64).sequences, want[i]):
                    raise AssertionError("other results")
        except Exception as e:                        # noqa: BLE001 (reported below)
            errors.append(f"{i}: {e}")

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in sets:
        c.close()
    assert not errors
