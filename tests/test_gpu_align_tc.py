"""The tensor-core alignment against the thread scan on the GPU: the same read
sets corrected by the default route and with the alignment's statistics form,
which keeps the thread scan. Integer and byte results: compared exactly.
Sizes where the kernel's paths change: candidate lists of several windows and
products, mates' lists longer than shared memory holds, few anchors (their
lists handed out in parts), equal and mixed lengths, more possible shifts than
the list holds (reads of short tandem repeats), both sides of the error rate
up to which it runs."""
import numpy as np
import pytest

import care_b200
from care_b200 import datagen

pytestmark = pytest.mark.gpu


def _reads(seed, n, lo, hi, genome, rate=0.01):
    rng = np.random.default_rng(seed)
    lengths = rng.integers(lo, hi + 1, n).astype(np.int32)
    start = (rng.random(n) * (genome.shape[0] - lengths + 1)).astype(np.int64)
    j = np.arange(hi)[None, :]
    rc = rng.random(n) < 0.5
    src = np.where(rc[:, None], start[:, None] + lengths[:, None] - 1 - j, start[:, None] + j)
    code = genome[np.clip(src, 0, genome.shape[0] - 1)]
    code = np.where(rc[:, None], 3 - code, code)
    err = rng.random((n, hi)) < rate
    code = np.where(err, (code + rng.integers(1, 4, (n, hi))) & 3, code)
    return datagen.ASCII[code], lengths


def _run(seqs, lengths, count_words, ranges, tuning=None, **opts):
    out = []
    # mirrored pairs count once: on the tensor cores those of any two lengths, in the statistics form of equal lengths
    same_count = not (tuning or {}).get("pair_mirror") or lengths.min() == lengths.max()
    with care_b200.Corrector(care_b200.default_options(**opts)) as c:
        c.upload_reads(care_b200.encode_reads(seqs, lengths), lengths)
        c.build_tables()
        if tuning:
            c.tuning = dict(care_b200.Tuning.from_dict({}).as_dict(), **tuning)
        c.count_word_compares(count_words)
        for first, count in ranges:
            r = c.correct_range(first, count)
            st = c.last_stats()
            if opts.get("max_error_rate", 0.2) > 0:      # with no error allowed the scan compares nothing
                assert (st["word_compares_run"] > 0) == count_words
            o = np.lexsort((r.cand_anchor_ids, r.cand_read_ids))
            out.append([r.status, r.num_edits, r.sequences, r.cand_read_ids[o], r.cand_anchor_ids[o], r.cand_shifts[o],
                        r.cand_use_edits[o], r.cand_sequences[o],
                        np.array([st["pairs"], st["word_compares"] if same_count else 0])])
    return out


def _same(seqs, lengths, ranges, **kw):
    a, b = _run(seqs, lengths, False, ranges, **kw), _run(seqs, lengths, True, ranges, **kw)
    for x, y in zip(a, b):
        for u, v in zip(x, y):
            assert np.array_equal(u, v)
    return a


@pytest.mark.parametrize("mirror", [0, 1])           # 1: pairs of any lengths answered with their mirrors
@pytest.mark.parametrize("lo,hi", [(100, 100), (50, 250), (33, 64), (256, 256)])
def test_long_candidate_lists(lo, hi, mirror):
    genome = np.random.default_rng(lo).integers(0, 4, 4 * (lo + hi))
    seqs, lengths = _reads(1, 1500, lo, hi, genome)
    res = _same(seqs, lengths, [(0, 1500), (3, 1), (17, 333)], kmerlength=16, num_maps=8, estimated_coverage=400.0,
                correct_candidates=1, min_overlap=30, tuning={"pair_mirror": mirror})
    assert res[0][8][0] > 1500 * 128                     # several windows of 128


@pytest.mark.parametrize("mirror", [0, 1])
def test_pairs_in_parts(mirror):
    genome = np.random.default_rng(5).integers(0, 4, 2500)
    seqs, lengths = _reads(2, 1200, 151, 151, genome)
    ranges = [(0, 2), (10, 128), (2, 700), (0, 1200)]
    for r in (ranges[:2], ranges[2:]):
        _same(seqs, lengths, r, kmerlength=20, num_maps=12, estimated_coverage=250.0, paired_end=1,
              tuning={"pair_mirror": mirror})


@pytest.mark.parametrize("unit", [1, 2, 3, 7])
def test_short_tandem_repeats(unit):
    rng = np.random.default_rng(unit)
    genome = np.concatenate([rng.integers(0, 4, 150), np.tile(rng.permutation(8)[:unit] & 3, 600 // unit),
                             rng.integers(0, 4, 150)])
    seqs, lengths = _reads(3, 160, 90, 120, genome, rate=0.02)
    _same(seqs, lengths, [(0, 160), (5, 20)], kmerlength=16, num_maps=8, estimated_coverage=400.0)


@pytest.mark.parametrize("mirror", [0, 1])
@pytest.mark.parametrize("lo,hi,unit", [(100, 100, 1), (150, 150, 2), (50, 250, 5), (256, 256, 4), (33, 64, 2)])
def test_overflowing_lists(lo, hi, unit, mirror):
    """Products with more possible shifts than the list holds, in one round of
    sums and in several, beside unique sequence."""
    rng = np.random.default_rng(unit + lo)
    genome = np.concatenate([rng.integers(0, 4, 2 * hi), np.tile(rng.permutation(8)[:unit] & 3, 2 * hi // unit),
                             rng.integers(0, 4, 2 * hi)])
    seqs, lengths = _reads(3, 300, lo, hi, genome, rate=0.02)
    _same(seqs, lengths, [(0, 300), (5, 20)], kmerlength=16, num_maps=8, estimated_coverage=400.0,
          correct_candidates=1, tuning={"pair_mirror": mirror})


@pytest.mark.parametrize("rate,overlap,ratio", [(0.0, 30, 0.3), (0.3, 1, 0.0), (0.30001, 30, 0.3), (0.2, 200, 1.0)])
def test_option_edges(rate, overlap, ratio):
    genome = np.random.default_rng(9).integers(0, 4, 3000)
    seqs, lengths = _reads(4, 800, 60, 200, genome)
    for mirror in (0, 1):
        _same(seqs, lengths, [(0, 800)], kmerlength=16, num_maps=16, estimated_coverage=80.0, max_error_rate=rate,
              min_overlap=overlap, min_overlap_ratio=ratio, tuning={"pair_mirror": mirror})
