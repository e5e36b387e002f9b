"""The MSA stage on the GPU against the CPU oracle where its paths change: more
rows than shared memory stages (rows staged in chunks, with refinement and
candidate correction), read lengths on and off the 16-base grid, columns
outside the anchor that candidate correction reads, a dataset coverage whose
refinement threshold is zero, every quality encoding. Integer and byte results:
compared exactly."""
import pytest

import _oracle
from care_b200 import datagen
from test_gpu_parity import compare_with_oracle, run_gpu

pytestmark = pytest.mark.gpu


def _check(tmp_path, rs, args):
    inp = str(tmp_path / "in.fq")
    rs.write_fastq(inp)
    res, tables = run_gpu([inp], args)
    compare_with_oracle([inp], args, res, tables)
    return res


@pytest.mark.parametrize("quality", ["", "-q --qualityScoreBits 1", "-q --qualityScoreBits 2", "-q --qualityScoreBits 8"])
def test_rows_staged_in_chunks(tmp_path, quality):
    rs = datagen.single_end_uneven(seed=81, genome_size=6000, coverage=220.0, Lmin=60, Lmax=130, repeat_fraction=0.0)
    res = _check(tmp_path, rs, f"-c 220 -k 20 -h 8 --pairmode SE --candidateCorrection {quality}")
    assert len(res.cand_read_ids) > 0


@pytest.mark.parametrize("L", [33, 64, 159, 160, 161, 256])
def test_lengths_around_the_grid(tmp_path, L):
    rs = datagen.single_end_uniform(seed=82, genome_size=40 * L, num_reads=1200, L=L)
    _check(tmp_path, rs, "-c 30 -k 17 -h 16 -q --qualityScoreBits 8 --pairmode SE --candidateCorrection")


@pytest.mark.parametrize("columns", [0, 1, 16, 40, 300])
def test_new_columns(tmp_path, columns, monkeypatch):
    flag = f" --candidateCorrectionNewColumns {columns}"
    parse = _oracle.opts_from_args

    def with_columns(args):
        o = parse(args.replace(flag, ""))
        o.new_columns_to_correct = columns
        return o
    monkeypatch.setattr(_oracle, "opts_from_args", with_columns)
    rs = datagen.single_end_uneven(seed=83, genome_size=8000, coverage=40.0, Lmin=50, Lmax=140, repeat_fraction=0.0)
    _check(tmp_path, rs, "-c 40 -k 18 -h 16 -q --qualityScoreBits 2 --pairmode SE --candidateCorrection" + flag)


@pytest.mark.parametrize("coverage", [1, 3, 4, 10])
def test_small_dataset_coverage(tmp_path, coverage):
    rs = datagen.single_end_uneven(seed=84, genome_size=60_000, coverage=9.0, Lmin=80, Lmax=140, repeat_fraction=0.3)
    _check(tmp_path, rs, f"-c {coverage} -k 18 -h 16 -q --qualityScoreBits 2 --pairmode SE --candidateCorrection")
