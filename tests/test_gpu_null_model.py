"""The null model against the plain-C oracle (oracle/dmst_oracle.c), bit for
bit: lengths around the kernel's code look-ahead, seed chunks and transposes,
jobs of reads of different lengths, reads whose seeds reach the exponent
clamps, and zero frameshift rates."""
import numpy as np
import pytest

import dummest_b200 as d
from dummest_b200 import synth
from oracle import port

pytestmark = pytest.mark.gpu

LENGTHS = [3, 4, 5, 10, 11, 15, 16, 17, 18, 31, 32, 33, 34, 47, 48, 49, 64, 65, 130, 701, 2500]


def _profile(M=25, seed=5):
    txt = synth.hmmer3_text([synth.make_profile(np.random.default_rng(seed), M, "null")])
    return d.finalize_hmm(txt)[1:]


def _reads(rng):
    reads = [synth.random_dna(rng, L, gc) for L in LENGTHS for gc in (0.3, 0.7)]
    reads += ["N" * 40, "A" * 900, "ACGTN" * 30, "TAA" * 500 + "ATG" * 500, "TGA" * 2000 + "AAA" * 2000]
    return reads


@pytest.mark.parametrize("rates", [{}, {"insert1": 0.0, "delete2": 0.0}, {"insert2": 0.0, "delete1": 0.0},
                                   {"insert1": 0.3, "insert2": 0.2, "delete1": 0.2, "delete2": 0.1}])
def test_null_model_equals_oracle(rates):
    values, params, bg = _profile()
    reads = _reads(np.random.default_rng(11))
    with d.Context(rates=rates) as ctx:
        pid = ctx.add_profile(values, params, bg)
        for sid, r in zip(ctx.add_dna(reads), reads):
            pre, suf, scales = ctx.null_model(sid, pid, len(r))
            want = port.null_model(bg, d.decode_dna(r), port.rates(**rates))
            np.testing.assert_array_equal(pre, want[0], err_msg=f"prefix seeds, L={len(r)}")
            np.testing.assert_array_equal(suf, want[1], err_msg=f"suffix seeds, L={len(r)}")
            np.testing.assert_array_equal(scales, np.asarray(want[2])[:3], err_msg=f"scales, L={len(r)}")


def test_jobs_of_ragged_reads_score_as_the_oracle():
    """Reads of 40 different lengths against two profiles: one job holds
    several lengths, and its pairs of several profiles."""
    rng = np.random.default_rng(3)
    profs = [_profile(30, 1), _profile(45, 2)]
    reads = [synth.random_dna(rng, L, 0.5) for L in range(200, 240)] + [synth.random_dna(rng, 3, 0.5)]
    with d.Context() as ctx:
        pids = [ctx.add_profile(*p) for p in profs]
        sids = ctx.add_dna(reads)
        for pid, p in zip(pids, profs):
            res = ctx.score_pairs(sids + sids, [pid] * len(sids) + [pids[0]] * len(sids))
            for r, got in zip(reads, res):
                mid, flt, _ = port.score_pair(*p, d.decode_dna(r))
                assert (got.mid.m, got.mid.e) == mid and (got.filter.m, got.filter.e) == flt


@pytest.mark.parametrize("rates", [{}, {"insert1": 1e-4, "insert2": 1e-6, "delete1": 1e-6, "delete2": 1e-4},
                                   {"insert1": 1e-25, "insert2": 1e-25, "delete1": 1e-25, "delete2": 1e-25}])
def test_scaled_passes_equal_oracle(rates):
    """Reads around the scaled passes' groups of 16 columns, reads whose
    composition drives the seeds past both ends of the float range, reads
    without a codon for long, and rates too small for the scaled passes."""
    values, params, bg = _profile(60, 8)
    rng = np.random.default_rng(12)
    order = np.argsort(bg[:20])
    aa = {d.decode_dna(a + b + c)[0]: a + b + c for a in "ACGT" for b in "ACGT" for c in "ACGT"}
    rare, common = (aa[int(order[k])] for k in (0, 19))
    reads = [synth.random_dna(rng, L, 0.5) for L in (18, 19, 20, 34, 35, 36, 50, 51, 66, 67)]
    reads += [rare * 800 + common * 800, common * 800 + rare * 800, common * 300 + rare * 600 + common * 300,
              "TAATAGTGA" * 60 + common * 300, synth.random_dna(rng, 9000, 0.35)]
    with d.Context(rates=rates) as ctx:
        pid = ctx.add_profile(values, params, bg)
        for sid, r in zip(ctx.add_dna(reads), reads):
            pre, suf, scales = ctx.null_model(sid, pid, len(r))
            want = port.null_model(bg, d.decode_dna(r), port.rates(**rates))
            np.testing.assert_array_equal(pre, want[0], err_msg=f"prefix seeds, L={len(r)}")
            np.testing.assert_array_equal(suf, want[1], err_msg=f"suffix seeds, L={len(r)}")
            np.testing.assert_array_equal(scales, np.asarray(want[2])[:3], err_msg=f"scales, L={len(r)}")
