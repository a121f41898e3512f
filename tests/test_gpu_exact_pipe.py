"""The exact path's stripe pipeline against the plain-C oracle, bit for bit:
profile lengths around its 64-row stripes, reads around its 32-column blocks,
one pair (a cluster of CTAs) to many, rows that rescale, anchors, and calls on
both streams that share its scratch."""
import numpy as np
import pytest

import dummest_b200 as d
from dummest_b200 import _ffi as F
from dummest_b200 import synth
from oracle import port

pytestmark = pytest.mark.gpu


def _case(M, lengths, seed, homolog=25):
    rng = np.random.default_rng(seed)
    prof = synth.make_profile(rng, M, f"exact{M}")
    reads = []
    for L in lengths:
        s = synth.random_dna(rng, L, 0.5)
        h = synth.sample_homolog(rng, prof, max_aa=homolog)[:L]
        reads.append(h + s[len(h):])
    return d.finalize_hmm(synth.hmmer3_text([prof]))[1:], reads


@pytest.mark.parametrize("M", [2, 31, 32, 62, 63, 64, 65, 127, 128, 129, 400])
def test_forced_exact_equals_oracle(M):
    p, reads = _case(M, [3, 4, 29, 30, 31, 32, 59, 60, 61, 62, 90, 91, 121, 250], M)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        got = ctx.score_pairs(sids, pid, d.MODE_MID | d.MODE_FORCE_EXACT)
        cols, _ = ctx.anchors(sids, pid)
    for r, g, (am, ae, ar) in zip(reads, got, cols):
        codes = d.decode_dna(r)
        mid, flt, _ = port.score_pair(*p, codes)
        assert g.exact_path and (g.mid.m, g.mid.e) == mid and (g.filter.m, g.filter.e) == flt, len(r)
        wm, we, wr = port.anchors(*p, codes)
        np.testing.assert_array_equal(am, wm)
        np.testing.assert_array_equal(ae[am != 0], np.asarray(we)[am != 0])
        np.testing.assert_array_equal(ar[am != 0], np.asarray(wr)[am != 0])


@pytest.mark.parametrize("M,n", [(300, 1), (300, 2), (300, 40), (300, 200), (900, 3), (1500, 1)])
def test_rescaled_rows_equal_oracle(M, n):
    p, reads = _case(M, [3 * M + 50, 2 * M, 700, 3 * M], M, homolog=M)
    idx = [k % len(reads) for k in range(n)]
    want = [port.score_pair(*p, d.decode_dna(r)) for r in reads[:n]]
    assert any(w[2][0] > 0 for w in want)  # rows that rescale
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        for mode in (d.MODE_MID, d.MODE_MID | d.MODE_FORCE_EXACT, d.MODE_MID | d.MODE_GRAPH):
            for k, g in zip(idx, ctx.score_pairs([sids[k] for k in idx], pid, mode)):
                assert (g.mid.m, g.mid.e) == want[k][0] and (g.filter.m, g.filter.e) == want[k][1]


def test_calls_in_flight_share_the_scratch():
    """Submitted calls of one, many and no exact pairs: the exact kernel moves
    between the context's two streams while the call before it is in flight."""
    p, reads = _case(500, [1600, 1500, 700, 400] * 60, 4, homolog=500)
    plain = [synth.random_dna(np.random.default_rng(k), 300, 0.5) for k in range(60)]
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        none = ctx.add_dna(plain)
        sets = [sids[:1], none, sids[:200], none[:5], sids, sids[:3], none, sids[:150]]
        want = []
        for s in sets:
            want.append([(r.mid, r.filter) for r in ctx.score_pairs(s, pid)])
        arrays = []
        for s in sets:
            a = (F.Pair * len(s))()
            for k, q in enumerate(s):
                a[k].seq, a[k].profile, a[k].min_prob_ratio = q, pid, -2.0
            arrays.append((a, ctx.submit_raw(a, d.MODE_MID)))
        while ctx.complete() is not None:
            pass
    for (_, res), w in zip(arrays, want):
        assert [(d.Score(r.mid.m, r.mid.e), d.Score(r.filter.m, r.filter.e)) for r in res] == w


@pytest.mark.parametrize("flag", [d.MODE_FORCE_EXACT, d.MODE_EXACT_SEQUENTIAL])
def test_filter_calls_have_no_exact_path(flag):
    """A filter call scores in float, whatever the exact-path flags."""
    p, reads = _case(90, [300, 200, 100, 310, 210, 110], 8)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        got = []
        for mode in (d.MODE_FILTER, d.MODE_FILTER | flag, d.MODE_FILTER):
            ctx.score_pairs(sids[3:], pid, d.MODE_FILTER)  # other results in the buffers
            got.append([(r.filter_f, r.filter_ln, r.exact_path) for r in ctx.score_pairs(sids[:3], pid, mode)])
    assert got[0] == got[1] == got[2] and not any(g[2] for g in got[1])


@pytest.mark.parametrize("M", [62, 63, 64, 65, 127, 128, 129])
def test_reads_around_the_32_column_blocks(M):
    """The kernel's window blocks are 32 columns; its first look ahead is two."""
    p, reads = _case(M, [32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129], M + 1)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        got = ctx.score_pairs(sids, pid, d.MODE_MID | d.MODE_FORCE_EXACT)
        cols, _ = ctx.anchors(sids, pid)
    for r, g, col in zip(reads, got, cols):
        codes = d.decode_dna(r)
        mid, flt, _ = port.score_pair(*p, codes)
        assert (g.mid.m, g.mid.e) == mid and (g.filter.m, g.filter.e) == flt, len(r)
        _same_anchors(col, port.anchors(*p, codes))


def _same_anchors(got, want):
    (am, ae, ar), (wm, we, wr) = got, want
    np.testing.assert_array_equal(am, wm)
    np.testing.assert_array_equal(ae[am != 0], np.asarray(we)[am != 0])
    np.testing.assert_array_equal(ar[am != 0], np.asarray(wr)[am != 0])


@pytest.mark.parametrize("M,n", [(300, 1), (300, 200), (900, 2)])
def test_anchors_of_rescaled_rows_equal_oracle(M, n):
    """One pair (both discovery sweeps side by side) and many (in turn), rows that
    rescale in both sweeps: the anchors' products carry both rows' counts."""
    p, reads = _case(M, [3 * M + 50, 2 * M, 700, 3 * M], M, homolog=M)
    want = [port.anchors(*p, d.decode_dna(r)) for r in reads[:n]]
    assert port.score_pair(*p, d.decode_dna(reads[0]))[2][0] > 0
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        cols, _ = ctx.anchors([sids[k % len(reads)] for k in range(n)], pid)
    for k, got in enumerate(cols):
        _same_anchors(got, want[k % len(reads)])
