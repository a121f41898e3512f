"""The stripe pipeline (calls of few pairs) against the plain-C oracle, bit for
bit: profile lengths around its 32- and 64-row stripes, reads around its
32-column blocks and shorter than a stripe, one pair (a cluster of CTAs) to
more pairs than clusters, every mode it serves."""
import numpy as np
import pytest

import dummest_b200 as d
from dummest_b200 import _ffi as F
from dummest_b200 import synth
from oracle import port

pytestmark = pytest.mark.gpu


def _case(M, lengths, seed):
    rng = np.random.default_rng(seed)
    prof = synth.make_profile(rng, M, f"pipe{M}")
    reads = []
    for L in lengths:
        s = synth.random_dna(rng, L, 0.5)
        h = synth.sample_homolog(rng, prof, max_aa=25)[:L]
        reads.append(h + s[len(h):])
    return d.finalize_hmm(synth.hmmer3_text([prof]))[1:], reads


@pytest.mark.parametrize("M", [2, 30, 31, 32, 62, 63, 64, 65, 127, 128, 300, 700])
def test_pipeline_equals_oracle(M):
    p, reads = _case(M, [3, 4, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 200, 331], M)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        mid = ctx.score_pairs(sids, pid, d.MODE_MID)
        graph = ctx.score_pairs(sids, pid, d.MODE_MID | d.MODE_GRAPH)
        flt = ctx.score_pairs(sids, pid, d.MODE_FILTER)
        one = [ctx.score_pairs([s], pid, d.MODE_MID)[0] for s in sids[-3:]]
    for r, m, g, f in zip(reads, mid, graph, flt):
        want_mid, want_flt, _ = port.score_pair(*p, d.decode_dna(r))
        for got in (m, g):
            assert (got.mid.m, got.mid.e) == want_mid and (got.filter.m, got.filter.e) == want_flt, len(r)
        assert f.filter_f == port.filter_pair(*p, d.decode_dna(r)), len(r)
    for a, b in zip(one, mid[-3:]):
        assert (a.mid, a.filter) == (b.mid, b.filter)


@pytest.mark.parametrize("n", [1, 2, 9, 18, 19, 74, 148, 149, 888, 889])
def test_cluster_shapes_agree(n):
    """Calls of n pairs on both sides of the cluster sizes and of the line to
    the batched kernel: every pair scores as it does in the batched schedule."""
    p, reads = _case(290, [150 + 3 * k for k in range(40)], 9)
    with d.Context() as ctx, d.Context(rows_per_lane=4) as batched:
        got = []
        for c in (ctx, batched):
            pid = c.add_profile(*p)
            sids = c.add_dna(reads)
            got.append(c.score_pairs([sids[k % 40] for k in range(n)], pid, F.MODE_MID))
    for a, b in zip(*got):
        assert (a.mid, a.filter, a.filter_f) == (b.mid, b.filter, b.filter_f)


@pytest.mark.parametrize("R", [1, 2, 3, 4])
def test_batched_stripe_transitions_equal_oracle(R):
    """The batched schedule with R rows per lane, whose lanes run from stripe
    to stripe: one to several stripes, reads shorter than a period, around a
    lane's lag, and longer than a stripe's fill."""
    S = 32 * R
    for M in (S - 1, S, 2 * S - 1, 3 * S + 5):
        p, reads = _case(M, [3, 4, 5, 31, 32, 33, S - 1, S, S + 3, S + 92, S + 93, S + 130, 3 * S + 101], M)
        with d.Context(rows_per_lane=R) as ctx:
            pid = ctx.add_profile(*p)
            sids = ctx.add_dna(reads)
            mid = ctx.score_pairs(sids, pid, d.MODE_MID)
            flt = ctx.score_pairs(sids, pid, d.MODE_FILTER)
        for r, m, f in zip(reads, mid, flt):
            want_mid, want_flt, _ = port.score_pair(*p, d.decode_dna(r))
            assert (m.mid.m, m.mid.e) == want_mid and (m.filter.m, m.filter.e) == want_flt, (M, len(r))
            assert f.filter_f == port.filter_pair(*p, d.decode_dna(r)), (M, len(r))


@pytest.mark.parametrize("M,n", [(256, 1776), (256, 1777), (300, 2368), (300, 2369), (1000, 1900)])
def test_wide_blocks_equal_oracle(M, n):
    """Calls of more short reads than the 12-warp blocks' warps and as many as
    the 16-warp blocks' (three rows per lane), and on both sides of them."""
    p, reads = _case(M, [30 + 3 * k for k in range(20)], M)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        got = ctx.score_pairs([sids[k % 20] for k in range(n)], pid, d.MODE_MID)
    want = [port.score_pair(*p, d.decode_dna(r)) for r in reads]
    for k, r in enumerate(got):
        assert ((r.mid.m, r.mid.e), (r.filter.m, r.filter.e)) == (want[k % 20][0], want[k % 20][1])
