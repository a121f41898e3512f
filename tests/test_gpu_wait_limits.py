"""Waits of the stripe pipelines that run out, and what the calls in flight and
the calls after them return.  A wait is made to run out by a budget of one poll
(dmst_set_wait_limit): the kernels are bounded and end by themselves."""
import numpy as np
import pytest

import dummest_b200 as d
from dummest_b200 import _ffi as F
from dummest_b200 import synth

pytestmark = pytest.mark.gpu


def _profile(M, seed=1):
    prof = synth.make_profile(np.random.default_rng(seed), M, f"wait{M}")
    return prof, d.finalize_hmm(synth.hmmer3_text([prof]))[1:]


def _reads(profs, lengths, seed=2):
    """Reads that begin with a homolog of the whole profile (rows that rescale)."""
    rng = np.random.default_rng(seed)
    out = []
    for prof, L in zip(profs, lengths):
        h = synth.sample_homolog(rng, prof, max_aa=3000, fs_rate=0.001)[:L]
        out.append(h + synth.random_dna(rng, L - len(h), 0.5) if L > len(h) else h)
    return out


def _pairs(sids, pids):
    a = (F.Pair * len(sids))()
    for k, (s, p) in enumerate(zip(sids, pids)):
        a[k].seq, a[k].profile, a[k].min_prob_ratio = s, p, -2.0
    return a


def _scores(res):
    return [(r.mid.m, r.mid.e, r.filter.m, r.filter.e) for r in res]


def _status(ctx):
    """Completes the oldest call: its results, or None for DMST_ETIMEOUT."""
    try:
        return ctx.complete()
    except d.DmstError as err:
        assert err.status == F.DMST_ETIMEOUT
        return None


# The call that gives up is (M, L) pairs, costliest first, each on its own
# cluster; a profile of one stripe waits for nothing.  The next call's clusters
# are others (one pair, one cluster) or the same ones and more.
@pytest.mark.parametrize("first,second", [([(50, 100000), (600, 6000)], [(600, 20000)]),
                                          ([(50, 60000), (50, 60000), (300, 9000)], [(300, 23000), (300, 22000)]),
                                          ([(600, 6000), (600, 5000), (600, 4100)], [(600, L) for L in range(250, 330)]),
                                          ([(1000, 2500)] * 20, [(1000, L) for L in range(100, 300)])])
def test_exact_call_behind_one_that_gave_up(first, second):
    """A call in flight behind one whose waits ran out uses the same ring buffer,
    cut into other slots: it must not take the entries left there for its own."""
    mode = d.MODE_MID | d.MODE_FORCE_EXACT
    profs = {M: _profile(M) for M in {M for M, _ in first + second}}
    with d.Context() as ctx:
        pids = {M: ctx.add_profile(*p) for M, (_, p) in profs.items()}
        a, b = (_pairs(ctx.add_dna(_reads([profs[M][0] for M, _ in q], [L for _, L in q])), [pids[M] for M, _ in q])
                for q in (first, second))
        want_a, want_b = (_scores(ctx.score_pairs_raw(q, mode)) for q in (a, b))
        for _ in range(3):
            ctx.set_wait_limit(1)
            ctx.submit_raw(a, mode)
            ctx.set_wait_limit(0)
            ctx.submit_raw(b, mode)
            assert _status(ctx) is None
            got = _status(ctx)
            assert got is None or _scores(got) == want_b
            assert _scores(ctx.score_pairs_raw(b, mode)) == want_b
            assert _scores(ctx.score_pairs_raw(a, mode)) == want_a
