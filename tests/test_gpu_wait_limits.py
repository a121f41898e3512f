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


def _case(M, lengths):
    prof, p = _profile(M)
    return p, _reads([prof] * len(lengths), lengths)


def _gives_up(ctx, call):
    """The call with a budget of one poll ends with DMST_ETIMEOUT."""
    ctx.set_wait_limit(1)
    with pytest.raises(d.DmstError) as err:
        call()
    assert err.value.status == F.DMST_ETIMEOUT
    ctx.set_wait_limit(0)


# two stripes of 64 rows (and R = 1: two of 32), many; one pair (a cluster of CTAs), one warp or more a stripe
@pytest.mark.parametrize("M,lengths", [(64, [700, 900]), (600, [1500, 1200]), (200, [400] * 300), (2000, [3000])])
def test_pipelined_calls_that_give_up(M, lengths):
    """Filter, mid, graph and search calls of few pairs: DMST_ETIMEOUT (the mid
    call's pairs go to the exact path, which has the same budget), and the same
    results as before once the budget is restored."""
    p, reads = _case(M, lengths)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        a = _pairs(ctx.add_dna(reads), [pid] * len(reads))
        gate = np.zeros(1, np.float32)
        calls = [lambda: ctx.score_pairs_raw(a, d.MODE_FILTER), lambda: ctx.score_pairs_raw(a, d.MODE_MID),
                 lambda: ctx.score_pairs_raw(a, d.MODE_MID | d.MODE_GRAPH), lambda: ctx.search_raw(a, gate)]
        results = lambda res: list(zip(_scores(res), [r.filter_f for r in res]))
        before = [results(call()) for call in calls]
        for call, want in zip(calls, before):
            for _ in range(2):
                _gives_up(ctx, call)
                assert results(call()) == want


@pytest.mark.parametrize("M,lengths", [(32, [300, 350]), (200, [700, 500, 900]), (130, [400] * 200)])
def test_adjoint_that_gives_up(M, lengths):
    """Gradients and posteriors run again on the one-warp kernel: the same log T
    and tables bit for bit, the gradient up to the order of its sums."""
    p, reads = _case(M, lengths)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        for mode in (F.ADJ_CKPT_OFF, F.ADJ_CKPT_ON):
            ctx.adjoint_checkpoint(mode)
            got, launches = [], []
            for limit in (0, 1, 0):
                ctx.set_wait_limit(limit)
                got.append((ctx.loglik_grad(sids, pid), ctx.posterior_summary(sids, pid)))
                ctx.loglik_grad(sids, pid)
                launches.append(ctx.last_timing()["launches"])
            assert launches[0] == launches[2] == launches[1] - 1  # the pipeline's and the one-warp kernel's
            (lt, gp, ge), (plt, tracks) = got[0]
            for (l2, gp2, ge2), (pl2, tr2) in got[1:]:
                assert np.array_equal(lt, l2) and np.array_equal(plt, pl2)
                for x, y in ((gp, gp2), (ge, ge2)):
                    np.testing.assert_allclose(x, y, rtol=1e-11, atol=1e-13 * np.abs(x).max())
                assert all(np.array_equal(u, v) for t, t2 in zip(tracks, tr2) for u, v in zip(t, t2))


def test_search_whose_two_pipelines_give_up():
    """A search's survivors run on the few-pair pipeline (the filter wave of 1,000
    pairs does not), and those it gives up go to the exact path, which gives up
    too: both rings are emptied before the next call that uses them."""
    p, reads = _case(300, [950] * 40 + [300] * 960)
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        a = _pairs(ctx.add_dna(reads), [pid] * len(reads))
        gate = np.zeros(1, np.float32)
        want = _scores(ctx.search_raw(a, gate))
        assert ctx.last_timing()["exact_pairs"] > 0
        for _ in range(2):
            _gives_up(ctx, lambda: ctx.search_raw(a, gate))
            assert _scores(ctx.search_raw(a, gate)) == want


def test_pairs_that_the_exact_path_takes_over():
    """A mid call in flight behind a filter call that gave up finds the ring not
    empty: its pairs are scored on the exact path, with every field as ever."""
    p, reads = _case(600, [1900, 1500, 400, 90])
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        a = _pairs(ctx.add_dna(reads), [pid] * len(reads))
        b = _pairs([r.seq for r in a][::-1], [pid] * len(reads))
        fields = lambda res: [(s, r.mid_ln, r.filter_ln, r.filter_f) for s, r in zip(_scores(res), res)]
        want = fields(ctx.score_pairs_raw(b, d.MODE_MID))
        ctx.set_wait_limit(1)
        ctx.submit_raw(a, d.MODE_FILTER)
        ctx.set_wait_limit(0)
        ctx.submit_raw(b, d.MODE_MID)
        assert _status(ctx) is None
        got = _status(ctx)
        assert got is not None and fields(got) == want
        assert all(r.flags & F.RES_EXACT_PATH for r in got)
        assert fields(ctx.score_pairs_raw(b, d.MODE_MID | d.MODE_FORCE_EXACT)) == want


def test_plain_schedule_that_gives_up():
    """Two stripes of 32 rows on two warps, one of 64 on the exact path: the mid
    call's pairs are taken over, the filter call ends with DMST_ETIMEOUT."""
    p, reads = _case(50, [400, 300])
    with d.Context(rows_per_lane=1) as ctx:
        pid = ctx.add_profile(*p)
        a = _pairs(ctx.add_dna(reads), [pid] * len(reads))
        plain = lambda mode: [(s, r.filter_f) for res in [ctx.score_pairs_raw(a, mode | d.MODE_PLAIN)]
                              for s, r in zip(_scores(res), res)]
        want = [plain(m) for m in (d.MODE_MID, d.MODE_FILTER)]
        ctx.set_wait_limit(1)
        assert plain(d.MODE_MID) == want[0]
        assert ctx.last_timing()["exact_pairs"] == len(reads)
        _gives_up(ctx, lambda: plain(d.MODE_FILTER))
        assert [plain(m) for m in (d.MODE_MID, d.MODE_FILTER)] == want


def test_traceback_whose_replay_gives_up():
    """950 pairs score on the batched schedule, which waits for nothing; the hits'
    replay gives up, and no traceback table is made from its stores."""
    prof, p = _profile(100)
    rng = np.random.default_rng(5)
    reads = [synth.sample_homolog(rng, prof, max_aa=30)[:200] + synth.random_dna(rng, 300 + 7 * k, 0.5) for k in range(4)]
    reads += [synth.random_dna(rng, 250, 0.5)] * 946
    flat = lambda sims: [[(s[:5], s[5].tolist()) for s in q] for q in sims]
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        gates = [100.0] * 4 + [-1.0] * 946
        want = flat(ctx.align(sids, pid, gates)[0])
        assert any(want) and ctx.last_align_timing()["hits"] > 0
        for _ in range(2):
            _gives_up(ctx, lambda: ctx.align(sids, pid, gates))
            t = ctx.last_align_timing()
            assert t["hits"] > 0 and t["tables_ms"] == 0.0  # scored, not traced
            assert flat(ctx.align(sids, pid, gates)[0]) == want
