"""The pipelined adjoint against the FP64 oracle and central differences: rows
around its 32-row stripes, reads around its 32-column blocks and 64-column
checkpoints, from one pair (a cluster of CTAs) to more pairs than clusters, and
a call that mixes pairs inside the range of its unscaled values with one far
beyond it (log T above 900 bits), which the scaled kernel takes."""
import ctypes as C

import numpy as np
import pytest

import dummest_b200 as d
from dummest_b200 import _ffi as F
from dummest_b200 import synth
from oracle import port

pytestmark = pytest.mark.gpu


def _profile(M, seed):
    rng = np.random.default_rng(seed)
    prof = synth.make_profile(rng, M, f"adj{M}")
    return rng, prof, d.finalize_hmm(synth.hmmer3_text([prof]))[1:]


def _check(values, params, bg, reads, n=None):
    idx = [k % len(reads) for k in range(n or len(reads))]
    codes = [d.decode_dna(r) for r in reads]
    v64, p64 = values.astype(np.float64), params.astype(np.float64)
    want = [port.log_total(v64, p64, bg, c) for c in codes]
    got = {}
    with d.Context() as ctx:
        pid = ctx.add_profile(values, params, bg)
        sids = ctx.add_dna(reads)
        for mode in (F.ADJ_CKPT_OFF, F.ADJ_CKPT_ON):
            ctx.adjoint_checkpoint(mode)
            got[mode] = ctx.loglik_grad([sids[k] for k in idx], pid)
        _, tracks = ctx.posterior_summary(sids, pid)
    logt, gp, ge = got[F.ADJ_CKPT_OFF]
    for k, q in enumerate(idx):
        assert abs(logt[k] - want[q]) <= 1e-10 * max(1.0, abs(want[q]))
    assert np.array_equal(logt, got[F.ADJ_CKPT_ON][0])  # the recomputed blocks are the stored ones
    for a, b in zip((gp, ge), got[F.ADJ_CKPT_ON][1:]):
        np.testing.assert_allclose(a, b, rtol=1e-11, atol=1e-13 * np.abs(a).max())
    # the gradient along a direction of all emissions, against FP64 central differences
    rng = np.random.default_rng(1)
    step = v64[:, 4:] * rng.uniform(-1, 1, size=(values.shape[0], 25)) * 1e-5
    total = lambda sign: sum(port.log_total(np.hstack([v64[:, :4], v64[:, 4:] + sign * step]), p64, bg, codes[q]) for q in idx)
    slope = (total(1) - total(-1)) / 2
    assert abs(float((ge * step).sum()) - slope) <= 1e-5 * np.abs(ge * step).sum() + 1e-9
    # the expected matches of a row: enter x d log T / d enter (gradient entry 10), summed over the reads
    match = np.sum([t[2] for t in tracks], axis=0)
    if n is None:
        np.testing.assert_allclose(match, params[:-1, 10].astype(np.float64) * gp[:-1, 10], rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("M", [2, 30, 31, 32, 63, 64, 65, 200])
def test_stripe_and_block_edges(M):
    rng, prof, p = _profile(M, M)
    lengths = [3, 4, 31, 32, 33, 34, 63, 64, 65, 95, 96, 97, 128, 129, 161]
    reads = [synth.random_dna(rng, L, 0.5) for L in lengths]
    reads += [synth.sample_homolog(rng, prof, max_aa=30) + synth.random_dna(rng, 20, 0.5)]
    _check(*p, reads)


@pytest.mark.parametrize("n", [1, 2, 19, 75, 300])
def test_cluster_shapes(n):
    rng, prof, p = _profile(130, 7)
    _check(*p, [synth.random_dna(rng, 60 + 7 * k, 0.5) for k in range(9)], n)


def test_pairs_beyond_the_unscaled_range():
    rng, prof, p = _profile(2000, 3)
    reads = [synth.sample_homolog(rng, prof, max_aa=2000, fs_rate=0.001), synth.random_dna(rng, 200, 0.5)]
    reads.append(synth.sample_homolog(rng, prof, max_aa=60) + synth.random_dna(rng, 50, 0.5))
    assert port.log_total(p[0].astype(np.float64), p[1].astype(np.float64), p[2], d.decode_dna(reads[0])) > 900 * np.log(2)
    _check(*p, reads)


def _budget_context(budget):
    ctx = d.Context()
    ctx.close()  # the same context anew, with the budget
    ctx.opts.device_budget_bytes = budget
    ctx.h = C.c_void_p()
    assert ctx.lib.dmst_ctx_create(C.byref(ctx.opts), C.byref(ctx.h)) == F.DMST_OK
    return ctx


@pytest.mark.parametrize("M,L,n", [(100, 900, 6), (31, 300, 1), (32, 301, 3)])
def test_automatic_store_follows_what_the_pipeline_holds(M, L, n):
    """The full forward store is taken when the budget holds it at once: 3 x 32
    doubles per stripe and step and a share of T per stripe, in units of 32, and
    two boundary rows of two doubles per stripe and column in each direction."""
    rng, prof, p = _profile(M, 5)
    reads = [synth.random_dna(rng, L, 0.5) for _ in range(n)]
    stripes = (M + 32) // 32
    need = 8 * n * ((stripes * (L + 31) * 96 + stripes + 31) // 32 * 32 + 4 * stripes * L)
    for budget, checkpointed in ((need, False), (need - 1, True)):
        with _budget_context(budget) as ctx:
            pid = ctx.add_profile(*p)
            ctx.loglik_grad(ctx.add_dna(reads), pid)
            assert ctx.adjoint_checkpoint() == checkpointed


def test_a_pair_beyond_the_budget_on_the_pipeline_alone():
    """A read whose stores fit the budget on the one-warp kernel (two boundary
    rows) and not on the pipeline (two per stripe and direction) runs on the
    former and takes no more memory than the budget; shorter reads of the call
    stay on the pipeline, and the results are those of a call without a budget."""
    torch = pytest.importorskip("torch")
    rng, prof, p = _profile(1000, 5)
    reads = [synth.random_dna(rng, L, 0.5) for L in (20000, 700, 400)]
    h = synth.sample_homolog(rng, prof, max_aa=60)
    reads = [r[:100] + h + r[100 + len(h):] for r in reads]
    stripes, L = 32, 20000
    states = stripes * ((L + 31 + 63) // 64) * 32 * 11  # checkpoints: 11 values per lane
    one_warp = 8 * (states + 2 * stripes * L + 40 + 2 * 64 * 96 + 4 * (L + 4) + 32)
    pipelined = 8 * (states + 4 * stripes * L)  # at least
    budget = (one_warp + pipelined) // 2
    assert one_warp < budget < pipelined
    got, held = [], []
    for limit in (budget, 0):
        with _budget_context(limit) as ctx:
            ctx.adjoint_checkpoint(F.ADJ_CKPT_ON)
            pid = ctx.add_profile(*p)
            sids = ctx.add_dna(reads)
            ctx.loglik_grad(sids[1:], pid)
            ctx.score_pairs(sids, pid, F.MODE_FILTER)  # the null model's buffers for these reads
            free = torch.cuda.mem_get_info()[0]
            got.append(ctx.loglik_grad(sids, pid))
            held.append(free - torch.cuda.mem_get_info()[0])
    assert held[0] <= budget + (4 << 20) < held[1]
    assert np.array_equal(got[0][0], got[1][0])
    for x, y in zip(got[0][1:], got[1][1:]):
        np.testing.assert_allclose(x, y, rtol=1e-11, atol=1e-13 * np.abs(y).max())
