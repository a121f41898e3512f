"""Traceback tables at the edges of their kernels: profiles around the exact
kernel's 64-row stripes, reads of a few lengths and around the
4096 columns that the optimal tables hold in shared memory.  A hit's
alignments do not depend on its company, so a hit traced alone (its two
discovery sweeps side by side, a block as wide as its read) equals the same hit
in a call of 200 (the sweeps in turn, blocks as wide as the longest read)."""
import numpy as np
import pytest

import dummest_b200 as d
from dummest_b200 import synth

pytestmark = pytest.mark.gpu


def _flat(sims):
    return [(s[:5], np.asarray(s[5]).tolist()) for s in sims]


@pytest.mark.parametrize("M,lengths", [(2, [40, 61]), (31, [93, 256, 257]), (62, [255, 190, 512]), (63, [511, 513]),
                                       (64, [300, 1025]), (129, [4095, 4096, 4097])])
def test_a_hit_alone_equals_the_hit_in_company(M, lengths):
    rng = np.random.default_rng(M)
    prof = synth.make_profile(rng, M, f"tables{M}")
    reads = []
    for L in lengths:
        h = synth.sample_homolog(rng, prof, max_aa=M)[:L - 7]
        s = synth.random_dna(rng, L - len(h), 0.5)
        reads.append(s[:5] + h + s[5:])
    p = d.finalize_hmm(synth.hmmer3_text([prof]))[1:]
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna(reads)
        idx = [k % len(reads) for k in range(200)]
        many, _ = ctx.align([sids[k] for k in idx], [pid] * len(idx), [100.0] * len(idx))
        alone = [ctx.align([s], [pid], [100.0])[0][0] for s in sids]
    assert M < 31 or all(alone)
    for k, got in zip(idx, many):
        assert _flat(got) == _flat(alone[k]), (M, len(reads[k]))


def test_a_long_hit_holds_24_bytes_per_cell():
    """The tables of a traced hit take 24 bytes per cell, and headroom of 30%."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    M, L = 1000, 50000
    prof = synth.make_profile(rng, M, "long")
    h = synth.sample_homolog(rng, prof, max_aa=M, fs_rate=0.001)
    read = synth.random_dna(rng, 20000, 0.5) + h
    read += synth.random_dna(rng, L - len(read), 0.5)
    p = d.finalize_hmm(synth.hmmer3_text([prof]))[1:]
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        sids = ctx.add_dna([read])
        ctx.anchors(sids, pid)
        ctx.align(sids, [pid], [-1.0])  # scored, not traced: every other buffer of the call
        free = torch.cuda.mem_get_info()[0]
        sims, _ = ctx.align(sids, [pid], [3e38])
        held = free - torch.cuda.mem_get_info()[0]
    assert sims[0]
    cells, per_column = (M + 1) * L, 400
    assert held <= 1.3 * (24 * cells + per_column * L) + (64 << 20), held / cells
