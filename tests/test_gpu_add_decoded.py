"""Decoded sequences in the blocks they are uploaded in: sequences around a
block's end and of a block and more score as the same letters decoded on the
device, and the host's memory holds one block beside the caller's codes."""
import os
import subprocess
import sys

import numpy as np
import pytest

import dummest_b200 as d
from dummest_b200 import synth

pytestmark = pytest.mark.gpu

BLOCK = 4 << 20
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("lengths", [[3], [3, 17, 16, 15], [700] * 12000, [BLOCK - 32, 16, 16, 16, 500],
                                     [300, BLOCK - 1, 300], [300, BLOCK + 1, 300, 301], [BLOCK, BLOCK + 16, 40]])
def test_blocks(lengths):
    rng = np.random.default_rng(len(lengths))
    p = d.finalize_hmm(synth.hmmer3_text([synth.make_profile(rng, 5, "blocks")]))[1:]
    letters = synth.random_dna(rng, sum(lengths), 0.5)
    at = np.cumsum([0] + lengths)
    dna = [letters[a:b] for a, b in zip(at, at[1:])]
    with d.Context() as ctx:
        pid = ctx.add_profile(*p)
        first = ctx.add_dna(dna[:1])
        got = ctx.add_decoded([d.decode_dna(s) for s in dna])
        want = ctx.add_dna(dna)
        # the reads at the ends, around each block and a few others
        pick = sorted({0, len(dna) - 1} | {k + e for k in np.flatnonzero(np.diff(at // BLOCK)) for e in (-1, 0, 1)
                                           if 0 <= k + e < len(dna)} | set(range(0, len(dna), 500)))
        scores = [[r.filter_f for r in ctx.score_pairs([ids[k] for k in pick], pid, d.MODE_FILTER)] for ids in (got, want)]
        assert scores[0] == scores[1]
        assert first == [0]


def test_host_memory_of_an_upload():
    """400 MB of codes take no copy of their own on the host."""
    code = """
import ctypes as C, resource
import numpy as np
import dummest_b200 as d
rss = lambda: resource.getrusage(resource.RUSAGE_SELF).ru_maxrss  # KB
with d.Context() as ctx:
    ctx.add_decoded([np.ones(1000, np.uint8)] * 10)
    L, n = 1000, 400000
    codes = np.ones(L * n, np.uint8)
    off = np.arange(n + 1, dtype=np.int64) * L
    before = rss()
    st = ctx.lib.dmst_seqs_add_decoded(ctx.h, codes.ctypes.data_as(C.POINTER(C.c_uint8)),
                                       off.ctypes.data_as(C.POINTER(C.c_int64)), n, None)
    assert st == 0 and ctx.seq_length(n) == L
    print("grown", rss() - before)
"""
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert int(out.stdout.split("grown")[1]) < 200 << 10
