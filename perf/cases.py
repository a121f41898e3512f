"""Performance cases of the search path: what a program that uses this package has it do.

Every case is one pass through the public API of dummest_b200.engine.Context,
from sequences in host memory to results in host memory.  Sizes follow the
configurations of bench.py and dummest_b200/synth.py (profiles of 50 to 2000
rows, reads of 75 to 3000 nt, windows of 10 kb, calibration sequences of
3 kb) and go down to a single read.

  kind        one pass
  score       reads of a FASTA batch (packed, or ASCII for one read) against
              profiles: mid-anchored score, or the float filter
  search      the two waves: filter on every pair, score on the survivors
  calibrate   random sequences of a new profile scored, Gumbel fit
  align       hits with their alignments (traceback)
  grad        log-likelihood and its gradient for a profile being refined
  posterior   posterior summary of the windows of a long hit region
  windows     prefilter hit rows to windows, cut from a resident genome,
              scored with the filter against the profiles that they name

Lengths and the choice of implanted reads depend on the case alone, so that
every seed costs the same; bases, emissions and implants come from the seed.
"""
import math
import random

import numpy as np
import torch

import dummest_b200 as d
from dummest_b200 import _ffi as F

# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # one read typed in or streamed against one family: launches and latency
        {"name": "one_read", "kind": "score", "filter": False, "profiles": 1, "mmin": 120, "mmax": 120, "reads": 1,
         "lmin": 300, "lmax": 300, "strands": 1, "tune": False, "shape_seed": 1},
        # short sequencer reads against a few families, default kernel shapes
        {"name": "batch_short", "kind": "score", "filter": False, "profiles": 16, "mmin": 40, "mmax": 300,
         "reads": 500, "lmin": 75, "lmax": 300, "strands": 2, "tune": False, "shape_seed": 2},
        # the batched configuration (64 families, ragged reads, both strands), kernel shapes tuned once
        {"name": "batch_mid", "kind": "score", "filter": False, "profiles": 64, "mmin": 50, "mmax": 800,
         "reads": 1000, "lmin": 150, "lmax": 3000, "strands": 2, "tune": True, "shape_seed": 3},
        # the lean filter pass alone over the same kind of batch
        {"name": "filter_batch", "kind": "score", "filter": True, "profiles": 32, "mmin": 50, "mmax": 800,
         "reads": 500, "lmin": 150, "lmax": 3000, "strands": 2, "tune": True, "shape_seed": 4},
        # filter, E-value gate and score on the survivors in one call
        {"name": "search", "kind": "search", "profiles": 32, "mmin": 50, "mmax": 800, "reads": 500, "lmin": 150,
         "lmax": 3000, "strands": 2, "gate": 1e6, "shape_seed": 5},
        # calibration of one new profile: 200 random sequences of 3 kb
        {"name": "calibrate", "kind": "calibrate", "m": 300, "trials": 200, "length": 3000, "shape_seed": 6},
        # a contig scanned with a long family: few long windows, some with frameshifted homologs
        {"name": "scan", "kind": "score", "filter": False, "profiles": 1, "mmin": 2000, "mmax": 2000, "reads": 8,
         "lmin": 10000, "lmax": 10000, "strands": 2, "tune": False, "shape_seed": 7},
        # hits with alignments: one family, reads that carry a homolog between random flanks
        {"name": "align", "kind": "align", "m": 400, "reads": 32, "flank": 500, "gate": 1e6, "shape_seed": 8},
        # a profile refined on a small family: gradient with the full forward store
        {"name": "grad_small", "kind": "grad", "m": 200, "reads": 64, "lmin": 300, "lmax": 1200, "ckpt": False,
         "shape_seed": 9},
        # a profile refined on a large family: column-checkpointed gradient
        {"name": "grad_ckpt", "kind": "grad", "m": 400, "reads": 1024, "lmin": 600, "lmax": 2400, "ckpt": True,
         "shape_seed": 10},
        # posterior decoding of the windows around hits
        {"name": "posterior", "kind": "posterior", "m": 400, "reads": 12, "lmin": 2000, "lmax": 3000,
         "shape_seed": 11},
        # the prefilter's hit rows: windows of a resident genome, decoded on the device and filtered
        {"name": "windows", "kind": "windows", "profiles": 8, "mmin": 100, "mmax": 400, "hits": 2000,
         "genome": 8_000_000, "records": 8, "shape_seed": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        c = _drawn(rng)
        if work(c)["flops"] <= most:
            return c


def _drawn(rng):
    kind = rng.choice(["score", "score", "score", "search", "calibrate", "scan", "align", "grad", "grad", "posterior",
                       "windows"])
    ss = rng.randrange(100, 1_000_000)
    if kind in ("score", "search"):
        # reads and profiles from one of each to the batched configuration's
        c = {"kind": kind, "profiles": _log_int(rng, 1, 64), "reads": _log_int(rng, 1, 700), "strands": rng.choice([1, 2])}
        c["mmin"] = _log_int(rng, 2, 300)
        c["mmax"] = _log_int(rng, c["mmin"], 800)
        c["lmin"] = _log_int(rng, 30, 1000)
        c["lmax"] = _log_int(rng, c["lmin"], 3000)
        if kind == "score":
            c.update(filter=rng.random() < 0.25, tune=rng.random() < 0.3)
        else:
            c["gate"] = 1e6
    elif kind == "calibrate":
        c = {"kind": kind, "m": _log_int(rng, 40, 900), "trials": _log_int(rng, 20, 400), "length": _log_int(rng, 500, 5000)}
    elif kind == "scan":
        L = _log_int(rng, 3000, 10000)
        c = {"kind": "score", "filter": False, "profiles": 1, "reads": rng.randrange(1, 9), "strands": 2, "tune": False,
             "lmin": L, "lmax": L}
        c["mmin"] = c["mmax"] = _log_int(rng, 700, 2000)
    elif kind == "align":
        c = {"kind": kind, "m": _log_int(rng, 40, 500), "reads": _log_int(rng, 1, 40), "flank": _log_int(rng, 50, 800),
             "gate": rng.choice([1.0, 1e6])}
    elif kind == "grad":
        c = {"kind": kind, "m": _log_int(rng, 30, 500), "reads": _log_int(rng, 1, 800), "ckpt": rng.random() < 0.5}
        c["lmin"] = _log_int(rng, 100, 1000)
        c["lmax"] = _log_int(rng, c["lmin"], 2400)
    elif kind == "posterior":
        c = {"kind": kind, "m": _log_int(rng, 60, 700), "reads": _log_int(rng, 1, 24)}
        c["lmin"] = _log_int(rng, 300, 2000)
        c["lmax"] = _log_int(rng, c["lmin"], 3000)
    else:
        c = {"kind": kind, "profiles": rng.randrange(1, 9), "hits": _log_int(rng, 20, 2000),
             "genome": _log_int(rng, 500_000, 8_000_000), "records": rng.randrange(1, 9)}
        c["mmin"] = _log_int(rng, 40, 200)
        c["mmax"] = _log_int(rng, c["mmin"], 400)
    c["shape_seed"] = ss
    return c


# ---------------------------------------------------------------------------
# Sizes of a case (from the case alone)
# ---------------------------------------------------------------------------
def _shape(case):
    """Profile lengths and read lengths."""
    rng = np.random.default_rng([case["shape_seed"], 17])

    def log_ints(lo, hi, n):
        return np.exp(rng.uniform(math.log(lo), math.log(hi), n)).round().astype(int)

    kind = case["kind"]
    if kind in ("score", "search"):
        return log_ints(case["mmin"], case["mmax"], case["profiles"]), log_ints(case["lmin"], case["lmax"], case["reads"])
    if kind == "windows":
        return log_ints(case["mmin"], case["mmax"], case["profiles"]), np.zeros(0, int)
    ms = np.array([case["m"]])
    if kind == "calibrate":
        return ms, np.full(case["trials"], case["length"] + 100)
    if kind == "align":
        return ms, np.full(case["reads"], 3 * case["m"] + 2 * case["flank"])
    return ms, log_ints(case["lmin"], case["lmax"], case["reads"])


def work(case):
    ms, ls = _shape(case)
    kind = case["kind"]
    if kind == "windows":  # a hit's window: the hit and 3 profile lengths on each side
        m = float(ms.mean())
        nt = case["hits"] * (6 * m + 90)
        return {"bytes": nt * 0.375 + case["hits"] * 140.0, "flops": 25.0 * nt * (m + 1)}
    strands = case.get("strands", 2 if kind == "align" else 1)
    nt = float(ls.sum()) * strands
    pairs = len(ms) * len(ls) * strands
    cells = float((ms + 1).sum()) * nt
    prof = float((ms + 1).sum()) * 144
    # flops of one cell: backward 24, forward with the mid product 28 (FP32); filter 25; gradient 67 and
    # posteriors 49 (FP64)
    if kind == "score" and case["filter"] or kind == "search":
        return {"bytes": nt * 0.375 + prof + pairs * 40.0, "flops": 25 * cells}
    if kind == "grad":
        return {"bytes": nt + prof + 8.0 * pairs + 288.0 * (case["m"] + 1), "flops": 67 * cells}
    if kind == "posterior":
        return {"bytes": nt + prof + 12.0 * nt + 8.0 * pairs * (case["m"] + 2), "flops": 49 * cells}
    return {"bytes": nt * (1 if kind == "align" else 0.375) + prof + pairs * 40.0, "flops": 52 * cells}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
_AA = "ACDEFGHIKLMNPQRSTVWY"
_CODE = {"A": "GCT GCC GCA GCG", "R": "CGT CGC CGA CGG AGA AGG", "N": "AAT AAC", "D": "GAT GAC", "C": "TGT TGC",
         "Q": "CAA CAG", "E": "GAA GAG", "G": "GGT GGC GGA GGG", "H": "CAT CAC", "I": "ATT ATC ATA",
         "L": "TTA TTG CTT CTC CTA CTG", "K": "AAA AAG", "M": "ATG", "F": "TTT TTC", "P": "CCT CCC CCA CCG",
         "S": "TCT TCC TCA TCG AGT AGC", "T": "ACT ACC ACA ACG", "W": "TGG", "Y": "TAT TAC", "V": "GTT GTC GTA GTG"}
_CODONS = [_CODE[a].split() for a in _AA]
_NCOD = np.array([len(c) for c in _CODONS])
_CODON_NT = np.zeros((20, 6, 3), np.uint8)  # 2-bit bases of each amino acid's codons
_CODON_AA = np.full(64, 23, np.int64)       # amino acid of each codon, 23 = stop
for _a, _cs in enumerate(_CODONS):
    for _k, _c in enumerate(_cs):
        _b = ["ACGT".index(x) for x in _c]
        _CODON_NT[_a, _k] = _b
        _CODON_AA[16 * _b[0] + 4 * _b[1] + _b[2]] = _a
_ACGT = np.frombuffer(b"ACGT", np.uint8)
_INS1, _INS2, _DEL1, _DEL2 = (np.float32(x) for x in (0.0171, 0.0018, 0.0328, 0.0083))  # default frameshift rates
_STOP, _BG_STOP = 0.0005, 0.046875


class _Profile:
    """A profile as a program holds it: emission rows, Params rows, background (float32)."""

    def __init__(self, rng, M):
        match = np.maximum(rng.dirichlet(np.full(20, 0.5), size=M), 1e-12)
        self.match = match / match.sum(1, keepdims=True)
        self.M = M
        mm, mi, md, ii, dd = 0.9 / 0.96, 0.03 / 0.96, 0.03 / 0.96, 0.4, 0.4
        keep = 1.0 - float(_INS1) - float(_INS2) - float(_DEL1) - float(_DEL2)
        alpha, delta = mi * keep, np.full(M, md * keep)
        delta[M - 1] = 0.0
        eps = np.full(M + 1, dd)
        eps[0] = 0.0
        p = np.zeros((M + 2, 11))
        p[:M + 1, 0], p[:M + 1, 1], p[:M + 1, 2], p[:M + 1, 3] = alpha * (1 - ii), _INS1, _INS2, ii
        p[:M, 6], p[:M, 7], p[:M, 8] = delta * (1 - eps[1:]), _DEL1, _DEL2
        p[:M, 9] = eps[:M] * (1 - eps[1:]) / (1 - eps[:M])
        p[:M, 10] = 1 - alpha - float(_INS1) - float(_INS2) - delta - float(_DEL1) - float(_DEL2)
        self.params = p.astype(np.float32)
        bg = np.exp(np.log(np.maximum(self.match, 1e-6)).mean(0))
        bg = bg / bg.sum() * (1 - _BG_STOP) / _NCOD
        v = np.zeros((M + 1, 29))
        v[:M, 4:24] = (1 - _STOP) * self.match / _NCOD
        v[M, 4:24] = bg
        v[:M, 24], v[:M, 25], v[:M, 26], v[:M, 27] = v[:M, 5], v[:M, 12], 1 / 64, _STOP / 3
        self.values = v.astype(np.float32)
        b = np.zeros(29)
        b[4:24], b[26], b[27] = bg, 1 / 64, _BG_STOP / 3
        self.bg = b.astype(np.float32)

    def homolog(self, rng, max_nt):
        """2-bit bases of a reverse-translated stretch of the profile with +-1 nt frameshifts."""
        n = min(self.M, max(1, max_nt // 3))
        at = int(rng.integers(0, self.M - n + 1))
        cdf = np.cumsum(self.match[at:at + n], axis=1)
        aa = np.minimum((rng.random((n, 1)) * cdf[:, -1:] > cdf).sum(1), 19)
        nt = _CODON_NT[aa, (rng.random(n) * _NCOD[aa]).astype(int)].reshape(-1)
        u = rng.random(len(nt))
        times = np.where(u < 0.0025, 0, np.where(u > 0.9975, 2, 1))
        return np.repeat(nt, times)[:max_nt]


def _reads(rng, case, ls, profiles, fraction):
    """2-bit reads; `fraction` of them carry a homolog of one of the profiles."""
    pick = np.random.default_rng([case["shape_seed"], 29])
    out = []
    for L in ls:
        gc = pick.uniform(0.4, 0.6)
        r = np.where(rng.random(L) < gc, rng.integers(1, 3, L), 3 * rng.integers(0, 2, L)).astype(np.uint8)
        p = profiles[int(pick.integers(0, len(profiles)))]
        share, where, flip, carries = pick.uniform(0.3, 1.0), pick.random(), pick.random() < 0.5, pick.random() < fraction
        if carries and L >= 12:
            h = p.homolog(rng, max(9, int(share * L)))
            if flip and fraction < 1:
                h = 3 - h[::-1]
            o = int(where * (L - len(h)))
            r[o:o + len(h)] = h
        out.append(r)
    return out


def _strands(reads, strands):
    return reads if strands == 1 else [s for r in reads for s in (r, 3 - r[::-1])]


def _pack(reads):
    words = []
    for r in reads:
        w = np.zeros((len(r) + 15) // 16 * 16, np.uint32)
        w[:len(r)] = r
        words.append((w.reshape(-1, 16) << (2 * np.arange(16, dtype=np.uint32))).sum(1, dtype=np.uint32))
    return np.concatenate(words)


def _pair_array(seqs, pids, ratio=-2.0):
    a = np.zeros(len(seqs), np.dtype([("seq", "<i4"), ("profile", "<i4"), ("min_prob_ratio", "<f4")]))
    a["seq"], a["profile"], a["min_prob_ratio"] = seqs, pids, ratio
    return (F.Pair * len(a)).from_buffer(a)


def _inputs(case, seed):
    """(profiles, 2-bit sequences) of a case: what prepare and exact both start from."""
    rng = np.random.default_rng([seed, case["shape_seed"]])
    ms, ls = _shape(case)
    profiles = [_Profile(rng, int(m)) for m in ms]
    kind = case["kind"]
    if kind in ("calibrate", "windows"):
        return profiles, []
    if kind == "align":
        reads = []
        for _ in ls:
            flanks = rng.integers(0, 4, (2, case["flank"])).astype(np.uint8)
            reads.append(np.concatenate([flanks[0], profiles[0].homolog(rng, 3 * case["m"]), flanks[1]]))
        return profiles, _strands(reads, 2)
    fraction = 1.0 if kind == "grad" else 0.5 if kind == "posterior" else 0.1 if len(ls) > 16 else 0.34
    return profiles, _strands(_reads(rng, case, ls, profiles, fraction), case.get("strands", 1))


_RESULT = np.dtype([("mid_m", "<f4"), ("mid_e", "<i4"), ("filter_m", "<f4"), ("filter_e", "<i4"), ("mid_ln", "<f8"),
                    ("filter_ln", "<f8"), ("filter_f", "<f4"), ("flags", "<i4")])
_WINDOW = np.dtype([("record", "<i4"), ("strand", "<i4"), ("start", "<i8"), ("end", "<i8"), ("profile_off", "<i8"),
                    ("profile_len", "<i4"), ("profile", "<i4")])
_CONTIG = np.dtype([("record", "<i4"), ("start", "<i4"), ("length", "<i4"), ("seq_id", "<i4"), ("name_off", "<i8"),
                    ("name_len", "<i4"), ("seq_id_rc", "<i4"), ("letter_off", "<i8"), ("record_length", "<i4"),
                    ("pipeline", "<i4"), ("w_start", "<i8"), ("w_end", "<i8"), ("true_length", "<i8"),
                    ("profile_off", "<i8"), ("profile_len", "<i4"), ("pad", "<i4")])
_ALIGNMENT = np.dtype([("pair", "<i4"), ("m", "<f4"), ("e", "<i4"), ("_", "<i4"), ("ln", "<f8"), ("anchor1", "<i4"),
                       ("anchor2", "<i4"), ("seg_begin", "<i8"), ("seg_count", "<i4"), ("pad", "<i4")])


class _State:
    pass


def _genome(case, rng, profiles):
    """(FASTA text, record names, lengths, hit rows of the prefilter); where the hits are comes from the case."""
    where = np.random.default_rng([case["shape_seed"], 41])
    per = case["genome"] // case["records"]
    names = ["chr%d" % (k + 1) for k in range(case["records"])]
    parts = []
    for name in names:
        seq = _ACGT[rng.integers(0, 4, per)]
        for _ in range(3):
            a = int(where.integers(0, per - 200))
            seq[a:a + int(where.integers(1, 200))] = ord("N")
        rows = per // 60
        body = np.full((rows, 61), ord("\n"), np.uint8)
        body[:, :60] = seq[:rows * 60].reshape(rows, 60)
        parts.append(b">" + name.encode() + b"\n" + body.tobytes() + seq[rows * 60:].tobytes() + b"\n")
    n = case["hits"]
    r, q = where.integers(0, case["records"], n), where.integers(0, len(profiles), n)
    f = np.array([1, 2, 3, -1, -2, -3])[where.integers(0, 6, n)]
    c, h = where.integers(1, per // 3 - 1, n), where.integers(0, 60, n)
    rows = ["PF%05d.1\t%s_frame=%+d\t45.0\t90\t10\t1\t1\t30\t%d\t%d\t1e-10\t55.0\n"
            % (q[k], names[r[k]], f[k], max(1, c[k] - h[k]), c[k] + h[k]) for k in range(n)]
    return b"".join(parts), names, [per] * len(names), "".join(rows).encode()


def prepare(case, seed):
    s = _State()
    kind = s.kind = case["kind"]
    profiles, seqs = _inputs(case, seed)
    s.ctx = d.Context(device=0)
    s.pids = [s.ctx.add_profile(p.values, p.params, p.bg) for p in profiles]
    n, P = len(seqs), len(profiles)
    if kind in ("score", "search"):
        s.lens = np.array([len(x) for x in seqs], np.int64)
        s.ascii = [_ACGT[x].tobytes() for x in seqs] if n <= 2 else None
        s.words = None if s.ascii else _pack(seqs)
        s.pairs = _pair_array(np.tile(np.arange(n, dtype=np.int32), P), np.repeat(np.array(s.pids, np.int32), n))
        if kind == "search":
            s.gate = np.full(P, case["gate"], np.float32)
            s.mode = F.MODE_MID
        else:
            s.mode = (F.MODE_FILTER if case["filter"] else F.MODE_MID) | (F.MODE_GRAPH if n > 2 else 0)
            if case["tune"]:  # once per program, on some of its reads
                s.ctx.add_packed(s.words, s.lens) if s.words is not None else s.ctx.add_dna(s.ascii)
                some = list(range(0, n, max(1, n // 200)))
                s.ctx.autotune(some * P, [p for p in s.pids for _ in some])
                s.ctx.clear_sequences()
    elif kind == "calibrate":
        s.args = (s.pids[0], case["length"], 100, case["trials"])
    elif kind == "align":
        s.ascii = [_ACGT[x].tobytes() for x in seqs]
        s.pairs = _pair_array(np.arange(n, dtype=np.int32), np.full(n, s.pids[0], np.int32), case["gate"])
        s.results = (F.Result * n)()
        # every alignment of a pass, in arrays with room for any of them
        s.alignments, s.segments = np.zeros(256 * n, _ALIGNMENT), np.zeros((4096 * n, 3), np.int32)
        s.fields = {k: s.alignments[k] for k in _ALIGNMENT.names if k not in ("_", "pad")}
    elif kind in ("grad", "posterior"):
        # the reads stay in the context from step to step
        s.seqs = s.ctx.add_packed(_pack(seqs), [len(x) for x in seqs])
        if kind == "grad":
            s.ctx.adjoint_checkpoint(F.ADJ_CKPT_ON if case["ckpt"] else F.ADJ_CKPT_AUTO)
            s.profile = (profiles[0].values, profiles[0].params, profiles[0].bg)
    else:
        text, s.names, s.record_lens, s.hits = _genome(case, np.random.default_rng([seed, case["shape_seed"], 3]), profiles)
        s.ctx.genome_load(text)
        s.pnames, s.plens = ["PF%05d.1" % k for k in range(P)], [p.M for p in profiles]
        s.contigs = (F.Contig * (4 * case["hits"] + 16))()
    return s


def _fields(array, dtype, skip=("_", "pad")):
    a = np.frombuffer(array, dtype)
    return {k: a[k] for k in dtype.names if k not in skip}


def run(s):
    ctx, kind = s.ctx, s.kind
    if kind in ("score", "search"):
        ctx.clear_sequences()
        if s.ascii:
            ctx.add_dna(s.ascii)
        else:
            ctx.add_packed(s.words, s.lens)
        res = ctx.search_raw(s.pairs, s.gate, s.mode) if kind == "search" else ctx.score_pairs_raw(s.pairs, s.mode)
        return _fields(res, _RESULT)
    if kind == "calibrate":
        fit, mid, flt = ctx.estimate_k(*s.args, return_scores=True)
        return {"fit": np.array([fit["lambda"], fit["K"], fit["lambda_filter"], fit["K_filter"]]), "mid": mid, "filter": flt}
    if kind == "align":
        ctx.clear_sequences()
        ctx.add_dna(s.ascii)
        al, segs = ctx.align_raw(s.pairs, s.results)
        for to, got in ((s.alignments, np.frombuffer(al, _ALIGNMENT) if len(al) else ()), (s.segments, segs)):
            to[:len(got)] = got
            to[len(got):] = 0
        return {"results": _fields(s.results, _RESULT), "count": len(al), "alignments": s.fields, "segments": s.segments}
    if kind == "grad":
        ctx.set_profile(s.pids[0], *s.profile)  # a refinement step's new parameters
        logt, gp, ge = ctx.loglik_grad(s.seqs, s.pids[0])
        return {"log_t": logt, "grad_params": gp, "grad_emit": ge}
    if kind == "posterior":
        logt, tracks = ctx.posterior_summary(s.seqs, s.pids[0])
        return {"log_t": logt, "column": np.concatenate([t[0] for t in tracks]),
                "row": np.concatenate([t[1] for t in tracks]), "match": np.concatenate([t[2] for t in tracks])}
    ctx.clear_sequences()
    windows, malformed, dropped = d.windows_from_hits(s.hits, s.names, s.record_lens, s.pnames, s.plens)
    n = ctx.add_windows_raw(windows, s.contigs)
    con = np.frombuffer(s.contigs, _CONTIG, n)
    have = con["seq_id"] >= 0
    pid = np.array(s.pids, np.int32)[np.frombuffer(windows, _WINDOW)["profile"][con["record"][have]]]
    res = ctx.score_pairs_raw(_pair_array(con["seq_id"][have], pid), F.MODE_FILTER)
    return {"contigs": {k: con[k] for k in _CONTIG.names if k != "pad"}, "results": _fields(res, _RESULT),
            "malformed": malformed, "dropped": dropped}


# ---------------------------------------------------------------------------
# The same results in 64 bits, in plain torch: null model, then the backward
# and forward recurrences one antidiagonal at a time, all rows and reads of a
# profile at once.
# ---------------------------------------------------------------------------
def _codes(r):
    c = np.zeros(len(r), np.int64)
    v = r.astype(np.int64)
    c[:-2] = _CODON_AA[16 * v[:-2] + 4 * v[1:-1] + v[2:]]
    return c


def _null(codes, bg):
    """(prefix seeds, suffix seeds, per-base factor) of one read."""
    L = len(codes)
    single, double = float(_INS1 + _DEL2), float(_INS2 + _DEL1)
    keep, sn, dn = 1.0 - single - double, single * 0.25, double * 0.0625
    g = bg[codes]

    def prefix(b):
        p = np.zeros(L + 3)  # p[i + 3] = prefix[i] b^(i+1)
        for i in range(L):
            cod = p[i] * g[i - 2] * keep * b ** 3 if i >= 3 else b ** (i + 1) * (g[0] if i == 2 else 0.25 ** (i + 1)) / 3
            p[i + 3] = cod + (p[i + 2] * sn * b if i > 0 else 0.0) + (p[i + 1] * dn * b * b if i >= 2 else 0.0)
        return p

    p = prefix(4.0)
    tot = p[L + 2] + p[L + 1] * (1 - single) * 0.25 * 4 + p[L] * (1 - single - double) * 0.0625 * 16
    b = min(4.0 / tot ** (1.0 / L), 2.0 ** 120)
    p = prefix(b)[3:]
    s = np.zeros(L + 4)  # s[i] = suffix[i] b^(L-i)
    s[L] = 1.0
    for i in range(L - 1, -1, -1):
        dbl = s[i + 2] if i + 1 < L else 4.0 / b
        cod = s[i + 3] * b ** 3 * g[i] * keep if i + 2 < L else 0.5 * keep * 2.0 ** (1 - 2 * (L - i)) * b ** (L - i)
        s[i] = cod + s[i + 1] * b * sn + dbl * b * b * dn
    return p, s[1:L + 1], b


def _reference(profile, reads, gradient=False):
    """mid, filter and T of each read; with gradient: the sums over cells of the adjoint, per read rows x terms."""
    M, n = profile.M, len(reads)
    E = torch.zeros(M + 1, 26, dtype=torch.float64)
    E[:, :25] = torch.from_numpy(profile.values[:, 4:].astype(np.float64))
    bgv = np.zeros(26)
    bgv[:25] = profile.bg[4:]
    bgv[24] = 0.0
    Lm = max(len(r) for r in reads)
    pad = M + 8
    code = torch.full((n, Lm + 2 * pad), 24, dtype=torch.int64)
    pre, suf = (torch.zeros(n, Lm + 2 * pad, dtype=torch.float64) for _ in range(2))
    live = torch.zeros(n, Lm + 2 * pad, dtype=torch.bool)
    bases = []
    for k, r in enumerate(reads):
        c = _codes(r)
        a, z, b = _null(c, bgv)
        bases.append(b)
        L = len(c)
        code[k, pad:pad + L] = torch.from_numpy(c)
        pre[k, pad:pad + L], suf[k, pad:pad + L] = torch.from_numpy(a), torch.from_numpy(z)
        live[k, pad:pad + L] = True
    b = torch.tensor(bases, dtype=torch.float64)[:, None]
    s1, s2, sC = b / 4, b * b / 16, b ** 3
    q = torch.from_numpy(profile.params[:M + 1].astype(np.float64))
    a0, a1, a2, b0, d0, d1, d2, eps, enter = (q[:, k][None] for k in (0, 1, 2, 3, 6, 7, 8, 9, 10))
    A1, A2, D1, D2, EN = a1 * s1, a2 * s2, d1 * s2, d2 * s1, enter * sC
    rows = torch.arange(M + 1)
    bg = torch.from_numpy(bgv)
    zero = torch.zeros(n, M + 1, dtype=torch.float64)

    def up(x):    # row i takes row i+1's value
        return torch.cat([x[:, 1:], zero[:, :1]], 1)

    def down(x):  # row i takes row i-1's
        return torch.cat([zero[:, :1], x[:, :-1]], 1)

    D = Lm + M
    fw, h = [], [(zero, zero, zero)] * 4  # of the last four diagonals: W0, Z0, match term for the row above
    y = zero
    for t in range(D):
        j = t - rows + pad
        ok = live[:, j]
        c2 = code[:, j - 2]
        (_, _, x3), (w3, z3, _), (w2, _, _), (w1, _, _) = h
        Z = sC * bg[c2] * (a0 * w3 + b0 * z3)
        y0 = down(y)
        win = x3 + down(D1 * w3) + down(D2 * w2) + y0  # row i-1 at columns j-3, j-2, j-1 and its Y0 at j
        W = torch.where(ok, A1 * w1 + A2 * w2 + pre[:, j] + win + Z, zero)
        Z = torch.where(ok, Z, zero)
        y = torch.where(ok, d0 * W + eps * y0, zero)
        h = h[1:] + [(W, Z, down(EN * E[rows, code[:, j + 1]] * W))]
        fw.append((W, y, Z))
    out = {"mid": torch.zeros(n, dtype=torch.float64), "filter": torch.zeros(n, dtype=torch.float64),
           "T": torch.zeros(n, dtype=torch.float64)}
    if gradient:
        g = torch.zeros(9, n, M + 1, dtype=torch.float64)
        ge = torch.zeros(n, M + 1, 26, dtype=torch.float64)
        cell = torch.zeros(n, Lm + 2 * pad, dtype=torch.float64)
    hist = [(zero, zero, zero)] * 4
    for t in range(D - 1, -1, -1):
        j = t - rows + pad
        ok = live[:, j]
        c = code[:, j + 1]
        (W1, Y1, _), (W2, _, _), (W3, _, Z3), (W4, _, _) = hist
        yn, n1, n2, n3 = up(Y1), up(W2), up(W3), up(W4)
        e = E[rows, c]
        zbg = Z3 * bg[c]
        W = torch.where(ok, n3 * e * EN + yn * d0 + n2 * D1 + n1 * D2 + zbg * a0 * sC + W2 * A2 + W1 * A1 + suf[:, j], zero)
        Y = torch.where(ok, eps * yn + W, zero)
        Z = torch.where(ok, b0 * sC * zbg + W, zero)
        F0, FY, FZ = fw[t]
        out["mid"] = torch.maximum(out["mid"], (F0 * W).amax(1))
        seeded = W * pre[:, j]
        out["filter"] = torch.maximum(out["filter"], seeded.amax(1))
        out["T"] += seeded.sum(1)
        if gradient:
            below = down(fw[t - 1][1]) if t > 0 else zero  # Y0 of row i-1 at column j
            me = torch.where(ok, F0 * n3 * sC, zero)
            for k, v in enumerate((F0 * zbg * sC, F0 * W1 * s1, F0 * W2 * s2, FZ * zbg * sC, F0 * yn, F0 * n2 * s2,
                                   F0 * n1 * s1, below * yn, me * e)):
                g[k] += torch.where(ok, v, zero)
            ge.scatter_add_(2, c[:, :, None], (me * enter)[:, :, None])
            col = j[None].expand(n, -1)
            cell.scatter_reduce_(1, col, F0 * W, "amax")
        hist = [(W, Y, Z)] + hist[:3]
    if gradient:
        out.update(g=g, ge=ge, cell=cell[:, pad:])
    return out


_EXACT_CELLS = 2.0e7  # about 20 seconds


def exact(case, seed):
    kind = case["kind"]
    ms, ls = _shape(case)
    cells = float((ms + 1).sum()) * float(ls.sum()) * case.get("strands", 1)
    if kind not in ("score", "grad", "posterior") or cells > _EXACT_CELLS or len(ms) * (ls.max() + ms.max()) > 8000:
        return None
    profiles, seqs = _inputs(case, seed)
    if kind == "score":
        got = [_reference(p, seqs) for p in profiles]
        mid, flt = (torch.cat([x[k] for x in got]).log().numpy() for k in ("mid", "filter"))
        if not (np.isfinite(mid).all() and np.isfinite(flt).all()):
            return None
        if case["filter"]:
            return {"mid_m": None, "mid_e": None, "filter_m": None, "filter_e": None, "mid_ln": None, "filter_ln": flt,
                    "filter_f": np.exp(flt), "flags": None}
        return {"mid_m": None, "mid_e": None, "filter_m": None, "filter_e": None, "mid_ln": mid, "filter_ln": flt,
                "filter_f": None, "flags": None}
    p = profiles[0]
    r = _reference(p, seqs, gradient=True)
    T = r["T"]
    if not (torch.isfinite(T).all() and torch.isfinite(r["g"]).all() and torch.isfinite(r["cell"]).all()):
        return None
    if kind == "grad":
        gp = np.zeros((p.M + 2, 11))
        gp[:p.M + 1, [0, 1, 2, 3, 6, 7, 8, 9, 10]] = (r["g"] / T[None, :, None]).sum(1).T.numpy()
        return {"log_t": T.log().numpy(), "grad_params": gp, "grad_emit": (r["ge"][:, :, :25] / T[:, None, None]).sum(0).numpy()}
    match = r["g"][8] * torch.from_numpy(p.params[:p.M + 1, 10].astype(np.float64)) / T[:, None]
    column = np.concatenate([(r["cell"][k, :len(x)] / T[k]).numpy() for k, x in enumerate(seqs)])
    return {"log_t": T.log().numpy(), "column": column, "row": None, "match": match.reshape(-1).numpy()}

