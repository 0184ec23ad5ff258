"""What a user of this framework has it do, as cases that can be timed.

Each case is one pass through the public Python entry points on data as a
caller holds it: reads as packed codes in host memory (or a FASTQ file), a
scorer that already holds its panel.  The panel scorer takes host arrays and
returns host arrays, so a pass covers the whole call: packing, upload, the
device work, the results back.

Sizes follow the benchmark's workloads (a 164-reference panel of 70-180 nt,
reads of about 110 nt, 2 x 150 nt pairs, a panel of 300-1000 nt references,
serving requests of 1-1000 reads) and the tests' ranges (reads to 5000 nt,
schemes that leave the int16 lanes).
"""
import math
import os
import tempfile

import numpy as np
import torch

from eschalign_b200 import GpuScorer, Mode, Scoring, adapter, synth
from eschalign_b200 import bam as EB
from eschalign_b200.server import Server

MODES = {"local": Mode.LOCAL, "semiglobal": Mode.SEMIGLOBAL}


def _case(name, kind, reads, refs, ref_lo, ref_hi, **kw):
    c = {"kind": kind, "reads": reads, "refs": refs, "ref_lo": ref_lo, "ref_hi": ref_hi,
         "mode": "local", "scheme": "2,-1,-10,-1", "both": True, "median": 110, "sigma": 0.4,
         "read_lo": 20, "read_hi": 1000, "wild": 0.0, "batches": 1, "rows": False}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one read against a tRNA-sized panel: an interactive query, all latency
        _case("single-read", "score", 1, 164, 70, 180),
        # a small ragged request with a few ambiguous bases, semi-global
        _case("small-request", "score", 61, 93, 60, 220, mode="semiglobal", sigma=0.5,
              read_hi=400, wild=0.01),
        # a burst of client requests of 1-1000 reads on a serving queue with
        # one scorer per mode
        _case("served-requests", "serve", 24, 164, 70, 180),
        # the small benchmark sample: 10 000 reads of 60-200 nt, one strand
        _case("sample-forward", "score", 10_000, 164, 70, 180, both=False, sigma=0.0,
              read_lo=60, read_hi=200),
        # the unpaired run's scoring: batches of 50 000 reads through the
        # feeder, both strands, local (the headline workload)
        _case("feeder-local", "score", 100_000, 164, 70, 180, batches=2),
        # whole score rows for a caller that ranks on its own, another scheme
        _case("rows-semiglobal", "score", 20_011, 164, 70, 180, mode="semiglobal",
              scheme="1,-1,-2,-1", rows=True),
        # the paired run's scoring: 2 x 150 nt mates with adapter read-through
        _case("pairs", "pairs", 50_000, 164, 70, 180, mode="semiglobal", batches=2),
        # a large panel of long references that does not fit shared memory,
        # few reads of 50-1000 nt
        _case("large-panel", "score", 300, 3001, 300, 1000, sigma=0.0, read_lo=50),
        # full-length transcripts: reads of 1100-5000 nt that run in passes
        _case("long-reads", "score", 257, 48, 400, 3000, sigma=0.0, read_lo=1100,
              read_hi=5000),
        # a finely scaled scheme whose scores leave the int16 lanes
        _case("wide-scores", "score", 10_007, 164, 70, 180, scheme="100,-100,-200,-30"),
        # coordinates and CIGARs of reads' winners (here: one reference a read)
        _case("traceback", "align", 100_000, 164, 70, 180, mode="semiglobal"),
        # the whole command-line run: FASTQ in, mapped, records, BAM out
        _case("fastq-to-bam", "bam", 30_000, 164, 70, 180),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    c = _draw(rng)
    while work(c)["flops"] > 4e12:  # no dearer than the largest listed ones
        c["reads"] //= 2
    return c


def _draw(rng):
    kind = rng.choice(["score"] * 7 + ["serve", "pairs", "pairs", "align", "align", "bam"])
    mode = rng.choice(["local", "local", "semiglobal"])
    scheme = rng.choice(["2,-1,-10,-1"] * 3 + ["1,-1,-2,-1", "3,-2,-5,-2"])
    refs, lo = _log(rng, 5, 400), rng.randint(40, 120)
    panel = (refs, lo, lo + rng.randint(10, 200))
    kw = {"mode": mode, "scheme": scheme, "median": rng.randint(60, 200),
          "sigma": rng.choice([0.0, 0.3, 0.5]), "read_lo": rng.randint(1, 40),
          "read_hi": rng.choice([300, 1000]), "wild": rng.choice([0.0, 0.0, 0.002])}
    if kind == "serve":
        return _case(None, kind, rng.randint(4, 30), *panel, **kw)
    if kind == "pairs":
        return _case(None, kind, _log(rng, 50, 40_000), min(refs, 200), *panel[1:],
                     batches=rng.choice([1, 2, 3]), **kw)
    if kind == "align":
        return _case(None, kind, _log(rng, 10, 100_000), *panel, **kw)
    if kind == "bam":
        return _case(None, kind, _log(rng, 500, 30_000), *panel, **kw)
    shape = rng.random()
    if shape < 0.15:  # long reads
        kw.update(sigma=0.0, read_lo=rng.randint(500, 1200), read_hi=rng.randint(2000, 5000))
        return _case(None, kind, _log(rng, 8, 200), rng.randint(5, 48), 300,
                     rng.randint(800, 3000), both=rng.random() < 0.7, **kw)
    if shape < 0.3:  # a large panel
        return _case(None, kind, _log(rng, 4, 250), _log(rng, 500, 3000), 300, 1000,
                     both=rng.random() < 0.7, **dict(kw, sigma=0.0))
    if shape < 0.4:  # wide scores
        return _case(None, kind, _log(rng, 50, 10_000), min(refs, 164), *panel[1:],
                     **dict(kw, scheme="100,-100,-200,-30"))
    reads = _log(rng, 1, 60_000)
    return _case(None, kind, reads, *panel, both=rng.random() < 0.7,
                 batches=rng.choice([1, 1, 3]) if reads > 1000 else 1,
                 rows=reads < 20_000 and rng.random() < 0.3, **kw)


# ---------------------------------------------------------------- inputs
def _lengths(case, rng, n):
    if case["sigma"] == 0.0:
        return rng.integers(case["read_lo"], case["read_hi"] + 1, n)
    return synth.lognormal_lengths(rng, n, case["median"], case["sigma"], case["read_lo"],
                                   case["read_hi"])


def _make(case, seed):
    """(panel, reads) of a case: uniform references (a case's lengths are its
    own, the bases the seed's), nine in ten reads cut from one and mutated,
    the rest random."""
    lens = np.random.default_rng(case["refs"]).integers(case["ref_lo"], case["ref_hi"] + 1,
                                                        case["refs"])
    rng = np.random.default_rng([seed, 1])
    refs = [synth.random_bases(rng, int(m)) for m in lens]
    rng = np.random.default_rng([seed, 2])
    n = case["reads"]
    if case["kind"] == "pairs":
        return refs, synth.pairs_c4(refs, n=n, seed=seed)[0]
    if case["kind"] == "serve":
        n = int(_request_sizes(case).sum())
    reads = synth.mixed_reads(rng, refs, _lengths(case, rng, n), 0.9, 0.08, 0.02, 0.01)
    if case["wild"]:
        reads.codes[rng.random(reads.codes.size) < case["wild"]] = 4
    return refs, reads


def _request_sizes(case):
    rng = np.random.default_rng([case["refs"], case["reads"]])
    return np.exp(rng.uniform(0, math.log(1000), case["reads"])).astype(np.int64)


def _cut(case, reads, per=1):
    """The case's reads as its batches (`per` reads stay together)."""
    n, k = len(reads) // per, case["batches"]
    return [reads.slice(per * (n * b // k), per * (n * (b + 1) // k)) for b in range(k)]


def _fastq(path, reads, seed):
    rng = np.random.default_rng([seed, 4])
    letters = np.frombuffer(b"ACGTN", np.uint8)[np.minimum(reads.codes, 4)].tobytes()
    qual = rng.integers(35, 74, reads.codes.size, dtype=np.uint8).tobytes()
    with open(path, "wb") as fh:
        for k, (o, n) in enumerate(zip(reads.off.tolist(), reads.lens.tolist())):
            fh.write(b"@read%d\n%b\n+\n%b\n" % (k, letters[o:o + n], qual[o:o + n]))


def prepare(case, seed):
    refs, reads = _make(case, seed)
    kind = case["kind"]
    scoring = Scoring.parse(case["scheme"])
    st = {"case": case}
    if kind == "serve":
        st["scorers"] = [GpuScorer(refs, scoring, m) for m in (Mode.LOCAL, Mode.SEMIGLOBAL)]
        st["server"] = Server(st["scorers"])
        ends = np.cumsum(_request_sizes(case))
        st["requests"] = [(k % 2, reads.slice(int(a), int(b)))
                          for k, (a, b) in enumerate(zip([0, *ends[:-1]], ends))]
        return st
    st["scorer"] = GpuScorer(refs, scoring, MODES[case["mode"]])
    if kind == "score":
        st["batches"] = _cut(case, reads)
    elif kind == "pairs":
        st["batches"] = _cut(case, reads, per=2)
        st["adapters"] = adapter.config()
    elif kind == "align":
        rng = np.random.default_rng([seed, 5])
        st["reads"] = reads
        st["jobs"] = np.stack([np.arange(len(reads)), rng.integers(0, len(refs), len(reads)),
                               rng.integers(0, 2, len(reads))], axis=1).astype(np.uint32)
    else:
        st["dir"] = tempfile.TemporaryDirectory()
        st["fastq"] = os.path.join(st["dir"].name, "reads.fastq")
        st["bam"] = os.path.join(st["dir"].name, "out.bam")
        _fastq(st["fastq"], reads, seed)
        st["names"] = [f"ref{k}" for k in range(len(refs))]
        st["letters"] = [np.frombuffer(b"ACGTN", np.uint8)[r].tobytes() for r in refs]
    return st


def _ints(a):
    """A record array as rows of 32-bit integers."""
    return a.view(np.int32).reshape(a.size, -1)


def _room(a, n):
    """`a` at the start of n zeroes: how many words there are depends on the reads."""
    out = np.zeros(n, a.dtype)
    out[:a.size] = a
    return out


def _scores(res):
    out = {"results": _ints(res.results), "ties": res.ties}
    if res.rows is not None:
        out["rows"] = res.rows
    return out


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "score":
        g, kw = st["scorer"], {"both_strands": case["both"], "full_rows": case["rows"]}
        if case["batches"] == 1:
            return _scores(g.score_batch(st["batches"][0], **kw))
        return [_scores(r) for r in g.score_batches(st["batches"], **kw)]
    if kind == "serve":
        sv = st["server"]
        tickets = [sv.submit(slot, reads, both_strands=True) for slot, reads in st["requests"]]
        return [_scores(sv.wait(t, 60_000)[0]) for t in tickets]
    if kind == "pairs":
        return [{"pairs": _ints(r.pairs), "pair_ties": r.pair_ties, "mates": _ints(r.mates.results),
                 "mate_ties": r.mates.ties, "adapters": r.adapters}
                for r in st["scorer"].score_pair_batches(st["batches"], st["adapters"],
                                                         min_score=20)]
    if kind == "align":
        a = st["scorer"].align(st["reads"], st["jobs"])
        return {"records": _ints(a.records), "ops": _room(a.ops, 64 * len(a))}
    EB.align_bam(st["scorer"], st["fastq"], st["bam"], st["names"], st["letters"],
                 both_strands=True, secondary=True)
    return _room(np.fromfile(st["bam"], dtype=np.uint8), (1 << 20) + 1000 * case["reads"])


def work(case):
    """Cells need about 12 integer operations each (two adds and a maximum
    for either gap state, an add and two or three maxima for the cell); the
    bytes are the reads, the panel and the results, once."""
    if case["kind"] == "pairs":
        n, mean = 2 * case["reads"], 110.0  # 150 nt less the adapter
    else:
        n = case["reads"]
        mean = case["median"] * math.exp(case["sigma"] ** 2 / 2)
        if case["sigma"] == 0.0:
            mean = (case["read_lo"] + case["read_hi"]) / 2
        if case["kind"] == "serve":
            n = int(n * 999 / math.log(1000))
    ref = (case["ref_lo"] + case["ref_hi"]) / 2
    strands = 2 if case["both"] or case["kind"] == "pairs" else 1
    bases = n * mean
    panel = case["refs"] * ref
    if case["kind"] == "align":
        return {"bytes": bases + panel + n * (12 + 40) + 16 * n, "flops": 12 * bases * ref}
    out = n * (16 + 4 * 8)
    if case["rows"]:
        out += 4 * n * strands * case["refs"]
    if case["kind"] == "bam":  # names and qualities in, records out
        bases, out = 2 * bases, 2 * bases
    return {"bytes": bases + panel + out, "flops": 12 * n * mean * strands * panel}


# ---------------------------------------------------------------- 64 bits
def _gotoh(q, qn, r, rn, scoring, local):
    """Scores of every query (rows of q, lengths qn) against every reference
    (rows of r, lengths rn) by anti-diagonals, in 64-bit integers."""
    neg = -(1 << 40)
    nq, n = q.shape
    nr, m = r.shape
    dev = q.device
    i = torch.arange(1, n + 1, device=dev)
    full = lambda v: torch.full((nq, nr, n + 1), v, dtype=torch.int64, device=dev)  # noqa: E731
    h1, h2, e, f = full(0), full(0), full(neg), full(neg)
    best = torch.full((nq, nr), 0 if local else neg, dtype=torch.int64, device=dev)
    rows_ok = i[None, :] <= qn[:, None]
    for d in range(2, n + m + 1):
        j = d - i
        on = (j >= 1) & (j <= m)
        x = r[:, (j - 1).clamp(0, m - 1)]
        match = (q[:, None, :] == x[None]) | (q[:, None, :] == 4) | (x[None] == 4)
        s = torch.where(match, scoring.match_score, scoring.mismatch)
        e2 = torch.maximum(e[..., 1:] + scoring.gap_extend, h1[..., 1:] + scoring.gap_open)
        f2 = torch.maximum(f[..., :-1] + scoring.gap_extend, h1[..., :-1] + scoring.gap_open)
        h = torch.maximum(torch.maximum(h2[..., :-1] + s, e2), f2)
        if local:
            h = h.clamp(min=0)
        cols_ok = on[None, :] & (j[None, :] <= rn[:, None])
        ok = rows_ok[:, None, :] & cols_ok[None]
        if not local:
            ok = ok & ((i[None, :] == qn[:, None])[:, None, :] | (j[None, :] == rn[:, None])[None])
        best = torch.maximum(best, torch.where(ok, h, neg).amax(-1))
        h2 = h1
        h1 = full(0)
        h1[..., 1:] = torch.where(on, h, 0)  # the zero border above row 1 and at column 0
        e, f = full(neg), full(neg)
        e[..., 1:] = torch.where(on, e2, neg)
        f[..., 1:] = torch.where(on, f2, neg)
    return best


def _padded(seqs, dev):
    n = max(s.size for s in seqs)
    a = np.full((len(seqs), n), 9, np.int64)
    for k, s in enumerate(seqs):
        a[k, :s.size] = s
    return torch.from_numpy(a).to(dev), torch.tensor([s.size for s in seqs], device=dev)


def exact(case, seed):
    """Scores are whole numbers; the small scoring cases are given here from
    plain 64-bit integer arithmetic, the rest would take too long."""
    if case["kind"] != "score" or case["batches"] != 1 or case["scheme"] == "100,-100,-200,-30" \
            or case["reads"] * case["refs"] > 60_000 or case["read_hi"] * case["ref_hi"] > 500_000:
        return None
    refs, reads = _make(case, seed)
    scoring = Scoring.parse(case["scheme"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rc = lambda s: np.where(s == 4, 4, 3 - s.astype(np.int64))[::-1]  # noqa: E731
    fwd = reads.list()
    seqs = fwd + [rc(s) for s in fwd] if case["both"] else fwd
    r, rn = _padded(refs, dev)
    rows = []
    per = max(1, int(2e7 / (case["refs"] * case["read_hi"])))
    for k in range(0, len(seqs), per):
        q, qn = _padded(seqs[k:k + per], dev)
        rows.append(_gotoh(q, qn, r, rn, scoring, case["mode"] == "local").cpu().numpy())
    rows = np.concatenate(rows)
    n, cap = len(fwd), 8
    results = np.zeros((n, 4), np.int32)
    ties = np.full((n, cap), 0xFFFFFFFF, np.uint32)
    for k in range(n):
        # candidates in order: reference by reference, forward before reverse
        cand = np.stack([rows[k], rows[n + k]], 1).ravel() if case["both"] else rows[k]
        best = cand.max()
        at = np.nonzero(cand == best)[0] * (1 if case["both"] else 2)
        rest = cand[cand != best]
        results[k] = (best, rest.max() if rest.size else -2**31, at.size, 2 * (at.size > cap))
        ties[k, :min(cap, at.size)] = at[:cap]
    out = {"results": results, "ties": ties}
    if case["rows"]:
        out["rows"] = rows.astype(np.int32)
    return out
