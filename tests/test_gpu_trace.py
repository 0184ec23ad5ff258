"""Traceback of winners on the CUDA path (esg_align_*) against the oracle.

Every job's score, coordinates and CIGAR must equal scalar::align
(crates/eschalign/src/scalar.rs:182-364, restated in oracle/esg_align.c):
the same end cell (first maximum of a column-major scan) and the same path
(diagonal, then insertion, then deletion; extending inside a gap; local mode
stopping at the first zero cell) -- not merely an optimal one."""
import numpy as np
import pytest

from eschalign_b200 import GpuScorer, Mode, Scoring, encode, synth
from tests.helpers import SCHEMES, Rng, fixture_panel, fixture_reads, golden, random_panel, \
    random_seq, reads_for, revcomp

pytestmark = pytest.mark.gpu


def check(oracle, g, reads, panel, jobs, scoring, local, what):
    got = g.align(reads, jobs)
    for k, (rd, ref, rev) in enumerate(jobs):
        q = revcomp(reads[rd]) if rev else reads[rd]
        want, wops = oracle.align(q, panel[ref], scoring, local)
        r = got.records[k]
        fields = ("score", "query_start", "query_end", "ref_start", "ref_end")
        assert tuple(int(r[f]) for f in fields) == tuple(int(want[f]) for f in fields), \
            (what, k, rd, ref, rev, r, want)
        assert list(got.ops_of(k)) == list(wops), (what, k, got.cigar(k), oracle.cigar_string(wops))
    return got


def test_trace_golden_cases(oracle):
    """The 192 parasail golden cases, each read against its own reference."""
    by = {}
    for c in golden()["cases"]:
        by.setdefault((c["mode"], tuple(c["scheme"])), []).append(c)
    for (mode, scheme), cases in by.items():
        for c in cases:
            q, r = encode(c["query"]), encode(c["reference"])
            with GpuScorer([r], Scoring(*scheme), Mode.LOCAL if mode == "local"
                           else Mode.SEMIGLOBAL) as g:
                got = check(oracle, g, [q], [r], [(0, 0, 0)], scheme, mode == "local",
                            c["name"])
                rec = got.records[0]
                assert (int(rec["query_start"]), int(rec["query_end"]), int(rec["ref_start"]),
                        int(rec["ref_end"])) == (c["query_start"], c["query_end"],
                                                 c["ref_start"], c["ref_end"])


@pytest.mark.parametrize("mode", [Mode.LOCAL, Mode.SEMIGLOBAL])
def test_trace_random_panel_all_jobs(oracle, mode):
    """Every (read, reference, strand) of a ragged 30-ref panel, five
    schemes: tiles of many jobs, each on its own reference."""
    rng = Rng(0x5EED_0701)
    letters = random_panel(rng, 30, 20, 260)
    panel = [encode(s) for s in letters]
    reads = reads_for(rng, letters, 25) + [np.zeros(0, np.uint8), encode("A")]
    jobs = [(i, r, v) for i in range(len(reads)) for r in range(len(panel)) for v in (0, 1)]
    for scoring in SCHEMES:
        with GpuScorer(panel, Scoring(*scoring), mode) as g:
            got = check(oracle, g, reads, panel, jobs, scoring, mode == Mode.LOCAL,
                        f"{mode.label} {scoring}")
            empty = [k for k, (i, _, _) in enumerate(jobs) if reads[i].size == 0]
            assert all(got.records[k]["score"] == 0 and got.records[k]["n_ops"] == 0
                       for k in empty)


def test_trace_long_reads_in_passes(oracle):
    """Reads over 32 stripes (512 nt) run alone in passes; up to 2500 nt
    against 700-900 nt references, both modes."""
    rng = Rng(0x5EED_0702)
    letters = random_panel(rng, 4, 700, 200)
    panel = [encode(s) for s in letters]
    reads = []
    for n in (513, 700, 1024, 1600, 2500):
        body = letters[n % 4]
        s = (body * 4)[:n]
        reads.append(encode(s))
    reads.append(encode(random_seq(rng, 900, 0.0)))
    jobs = [(i, r, v) for i in range(len(reads)) for r in (0, 3) for v in (0, 1)]
    for mode in (Mode.LOCAL, Mode.SEMIGLOBAL):
        with GpuScorer(panel, Scoring(2, -1, -10, -1), mode) as g:
            check(oracle, g, reads, panel, jobs, (2, -1, -10, -1), mode == Mode.LOCAL,
                  f"long {mode.label}")


def test_trace_wildcards_on_fixture_panel(oracle):
    """The ambiguous tRNA panel (wildcards in the references) and the
    fixture reads."""
    panel = fixture_panel("trna_ambiguous")
    reads = fixture_reads()
    jobs = [(i, r, 0) for i in range(len(reads)) for r in range(0, len(panel), 3)]
    for mode in (Mode.LOCAL, Mode.SEMIGLOBAL):
        with GpuScorer(panel, Scoring(), mode) as g:
            check(oracle, g, reads, panel, jobs, (2, -1, -10, -1), mode == Mode.LOCAL,
                  f"trna {mode.label}")


def test_trace_winners_of_a_scored_batch(oracle):
    """The flow of map_reads_scored: score a C2 sample, then trace each
    read's first tie straight from the batch's reads on the device."""
    refs = synth.panel_tiles()
    reads = synth.reads_c2(refs, n=1500)
    with GpuScorer(refs, Scoring(), Mode.LOCAL) as g:
        b = g.submit(g.prepare(reads.tuple(), both_strands=True))
        res = g.finish(b, keep=True)
        jobs = [(k, int(res.ties[k, 0]) >> 1, int(res.ties[k, 0]) & 1)
                for k in range(len(reads)) if res.results["n_tied"][k] > 0]
        got = g.align_batch(b, jobs)
        b.free()
    rl = reads.list()
    for k, (rd, ref, rev) in enumerate(jobs):
        q = revcomp(rl[rd]) if rev else rl[rd]
        want, wops = oracle.align(q, refs[ref], (2, -1, -10, -1), True)
        rec = got.records[k]
        assert int(rec["score"]) == int(res.results["best"][rd]) == int(want["score"])
        assert (int(rec["query_start"]), int(rec["ref_start"]), int(rec["ref_end"])) == \
            (int(want["query_start"]), int(want["ref_start"]), int(want["ref_end"]))
        assert list(got.ops_of(k)) == list(wops)


def test_trace_pair_winners_on_trimmed_mates(oracle):
    """A paired batch's reads on the device are the trimmed mates: trace the
    first tie of each pair (mate 1 on the template strand, mate 2 on the
    other, pair.rs:135-137) against the oracle on the trimmed codes."""
    from eschalign_b200 import adapter
    refs = synth.panel_tiles()[:40]
    P, _ = synth.pairs_c4(refs, n=200, seed=21)
    mates = P.list()
    trimmed, _ = oracle.trim_pairs(mates)
    with GpuScorer(refs, Scoring(), Mode.SEMIGLOBAL) as g:
        b = g.submit(g.prepare_pairs(mates, adapters=adapter.config()))
        got = g.finish_pairs(b, keep=True)
        jobs = []
        for p in range(len(mates) // 2):
            if got.pairs["n_tied"][p] == 0:
                continue
            c = int(got.pair_ties[p, 0])
            ref, t = c >> 1, c & 1
            jobs += [(2 * p, ref, t), (2 * p + 1, ref, 1 - t)]
        al = g.align_batch(b, jobs)
        b.free()
    for k, (rd, ref, rev) in enumerate(jobs):
        q = revcomp(trimmed[rd]) if rev else trimmed[rd]
        want, wops = oracle.align(q, refs[ref], (2, -1, -10, -1), False)
        rec = al.records[k]
        assert int(rec["score"]) == int(want["score"]), k
        assert (int(rec["query_start"]), int(rec["query_end"]), int(rec["ref_start"]),
                int(rec["ref_end"])) == (int(want["query_start"]), int(want["query_end"]),
                                         int(want["ref_start"]), int(want["ref_end"])), k
        assert list(al.ops_of(k)) == list(wops), k
    # each pair's two traced mates add up to the ranked sum
    for p in range(0, len(jobs), 2):
        pi = jobs[p][0] // 2
        assert int(al.records[p]["score"]) + int(al.records[p + 1]["score"]) == \
            int(got.pairs["best"][pi])


@pytest.mark.parametrize("mode", [Mode.LOCAL, Mode.SEMIGLOBAL])
def test_trace_tagged_values_at_their_edges(oracle, mode):
    """Read lengths around a stripe of 28 and 32 rows, the last length and the
    last reference on the tagged values and the first past them, references
    of one base, gaps of hundreds of bases, free gap extension (ties between
    extending and opening), wildcards, and a scheme whose longer jobs pass the
    bound on 16-bit scores."""
    rng = np.random.default_rng(0x7A6)
    panel = [rng.integers(0, 5 if m == 300 else 4, m).astype(np.uint8)
             for m in (1, 33, 300, 1200, 1700, 1701)]
    reads = []
    for k, n in enumerate((1, 27, 28, 29, 32, 33, 56, 57, 64, 224, 225, 896, 1023, 1024, 1025)):
        ref = panel[2 + k % 4]
        cut = np.concatenate([ref[:n - n // 2], ref[-(n // 2):]]) if n > 1 else ref[:1]
        r = np.resize(cut, n).copy()  # both ends of a reference: one long deletion
        if k % 3 == 1:
            r[n // 3:n // 2] = rng.integers(0, 4, n // 2 - n // 3)
        reads.append(r.astype(np.uint8))
    big = panel[3]
    reads.append(np.concatenate([big[:300], rng.integers(0, 4, 200).astype(np.uint8), big[300:600]]))
    jobs = [(i, r, v) for i in range(len(reads)) for r in range(len(panel)) for v in (0, 1)
            if v == 0 or i % 4 == 0]
    for scoring in ((2, -1, -10, -1), (3, -2, -4, 0), (2, -1, 0, 0), (60, -40, -90, -2)):
        with GpuScorer(panel, Scoring(*scoring), mode) as g:
            check(oracle, g, reads, panel, jobs, scoring, mode == Mode.LOCAL,
                  f"tags {mode.label} {scoring}")


# a mismatch below the gap open, or below the extension: a gap from the border
# beats a mismatch at the first or last bases
BORDER_GAPS = [(1, -4, -6, -1), (5, -4, -8, -1), (2, -3, -2, -1), (2, -3, -1, -5), (1, -4, -2, -1),
               (2, -8, -4, -2), (100, -100, -200, -30)]


def overhanging_read(rng, ref, lead, changed):
    """`lead` bases before the reference, with its first `changed` ones changed."""
    body = ref.copy()
    body[:changed] = np.where(body[:changed] > 3, 0, 3 - body[:changed])
    return np.concatenate([rng.integers(0, 4, lead).astype(np.uint8), body])


@pytest.mark.parametrize("mode", [Mode.LOCAL, Mode.SEMIGLOBAL])
@pytest.mark.parametrize("scoring", BORDER_GAPS)
def test_trace_gaps_from_the_border(oracle, mode, scoring):
    """A deletion of a reference's first bases is opened at the zero border,
    in the first column of every row of a stripe, as an insertion is in the
    first row: reads that hang over a reference's start or, mirrored, its end,
    of lengths on both sides of a stripe of 28 and 32 rows."""
    rng = np.random.default_rng(0xB0D)
    panel = [rng.integers(0, 5 if m == 90 else 4, m).astype(np.uint8)
             for m in (7, 20, 27, 28, 33, 60, 90, 140)]
    reads = []
    for k, lead in enumerate((1, 2, 5, 8, 17, 40)):
        for j, ref in enumerate(panel):
            reads.append(overhanging_read(rng, ref, lead, 1 + (j + k) % 6))
            reads.append(overhanging_read(rng, ref[::-1], lead, 1 + (j + k) % 6)[::-1].copy())
    jobs = [(i, r, v) for i in range(len(reads)) for r in range(len(panel)) for v in (0, 1)
            if r == i // 2 % len(panel) or (i + r) % 5 == 0]
    with GpuScorer(panel, Scoring(*scoring), mode) as g:
        got = check(oracle, g, reads, panel, jobs, scoring, mode == Mode.LOCAL,
                    f"border {mode.label} {scoring}")
        rows = g.score_batch(reads, both_strands=True, full_rows=True).rows
    for k, (rd, ref, rev) in enumerate(jobs):
        assert int(got.records[k]["score"]) == int(rows[rd + rev * len(reads), ref])


def test_trace_leading_deletion_by_hand(oracle):
    """A deletion of three bases and twenty matches, worked out by hand."""
    ref, read = encode("GGGACGTTGCAAGCTTACGATCA"), encode("CCCCCACGTTGCAAGCTTACGATCA")
    for scoring, score in (((1, -4, -6, -1), 12), ((5, -4, -8, -1), 90), ((2, -3, -2, -1), 36),
                           ((100, -100, -200, -30), 1740)):
        with GpuScorer([ref], Scoring(*scoring), Mode.SEMIGLOBAL) as g:
            got = g.align([read], [(0, 0, 0)])
        rec = got.records[0]
        assert (int(rec["score"]), got.cigar(0), int(rec["query_start"]), int(rec["query_end"]),
                int(rec["ref_start"]), int(rec["ref_end"])) == (score, "3D20M", 5, 25, 0, 23)


def test_trace_short_of_device_memory():
    """With 300 MiB of device memory left, jobs whose scratch would be 512 MiB
    run on fewer warps, to the same records."""
    import torch
    refs = synth.panel_tiles()
    reads = synth.reads_c2(refs, n=20_000, seed=0x5EED_0B0E).tuple()
    jobs = [(k, k % len(refs), k & 1) for k in range(20_000)]
    with GpuScorer(refs, Scoring(), Mode.SEMIGLOBAL) as g:
        want = g.align(reads, jobs)
    with GpuScorer(refs, Scoring(), Mode.SEMIGLOBAL) as g:
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8,
                          device="cuda")
        try:
            got = g.align(reads, jobs)
        finally:
            del hog
            torch.cuda.empty_cache()
    assert np.array_equal(got.records, want.records) and np.array_equal(got.ops, want.ops)


@pytest.mark.parametrize("mode", [Mode.LOCAL, Mode.SEMIGLOBAL])
@pytest.mark.parametrize("n,scoring", [(600, (1000, 0, -300, -300)), (1100, (2, 0, -3, -1)),
                                       (1700, (2, 0, -3, -1)), (2600, (5, 0, -9, -2))])
def test_trace_equal_ends_in_two_passes(oracle, mode, n, scoring):
    """A long read's passes each walk every column: of equal ends in two
    passes, rows a whole number of passes (512 rows) apart, the one in the
    smaller column is the alignment's, whichever pass it is in."""
    a, b = encode("ACCACAACCA"), encode("CAAACCACCC")
    t, g = encode("T" * 20), encode("G" * n)
    reads, panel = [], []
    if mode == Mode.LOCAL:
        panel = [np.concatenate([a, t, b]), np.concatenate([b, t, a])]
        for at in (3, 60, 70):
            for apart in range(512, n - at - 10, 512):
                r = g.copy()
                r[at:at + 10], r[at + apart:at + apart + 10] = b, a
                reads.append(r)
    else:
        # the last row ends in column 1, a row of an earlier pass in the last
        panel = [np.concatenate([encode("A"), t, encode("C")])]
        for apart in range(512, n, 512):
            r = g.copy()
            r[n - 1 - apart], r[n - 1] = 1, 0
            reads.append(r)
    jobs = [(i, r, 0) for i in range(len(reads)) for r in range(len(panel))]
    with GpuScorer(panel, Scoring(*scoring), mode) as sc:
        got = check(oracle, sc, reads, panel, jobs, scoring, mode == Mode.LOCAL,
                    f"passes {mode.label} {n}")
    if mode == Mode.SEMIGLOBAL:
        assert all(int(r["ref_end"]) == 1 and int(r["query_end"]) == n for r in got.records)
