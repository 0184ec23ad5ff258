"""The batched kernel's shapes and lane formats at their edges, against the
scalar oracle by equality: read lengths around a stripe of 16, 28 and 32
rows, the lengths where the shape changes (224 / 225, 1024 / 1025) and where
a long read's last pass changes its stripes (512 rows past a pass), and
panels whose largest score is the last the f16 lanes hold (2047) and the
first they do not."""
import numpy as np
import pytest

from eschalign_b200 import GpuError, GpuScorer, Mode, Scoring
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu

SHORT = [1, 15, 16, 17, 27, 28, 29, 31, 32, 33, 55, 56, 57, 63, 64, 65, 111, 112, 113, 224, 225]
LONG = [895, 897, 1023, 1024, 1025, 1535, 1536, 1537, 2047, 2048, 2049, 2560, 2561]
INT32 = ((2, 256, 64), (1, 256, 64))  # KERNEL_INT32, KERNEL_PLAIN32
DEFAULT = ((0, 16, 64), (0, 16, 1))  # KERNEL_AUTO on the default split


def _reads(rng, panel, lens):
    out = []
    for k, n in enumerate(lens):
        ref = panel[k % len(panel)]
        r = np.resize(ref, n).copy()
        hit = rng.random(n) < 0.08
        r[hit] = rng.integers(0, 5 if k % 3 == 0 else 4, int(hit.sum()))
        out.append(r.astype(np.uint8))
    return out


@pytest.mark.parametrize("mode", [Mode.LOCAL, Mode.SEMIGLOBAL])
@pytest.mark.parametrize("lens,spread", [(SHORT, (1, 31, 90, 130)), (LONG, (20, 40, 300))],
                         ids=["short", "long"])
def test_shapes_at_their_edges(oracle, mode, lens, spread):
    rng = np.random.default_rng(len(lens))
    panel = [rng.integers(0, 5 if n == 90 else 4, n).astype(np.uint8) for n in spread]
    reads = _reads(rng, panel, lens)
    for scoring in ((2, -1, -10, -1), (3, 1, -5, -2), (2, -3, -1, -5)):
        check(oracle, panel, reads, scoring, mode, "shape edges", kernels=DEFAULT)


@pytest.mark.parametrize("mode", [Mode.LOCAL, Mode.SEMIGLOBAL])
def test_int32_lanes_at_their_edges(oracle, mode):
    """Chains of 1-32 lanes, one to four passes, one reference and lists
    short enough for fewer references a unit."""
    rng = np.random.default_rng(32)
    panel = [rng.integers(0, 5 if n == 40 else 4, n).astype(np.uint8) for n in (1, 2, 31, 40, 300)]
    reads = _reads(rng, panel, SHORT + [896, 897, 1024, 1025, 3073])
    for scoring in ((100, -100, -200, -30), (2, -3, -1, -5)):
        check(oracle, panel, reads, scoring, mode, "int32 edges", kernels=INT32)
        check(oracle, panel[3:4], reads[8:11], scoring, mode, "int32, one reference",
              kernels=INT32)


@pytest.mark.parametrize("match,length", [(23, 89), (32, 64), (89, 23), (127, 16), (127, 17)])
def test_last_score_of_the_f16_lanes(oracle, match, length):
    """match x length = 2047 is the largest score kept as an f16 subnormal;
    2048 takes the int16 lanes, as does 127 x 17."""
    rng = np.random.default_rng(match)
    panel = [rng.integers(0, 4, length).astype(np.uint8) for _ in range(3)]
    panel.append(np.full(length, 4, np.uint8))  # wildcards: every read scores the most
    reads = _reads(rng, panel, [length, length - 1, length + 40, 5]) + [p.copy() for p in panel]
    for scoring in ((match, 0, -7, -1), (match, -match + 127 - match, -1, -1)):
        if scoring[1] < match:
            check(oracle, panel, reads, scoring, Mode.LOCAL, "f16 limit", kernels=DEFAULT)


def test_scorers_over_panels_of_different_sizes(oracle):
    """A scorer over a small panel made later leaves one over a larger panel
    (more shared memory a CTA) usable."""
    rng = np.random.default_rng(5)
    big = [rng.integers(0, 4, 900).astype(np.uint8) for _ in range(60)]
    small = [rng.integers(0, 4, 50).astype(np.uint8)]
    reads = _reads(rng, big, [40, 100, 300])
    with GpuScorer(big, Scoring(), Mode.LOCAL) as g, GpuScorer(small, Scoring(), Mode.LOCAL) as h:
        assert g.info()["panel_bytes"] > 48 * 1024
        rows = g.score_batch(reads, full_rows=True).rows
        assert (h.score_batch(reads, full_rows=True).rows ==
                oracle.score_matrix(reads, small, (2, -1, -10, -1), True)).all()
    assert (rows == oracle.score_matrix(reads, big, (2, -1, -10, -1), True)).all()


@pytest.mark.parametrize("mode", [Mode.LOCAL, Mode.SEMIGLOBAL])
@pytest.mark.parametrize("cap", [1, 8, 32])
def test_small_batches_without_a_split(oracle, mode, cap):
    """A scorer left to itself puts a few reads on 8- or 16-row stripes, a
    panel chunk per reference pair, and merges the chunks straight into the
    results: one to forty reads (empty ones, ones past those stripes among
    them) against one to 90 references, a third of them the same, so that tie
    sets span many chunks and outrun the list."""
    rng = np.random.default_rng(cap)
    same = rng.integers(0, 4, 60).astype(np.uint8)
    panel = [same if k % 3 == 0 else rng.integers(0, 4, int(rng.integers(20, 140))).astype(np.uint8)
             for k in range(90)]
    sc = (2, -1, -10, -1)
    local = mode == Mode.LOCAL
    for n_refs in (1, 2, 90):
        refs = panel[:n_refs]
        with GpuScorer(refs, Scoring(*sc), mode, tie_capacity=cap) as g:
            for lens in ([60], [0, 8, 9], [255, 256, 257, 513, 0], SHORT + SHORT[::-1]):
                reads = _reads(rng, refs, lens)
                want, ties, _ = oracle.scalar_map_batch(reads, refs, sc, local, True, cap=cap)
                got = g.score_batch(reads, both_strands=True)
                for f in ("best", "suboptimal", "n_tied"):
                    assert (got.results[f] == want[f]).all(), (n_refs, lens, f)
                for k in range(len(reads)):
                    m = min(int(want["n_tied"][k]), cap)
                    assert list(got.ties[k, :m]) == list(ties[k][:m]), (n_refs, lens, k)
                    assert (got.ties[k, m:] == 0xFFFFFFFF).all()
                rows = g.score_batch(reads, both_strands=True, full_rows=True).rows
                rc = [oracle.revcomp(r) for r in reads]
                assert (rows == oracle.score_matrix(reads + rc, refs, sc, local)).all()
                one = g.score_batch(reads)
                fwd, _, _ = oracle.scalar_map_batch(reads, refs, sc, local, False, cap=cap)
                assert (one.results["best"] == fwd["best"]).all()


@pytest.mark.parametrize("kernel", ["empty", "int32"])
def test_chunk_states_of_few_tiled_queries(oracle, kernel):
    """One read for the batched kernel among 20 000 that are empty (or, past
    what its lanes hold, on the int32 lanes): the panel is cut into chunks for
    the one, but the memory of their states, held for every query, stays
    within 64 chunks a query or 32 queries to each of the device's tasks."""
    rng = np.random.default_rng(21)
    same = rng.integers(0, 4, 12).astype(np.uint8)
    panel = [same if k % 5 == 0 else rng.integers(0, 4, int(rng.integers(8, 14))).astype(np.uint8)
             for k in range(2100)]
    n, cap, sc = 20_000, 8, (2, -1, -10, -1)
    reads = [np.zeros(0, np.uint8)] * n
    mode = Mode.LOCAL
    if kernel == "int32":
        # semi-global lanes hold 2 |open| + (min(n, L) - 1) |extend| < 15000:
        # with this extension reads up to 15 bases of a 16-base reference
        sc, mode = (2, -1, -10, -1000), Mode.SEMIGLOBAL
        panel[7] = rng.integers(0, 4, 40).astype(np.uint8)
        reads = [rng.integers(0, 4, 30).astype(np.uint8) for _ in range(n)]
    reads[n // 2] = same.copy()
    with GpuScorer(panel, Scoring(*sc), mode, tie_capacity=cap) as g:
        tasks = 32 * 4 * g.info()["batched_blocks"]
        got = g.score_batch(reads, both_strands=True)
    st = got.stats
    assert st["queries_batched"] == 2 and st["panel_chunks"] > 1
    n_q, row = 2 * n, 16 + 4 * cap
    assert st["panel_chunks"] <= max(64, -(-32 * tasks // n_q))
    rest = 64 * n_q + (n_q + 2) * row + 4 * len(panel) * (n_q if kernel == "int32" else 1) + (1 << 20)
    assert st["device_bytes"] <= max(64 * n_q, 32 * tasks + n_q) * row + rest
    want, ties, _ = oracle.scalar_map_batch(reads[n // 2:n // 2 + 1], panel, sc,
                                            mode == Mode.LOCAL, True, cap=cap)
    for f in ("best", "suboptimal", "n_tied"):
        assert got.results[f][n // 2] == want[f][0], f
    assert list(got.ties[n // 2, :cap]) == list(ties[0][:cap])
    if kernel == "empty":
        assert (np.delete(got.results["flags"], n // 2) & 1).all()


@pytest.mark.parametrize("merge", ["fused", "unfused"])
def test_chunks_past_64(oracle, merge):
    """A panel of more than 1024 reference pairs, ties spread over it, cut
    into up to 1024 chunks: what a scorer does by itself and what
    set_chunking(1024) gives back after a smaller cap; merged straight into
    the results or, with a read on the int32 lanes in the batch, apart."""
    rng = np.random.default_rng(1024)
    same = rng.integers(0, 4, 12).astype(np.uint8)
    panel = [same if k % 7 == 0 else rng.integers(0, 4, int(rng.integers(8, 14))).astype(np.uint8)
             for k in range(2101)]
    panel[7] = rng.integers(0, 4, 40).astype(np.uint8)
    sc, cap = (2, -1, -10, -1000), 32
    reads = [same.copy(), rng.integers(0, 4, 9).astype(np.uint8), np.zeros(0, np.uint8)]
    if merge == "unfused":
        reads.append(rng.integers(0, 4, 30).astype(np.uint8))  # past the semi-global lanes
    want, ties, _ = oracle.scalar_map_batch(reads, panel, sc, False, True, cap=cap)
    with GpuScorer(panel, Scoring(*sc), Mode.SEMIGLOBAL, tie_capacity=cap) as g:
        for bad in (0, 1025):
            with pytest.raises(GpuError):
                g.set_chunking(bad)
        for chunks in (None, 1, 64, 1024):
            if chunks:
                g.set_chunking(chunks)
            got = g.score_batch(reads, both_strands=True)
            assert got.stats["panel_chunks"] == (chunks or 1024)
            assert got.stats["queries_plain"] == (2 if merge == "unfused" else 0)
            for f in ("best", "suboptimal", "n_tied"):
                assert (got.results[f] == want[f]).all(), (chunks, f)
            for k in range(len(reads)):
                m = min(int(want["n_tied"][k]), cap)
                assert list(got.ties[k, :m]) == list(ties[k][:m]), (chunks, k)
                assert (got.ties[k, m:] == 0xFFFFFFFF).all()


@pytest.mark.parametrize("scoring", [(100, -27, -7, -1), (120, -7, -7, -1), (64, -63, 0, 0),
                                     (127, 0, 0, -1), (23, -104, 0, -1), (89, -38, -30, -2)])
def test_f16_lanes_up_to_their_table_and_score(oracle, scoring):
    """Schemes whose largest table byte is the last that fits (match less a
    negative mismatch 127; 23, -104 reaches it with the largest offset), panels
    whose largest score is the last one the f16 lanes hold and one base more,
    all taken by the batched kernel."""
    match = scoring[0]
    assert match - min(scoring[1], 0) == 127
    rng = np.random.default_rng(match)
    for length in (2047 // match, 2047 // match + 1):
        panel = [rng.integers(0, 4, length).astype(np.uint8) for _ in range(3)]
        panel.append(np.full(length, 4, np.uint8))  # wildcards: every read scores the most
        reads = _reads(rng, panel, [length, length - 1, length + 40, 5, 300, 1100])
        reads += [p.copy() for p in panel]
        with GpuScorer(panel, Scoring(*scoring), Mode.LOCAL) as g:
            assert g.info()["batched_ok"]
            assert g.prepare(reads, both_strands=True).work_split() == (2 * len(reads), 0)
        check(oracle, panel, reads, scoring, Mode.LOCAL, "f16 limit", kernels=DEFAULT)
