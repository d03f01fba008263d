"""Server batches of several chunks of query columns, with references that do not end on a chunk's 64-column tiles: the
pair stage of a chunk stops at the last column that its count kernel counted. Several batches through one server (records of
an earlier batch stand behind a chunk's end) against the popcount path and, for the counters, against each query alone."""
import numpy as np
import pytest

from tests.conftest import run_tn93

L = 300


def _codes(n, three, two, seed):
    rng = np.random.default_rng(seed)
    base = np.random.default_rng(17).integers(0, 4, L)
    s = np.where(rng.random((n, L)) < 0.03, rng.integers(0, 4, (n, L)), base[None]).astype(np.uint8)
    for codes, rate in (((5, 6, 7, 8, 9, 10), two), ((11, 12, 13, 14), three), ((17,), 0.01)):
        hit = rng.random((n, L)) < rate
        s[hit] = rng.choice(codes, int(hit.sum()))
    if three:
        s[:, 7] = 11  # a three-fold code in every sequence: under average every pair takes the site-order walk
    return s


def _fasta(tag, codes):
    from swifttn93_b200 import Fasta, synth

    return Fasta(synth.to_fasta([f"{tag}{i}" for i in range(len(codes))], codes), expect_len=L)


def _batches(three):
    return [[_fasta(f"b{b}q{k}_", _codes(n, three, 0.02 + 0.05 * b, 100 * b + k)) for k, n in enumerate(sizes)]
            for b, sizes in enumerate(((400, 1, 350, 33, 300, 64), (37, 500, 7, 600)))]


@pytest.mark.gpu
@pytest.mark.parametrize("nref,mode,g,overlap,three", [
    (83, "resolve", 0.05, 0, 0.01), (96, "resolve", 0.05, 100, 0.01), (112, "resolve", 0.05, 100, 0.0),
    (83, "resolve", 1.0, 5, 0.01), (83, "average", 1.0, 5, 0.01), (112, "gapmm", 1.0, 5, 0.002), (83, "RYN", 0.05, 5, 0.01)])
def test_chunks_end_where_the_counts_end(nref, mode, g, overlap, three):
    from swifttn93_b200 import Engine, Options, ResidentReference

    ref, work = _fasta("r", _codes(nref, three, 0.02, 5)), _batches(three)
    opts = Options(threshold=1000.0, mode=mode, resolve_fraction=g, min_overlap=overlap)
    out, counters = {}, {}
    for path in ("popc", "tc"):
        eng = Engine()
        eng.set_count_path(path)
        res = ResidentReference(eng, ref, opts, max_batch_sequences=1200, max_batch_queries=8)
        got = [res.batch(q) for q in work]
        out[path] = [[(b, s.json(nref, q.n, second_file=True)) for (b, s), q in zip(r, qs)] for r, qs in zip(got, work)]
        counters[path] = [(r[0][1].pairs_replayed, r[0][1].logs_ambiguous) for r in got]
        if path == "tc":  # each query alone: one chunk
            alone = [[res.batch([q])[0][1] for q in qs if q.n < 449] for qs in work]
            whole = [[q.n < 449 for q in qs] for qs in work]
        res.close()
        eng.close()
    assert out["tc"] == out["popc"]
    assert all(whole[0])
    assert counters["tc"][0] == (sum(s.pairs_replayed for s in alone[0]), sum(s.logs_ambiguous for s in alone[0]))
    if three and mode == "average":
        assert counters["tc"][0][0] == nref * sum(q.n for q in work[0])


@pytest.mark.gpu
def test_chunks_with_an_unpacked_reference_vs_oracle(oracle_bin, tmp_path):
    """A reference sequence of more than 1,023 events keeps the fused kernel."""
    from swifttn93_b200 import Engine, Fasta, Options, ResidentReference, synth
    from swifttn93_b200.serve import header_line

    rng = np.random.default_rng(3)
    n, Lw = 83, 1400
    base = rng.integers(0, 4, Lw)

    def codes(m):
        s = np.where(rng.random((m, Lw)) < 0.03, rng.integers(0, 4, (m, Lw)), base[None]).astype(np.uint8)
        for c, rate in (((5, 6, 7, 8, 9, 10), 0.03), ((11, 12, 13, 14), 0.0005)):
            hit = rng.random((m, Lw)) < rate
            s[hit] = rng.choice(c, int(hit.sum()))
        return s

    rc = codes(n)
    rc[4, 100:1250] = 5
    ref = synth.to_fasta([f"r{i}" for i in range(n)], rc)
    refp = tmp_path / "ref.fa"
    refp.write_bytes(ref)
    opts = Options(threshold=1000.0, mode="resolve", resolve_fraction=0.05, min_overlap=100)
    eng = Engine()
    res = ResidentReference(eng, Fasta(ref), opts, max_batch_sequences=1100, max_batch_queries=4)
    for b in range(2):
        queries = [synth.to_fasta([f"b{b}q{k}_{i}" for i in range(m)], codes(m)) for k, m in enumerate((500, 90, 430))]
        out = res.batch([Fasta(q, expect_len=Lw) for q in queries])
        for k, q in enumerate(queries):
            qp = tmp_path / f"q{k}.fa"
            qp.write_bytes(q)
            ro, fb, so, _ = run_tn93(oracle_bin, ["-t", "1000", "-a", "resolve", "-g", "0.05", "-l", "100", "-s", str(qp)],
                                     refp, tmp_path)
            assert ro == 0
            assert header_line(opts) + out[k][0] == fb, (b, k)
            assert out[k][1].json(n, Fasta(q).n, second_file=True) == so, (b, k)
    res.close()
    eng.close()
