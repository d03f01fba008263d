"""Contexts with a memory budget that holds a call's own buffers but not what only makes it faster: the call runs, with the
bytes of an unlimited context. The budgets are what the calls take without those buffers, found by halving, and half a
megabyte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _codes(n, L, ambiguous, seed=1, divergence=0.02):
    rng = np.random.default_rng(seed)
    base = rng.integers(0, 4, L)
    s = np.where(rng.random((n, L)) < divergence, rng.integers(0, 4, (n, L)), base[None]).astype(np.uint8)
    hit = rng.random((n, L)) < ambiguous
    s[hit] = rng.choice((5, 6, 7, 8, 9, 10), int(hit.sum()))
    return s


def _names(n):
    return [f"seq{i:05d}" for i in range(n)]


def _engine(megabytes):
    from swifttn93_b200 import Engine

    return Engine(hbm_budget=int(megabytes * 2**20))


@pytest.mark.parametrize("n,L,ambiguous,path,megabytes", [
    (1200, 9000, 0.095, "tc", 139.5), (1200, 9000, 0.095, "popc", 70.5), (300, 20000, 0.5, "tc", 61.0)],
    ids=["packed", "popcount", "unpacked"])
def test_run_without_room_for_event_offsets(n, L, ambiguous, path, megabytes):
    from swifttn93_b200 import Options

    o, got = Options(threshold=1000.0, mode="resolve", min_overlap=20), []
    for budget in (0, megabytes):
        eng = _engine(budget)
        eng.set_count_path(path)
        s = eng.upload(_codes(n, L, ambiguous), _names(n))
        for _ in range(2):
            body, summ = eng.run(s, o)
            got.append((body, summ.json(n)))
        eng.free(s)
        eng.close()
    assert all(g == got[0] for g in got)


@pytest.mark.parametrize("mode,servers,megabytes", [("resolve", 1, 86.0), ("average", 1, 86.0), ("resolve", 2, 210.3)])
def test_server_without_room_for_offsets_and_larger_chunks(mode, servers, megabytes):
    """One server, and two on one context of which the first has to give its extras back."""
    from swifttn93_b200 import Fasta, Options, ResidentReference, synth

    ref = Fasta(synth.to_fasta(_names(2000), _codes(2000, 3000, 0.1)))
    queries = [Fasta(synth.to_fasta([f"q{k}_{i}" for i in range(n)], _codes(n, 3000, 0.1, k + 5)), expect_len=3000)
               for k, n in enumerate((300, 200, 90))]
    o, got = Options(threshold=1000.0, mode=mode, min_overlap=20), []
    for budget in (0, megabytes):
        eng = _engine(budget)
        for res in [ResidentReference(eng, ref, o, 600, 4) for _ in range(servers)] * 2:
            got.append([(b, s.json(ref.n, q.n, second_file=True)) for (b, s), q in zip(res.batch(queries), queries)])
        eng.close()
    assert all(g == got[0] for g in got)


def test_batch_whose_records_leave_no_room_for_what_follows():
    """A batch of which every alignment runs again alone (a logarithm band of half a unit lists more pairs than the batch's
    list holds): the larger records are given back for those runs."""
    from swifttn93_b200 import HostAlignment, Options

    shapes = ((50, 900), (700, 2500), (900, 1500), (1100, 2900), (333, 1111))
    alns = [HostAlignment(_codes(n, L, 0.05, n), _names(n)) for n, L in shapes]
    opts = [Options(threshold=1000.0, mode=m, resolve_fraction=0.05, min_overlap=20)
            for m in ("resolve", "average", "resolve", "resolve", "gapmm")]
    got = []
    for budget in (0, 380.2):
        eng = _engine(budget)
        eng.set_log_band(0.5, 2.0**34)
        got.append([(b, s.json(n)) for (b, s), (n, _) in zip(eng.batch_run(alns, opts), shapes)])
        eng.close()
    assert got[0] == got[1]
