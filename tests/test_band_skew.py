"""Sets whose first rows report little and the rest much: the large bands that the first rows bring about hand their text over
in pieces of whole rows, in order, and small bands follow when more rows are left. Text and summary against the oracle, and
under a budget that the small bands fit."""
import numpy as np
import pytest

from tests.conftest import run_tn93
from tests.test_budget import _engine

pytestmark = pytest.mark.gpu


def _skewed(n, L, panel, name="s"):
    """panel unrelated sequences, then close ones; every 97th of those unrelated too, so that some rows have no text"""
    rng = np.random.default_rng(n + L)
    alpha = np.frombuffer(b"ACGT", dtype=np.uint8)
    base = rng.integers(0, 4, L)
    s = np.where(rng.random((n, L)) < 0.005, rng.integers(0, 4, (n, L)), base[None])
    far = np.arange(n) < panel
    far[panel::97] = True
    s[far] = rng.integers(0, 4, (int(far.sum()), L))
    rows = alpha[s]
    rows[rng.random((n, L)) < 0.01] = ord("R")
    return b"".join(b">%s%05d\n" % (name.encode(), i) + rows[i].tobytes() + b"\n" for i in range(n))


@pytest.mark.parametrize("n,panel,extra", [(6000, 120, []), (6000, 1900, ["-0", "-f", "csvn"]), (9000, 130, ["-f", "csvn"])],
                         ids=["pieces", "late", "back-to-small"])
def test_skewed_set_vs_oracle(engine_cli, oracle_bin, tmp_path, n, panel, extra):
    inp = tmp_path / "a.fa"
    inp.write_bytes(_skewed(n, 100, panel))
    flags = ["-t", "0.05", "-a", "resolve", "-l", "20", *extra]
    ro, fo, so, _ = run_tn93(oracle_bin, flags, inp, tmp_path)
    rg, fg, sg, eg = run_tn93(engine_cli, flags, inp, tmp_path)
    assert ro == 0 and rg == 0, eg[-300:]
    assert len(fo) > (100 << 20)
    assert fg == fo and sg == so


@pytest.mark.parametrize("megabytes", [100.0, 205.0, 420.0, 700.0])
def test_skewed_set_within_a_budget(megabytes):
    """The small bands take 204 MB here with their texts in one piece each and 93 in pieces of a few rows; one band of everything
    that is left, with its text in one piece, took 691."""
    from swifttn93_b200 import Fasta, Options

    data = Fasta(_skewed(3200, 300, 300, "a_rather_long_sequence_name_"))
    o, got = Options(threshold=0.02, mode="resolve", min_overlap=20), []
    for budget in (0, megabytes):
        eng = _engine(budget)
        s = eng.upload(data)
        for _ in range(2):
            body, summ = eng.run(s, o)
            got.append((body, summ.json(s.N)))
        eng.close()
    assert len(got[0][0]) > (180 << 20) and all(g == got[0] for g in got)


@pytest.mark.parametrize("megabytes,then", [(274.7, "batch"), (194.3, "server")])
def test_large_bands_leave_room_for_later_calls(megabytes, then):
    """A run in large bands, then a batch or a server whose buffers fit beside those of a run in small bands."""
    from swifttn93_b200 import Fasta, HostAlignment, Options, ResidentReference, synth
    from tests.test_budget import _codes, _names

    far = HostAlignment(_codes(2700, 150, 0.0, divergence=0.75), _names(2700))
    o = Options(threshold=1000.0, mode="resolve", resolve_fraction=0.05, min_overlap=20)
    got = []
    for budget in (0, megabytes):
        eng = _engine(budget)
        s = eng.upload(far)
        body, summ = eng.run(s, Options(threshold=0.02, mode="resolve", min_overlap=20))
        eng.free(s)
        out = [body, summ.json(2700)]
        if then == "batch":
            shapes = ((50, 900), (700, 2500), (900, 1500), (1100, 2900), (333, 1111))
            out += [b for b, _ in eng.batch_run([HostAlignment(_codes(n, L, 0.05, n), _names(n)) for n, L in shapes], [o] * 5)]
        else:
            ref = Fasta(synth.to_fasta(_names(2000), _codes(2000, 3000, 0.1)))
            q = Fasta(synth.to_fasta([f"q{i}" for i in range(300)], _codes(300, 3000, 0.1, 5)), expect_len=3000)
            out += [ResidentReference(eng, ref, o, 600, 4).batch([q])[0][0]]
        got.append(out)
        eng.close()
    assert got[0] == got[1]
