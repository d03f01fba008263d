"""The writer's lines by 8-byte words: every byte against the oracle for names of every length around a word and the
longest that goes by words (64), names that share a word with their neighbours, column numbers around powers of ten, short
lines, and distances of zero, below 1e-4 (exponents) and above 1."""
import tempfile
from pathlib import Path

import numpy as np
import pytest

from tests.conftest import run_tn93

pytestmark = pytest.mark.gpu


def _codes(n, L, rate):
    rng = np.random.default_rng(n + L)
    s = np.where(rng.random((n, L)) < rate * rng.random((n, 1)), rng.integers(0, 4, (n, L)), rng.integers(0, 4, L)[None])
    s[n // 2:n // 2 + 5] = s[0]
    return s.astype(np.uint8)


@pytest.mark.parametrize("fmt", ["csv", "csvn"])
@pytest.mark.parametrize("n,L,rate,names,t", [
    (150, 700, 0.3, [1, 2, 3], "1000"), (90, 700, 0.3, list(range(1, 40)), "1000"), (40, 60, 1.2, [62, 63, 64, 65, 66, 7], "1000"),
    (33, 20000, 0.0004, [8, 16, 17], "1000"), (1103, 300, 0.2, [13, 14], "0.02"), (20, 500, 0.2, [200, 5, 1500], "1000")])
def test_text_vs_oracle(engine_cli, oracle_bin, n, L, rate, names, t, fmt):
    from swifttn93_b200 import synth

    ids = [(f"{i:x}" + "abcdefghijklmnopqrstuvwxyz" * 60)[:max(names[i % len(names)], len(f"{i:x}"))] for i in range(n)]
    with tempfile.TemporaryDirectory() as td:
        td = Path(td)
        inp = td / "a.fa"
        inp.write_bytes(synth.to_fasta(ids, _codes(n, L, rate)))
        flags = ["-t", t, "-l", "20", "-a", "resolve", "-f", fmt]
        ro, fo, so, _ = run_tn93(oracle_bin, flags, inp, td)
        rg, fg, sg, err = run_tn93(engine_cli, flags, inp, td)
    assert ro == rg == 0, err[-300:]
    assert fo == fg and so == sg
