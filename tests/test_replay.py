"""Order-dependent pairs (three-fold codes): their sites from the sequences' merged events (32 events or fewer in each) or
from the planes (more, N runs, gapmm), and many pairs to a warp; every output byte against the oracle."""
import tempfile
from pathlib import Path

import numpy as np
import pytest

from tests.conftest import run_tn93

pytestmark = pytest.mark.gpu


def _codes(n, L, events, n_runs):
    """Sequence i has events - 3 .. events + 2 ambiguity codes, a third of them three-fold, many at shared columns."""
    rng = np.random.default_rng(n * L + events)
    s = np.where(rng.random((n, L)) < 0.05, rng.integers(0, 4, (n, L)), rng.integers(0, 4, L)[None]).astype(np.uint8)
    s[rng.random((n, L)) < 0.02] = 17
    shared = rng.choice(L, min(L, 2 * events + 8), replace=False)
    for i in range(n):
        k = min(L, max(0, events - 3 + i % 6))
        at = rng.choice(shared, min(k, len(shared)), replace=False)
        s[i, at] = rng.choice([5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 4], len(at))
        if n_runs:
            a = int(rng.integers(0, L))
            s[i, a:a + 60] = 15
    return s


@pytest.mark.parametrize("mode,g", [("resolve", 1.0), ("resolve", 0.03), ("average", 1.0), ("skip", 1.0), ("gapmm", 1.0), ("RYN", 0.05)])
@pytest.mark.parametrize("n,L,events,n_runs", [(2, 40, 3, 0), (130, 300, 5, 0), (60, 700, 32, 0), (40, 500, 64, 0), (40, 900, 6, 1)])
def test_vs_oracle(engine_cli, oracle_bin, n, L, events, n_runs, mode, g):
    from swifttn93_b200 import synth

    with tempfile.TemporaryDirectory() as td:
        td = Path(td)
        inp = td / "a.fa"
        inp.write_bytes(synth.to_fasta([f"s{i}" for i in range(n)], _codes(n, L, events, n_runs)))
        flags = ["-t", "1000", "-l", "20", "-a", mode, "-g", str(g)]
        ro, fo, so, _ = run_tn93(oracle_bin, flags, inp, td)
        rg, fg, sg, err = run_tn93(engine_cli, flags, inp, td)
    assert ro == rg == 0, err[-300:]
    assert fo == fg and so == sg
