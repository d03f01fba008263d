"""The -g test's AVERAGE pairs, finished in the pair kernel from difference tables: every output byte against the
oracle, where most pairs fall back. Sizes sit on tile and word edges; N runs switch the N plane on; half-ambiguous
sequences leave the packed event sums (more than 1,023 events); three-fold codes still need the site-order walk."""
import tempfile
from pathlib import Path

import numpy as np
import pytest

from tests.conftest import run_tn93

pytestmark = pytest.mark.gpu
TWO, THREE, N, GAP = (5, 6, 7, 8, 9, 10), (11, 12, 13, 14), 15, 17


def _alignment(seed, n, L, two, three, n_runs):
    rng = np.random.default_rng(seed)
    s = np.where(rng.random((n, L)) < 0.04, rng.integers(0, 4, (n, L)), rng.integers(0, 4, L)[None]).astype(np.uint8)
    for codes, rate in ((TWO, two), (THREE, three), ((N,), 0.002), ((GAP,), 0.01)):
        hit = rng.random((n, L)) < rate
        s[hit] = rng.choice(codes, int(hit.sum()))
    for i in range(n):
        for _ in range(rng.poisson(n_runs)):
            a = int(rng.integers(0, L))
            s[i, a:a + int(rng.integers(10, max(11, L // 12)))] = N
    return s


@pytest.mark.parametrize("mode", ["resolve", "RYN"])
@pytest.mark.parametrize("n,L,two,three,n_runs,g", [
    (33, 65, 0.05, 0.0, 0.0, 0.02), (64, 700, 0.02, 0.0, 0.0, 0.015), (97, 1300, 0.005, 0.0, 3.0, 0.05),
    (40, 640, 0.03, 0.002, 2.0, 0.03), (24, 2700, 0.5, 0.0, 0.0, 0.1), (24, 2700, 0.5, 0.0005, 1.0, 0.4)])
def test_average_pairs_vs_oracle(engine_cli, oracle_bin, n, L, two, three, n_runs, g, mode):
    from swifttn93_b200 import synth

    codes = _alignment(n * 7 + L, n, L, two, three, n_runs)
    with tempfile.TemporaryDirectory() as td:
        td = Path(td)
        inp = td / "a.fa"
        inp.write_bytes(synth.to_fasta([f"s{i}" for i in range(n)], codes))
        flags = ["-t", "1000", "-l", "20", "-a", mode, "-g", str(g)]
        ro, fo, so, _ = run_tn93(oracle_bin, flags, inp, td)
        rg, fg, sg, err = run_tn93(engine_cli, flags, inp, td)
    assert ro == rg == 0, err[-300:]
    assert fo == fg and so == sg
