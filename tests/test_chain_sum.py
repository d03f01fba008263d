"""Row sums added in groups with the bits of one term after the other (chain_sum.cuh): the scheme on the CPU, and the
engine's sums against a sequential sum of its own distances at row lengths around its groups of 32 and 128."""
import subprocess

import numpy as np
import pytest

from tests.conftest import REPO


def test_scheme_against_sequential_sums(tmp_path):
    exe, src = tmp_path / "chain_check", REPO / "swifttn93_b200" / "csrc"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{src}",
                        str(REPO / "tests" / "native" / "chain_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 33, 34, 129, 130, 161, 1500])
def test_row_sums_equal_sequential_sums(n):
    """A whole run's sums against its row bands' (one summary per row), its columns cut where a row's terms start
    (-s: rows of one file against the other), whose sums of few terms take the one-by-one path."""
    from swifttn93_b200 import Engine, Options

    rng = np.random.default_rng(n)
    codes = np.where(rng.random((n, 400)) < 0.05, rng.integers(0, 4, (n, 400)), rng.integers(0, 4, 400)[None]).astype(np.uint8)
    codes[n // 2:n // 2 + 3] = codes[0]  # some distances of zero
    counts = 1 + np.arange(n) % 2 * (np.arange(n) % 5)
    eng, o = Engine(), Options(threshold=1000.0, mode="resolve", resolve_fraction=0.05, min_overlap=5, format="csv")
    s = eng.upload(codes, [f"s{i}" for i in range(n)], counts)
    _, whole, rows = eng.run_rows(s, o, 0, n)
    for i in sorted({0, 1, n // 3, n - 2} & set(range(n - 1))):
        # one column at a time: each pair's distance is the sum of a run of one row against one column
        terms = []
        pair = None
        for j in range(i + 1, n) if n <= 161 else ():
            if pair is not None:
                eng.free(pair)
            pair = eng.upload(codes[[i, j]], ["a", "b"], None)
            terms.append(eng.run_rows(pair, o, 0, 1)[2][0, 0] * float(counts[i] * counts[j]))
        if pair is not None:
            eng.free(pair)
            total = 0.0
            for t in terms:
                total += t
            assert rows[i, 0] == total
    mean = 0.0
    for r in rows:
        mean += r[0]
    assert whole.mean[0] == mean
    eng.close()
