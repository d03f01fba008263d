"""The pair stage in two kernels over the pairs' records (event_kernel and formula_kernel; average, gapmm and skip take the
weighted operand image instead of events): its tables on the CPU, and its bytes against the popcount path's fused kernel
at the edges of its 64-wide tiles, odd first rows and columns, and the record width's change at 2,048 columns."""
import subprocess

import numpy as np
import pytest

from tests.conftest import REPO


def test_tables_stand_for_the_site_contributions(tmp_path):
    exe, src = tmp_path / "tables_check", REPO / "swifttn93_b200" / "csrc"
    r = subprocess.run(["g++", "-O1", "-std=c++17", f"-I{src}", str(REPO / "tests" / "native" / "tables_check.cpp"),
                        str(src / "tables.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _codes(n, L, three):
    rng = np.random.default_rng(n * 31 + L)
    s = np.where(rng.random((n, L)) < 0.05, rng.integers(0, 4, (n, L)), rng.integers(0, 4, L)[None]).astype(np.uint8)
    for codes, rate in (((5, 6, 7, 8, 9, 10), 0.03), ((11, 12, 13, 14), three), ((4, 15, 16), 0.004), ((17,), 0.03)):
        hit = rng.random((n, L)) < rate
        s[hit] = rng.choice(codes, int(hit.sum()))
    s[:, :3] = 2  # constant columns
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["resolve", "average", "gapmm", "skip", "RYN"])
@pytest.mark.parametrize("n,L,three", [(2, 9, 0.0), (63, 300, 0.0), (64, 131, 0.01), (65, 700, 0.0), (129, 640, 0.002),
                                       (70, 2047, 0.0), (66, 2048, 0.001)])
def test_records_path_equals_popcount_path(n, L, three, mode):
    from swifttn93_b200 import Engine, Options

    eng = Engine()
    s = eng.upload(_codes(n, L, three), [f"s{i}" for i in range(n)], 1 + np.arange(n) % 3)
    got = {}
    for path in ("popc", "tc"):
        eng.set_count_path(path)
        got[path] = out = []
        for g in (0.05, 1.0):
            o = Options(threshold=1000.0, mode=mode, resolve_fraction=g, min_overlap=5)
            body, summ = eng.run(s, o)
            out.append((body, summ.json(n), summ.mean, summ.max, summ.pairs_replayed if three == 0.0 and g == 1.0 else None))
            if n > 2:
                n1 = n // 2 | 1  # columns from an odd index, rows from an odd index
                body, summ = eng.run(s, o, n1=n1)
                out.append((body, summ.json(n1, n - n1, True)))
                body, summ, rows = eng.run_rows(s, o, n1, n - 1)
                out.append((body, rows.tobytes(), summ.links))
    assert got["tc"] == got["popc"]
    eng.close()
