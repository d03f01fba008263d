"""Batches whose alignments take the pair stage in two kernels (and the weighted operand image under average, gapmm and
skip), beside ones that keep the fused kernel (N plane under resolve, more than 1,023 events): each alignment's text and
summary equal those of the popcount path, at the edges of the 64-wide tiles, of the formula's segments and of the record
widths; a batch whose larger records do not fit the context's memory still runs."""
import numpy as np
import pytest

from tests.test_pair_split import _codes

pytestmark = pytest.mark.gpu


def _batch():
    from swifttn93_b200 import HostAlignment, Options

    out = []
    shapes = [(2, 9, 0.0), (63, 300, 0.0), (65, 131, 0.01), (129, 640, 0.002), (70, 2047, 0.0), (66, 2048, 0.001), (300, 90, 0.0)]
    for n, L, three in shapes:
        for mode in ("resolve", "average", "gapmm", "skip", "RYN"):
            codes = _codes(n, L, three)
            if L == 131:
                codes[:, 5:60] = 15  # N runs: the N plane under resolve
            if L == 2048 and mode == "resolve":
                codes[3, 100:1500] = 5  # more than 1,023 events
            g = 0.05 if n % 2 else 1.0
            out.append((HostAlignment(codes, [f"s{i}" for i in range(n)], 1 + np.arange(n) % 3),
                        Options(threshold=1000.0, mode=mode, resolve_fraction=g, min_overlap=5)))
    return out


def test_batch_equals_popcount_path():
    from swifttn93_b200 import Engine

    work = _batch()
    eng = Engine()
    got = {}
    for path in ("popc", "tc"):
        eng.set_count_path(path)
        r = eng.batch_run([a for a, _ in work], [o for _, o in work])
        got[path] = [(body, s.json(a.n), s.mean, s.max) for (body, s), (a, _) in zip(r, work)]
    for k, (p, t) in enumerate(zip(got["popc"], got["tc"])):
        assert p == t, (work[k][0].n, work[k][0].L, work[k][1].mode)
    eng.close()


def test_batch_without_room_for_its_records_takes_the_fused_kernel():
    from swifttn93_b200 import Engine, HostAlignment, Options

    n, L = 1500, 2100
    alns = [HostAlignment(_codes(n, L, 0.0), [f"s{i}" for i in range(n)])]
    opts = [Options(threshold=0.01, mode="resolve", resolve_fraction=0.05, min_overlap=5)]
    eng = Engine()
    want = eng.batch_run(alns, opts)[0]
    eng.close()
    # distances 8 n^2, queue 4 n^2, records 16 n^2 (fused) or 32 n^2 (32 L past 16 bits), images and the rest about 25 MB
    eng = Engine(hbm_budget=(12 + 16 + 8) * n * n + (25 << 20))
    body, s = eng.batch_run(alns, opts)[0]
    assert body == want[0] and s.json(n) == want[1].json(n)
    eng.close()
