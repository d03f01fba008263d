"""Uploads from pageable memory in pinned pieces (4 MB on) give the same set as a direct copy from pinned memory: sizes
around the limit and around a piece, and a batch of alignments of which some are too small to be staged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _codes(n, L):
    rng = np.random.default_rng(n + L)
    s = np.where(rng.random((n, L)) < 0.02, rng.integers(0, 4, (n, L)), rng.integers(0, 4, L)[None]).astype(np.uint8)
    s[rng.random((n, L)) < 0.001] = 6
    return s


def _pinned(codes):
    import torch

    return torch.from_numpy(codes).pin_memory().numpy()


@pytest.mark.parametrize("n,L", [(200, 20971), (200, 20972), (64, 65536), (101, 52001), (300, 40003)])
def test_upload_in_pieces_equals_direct_copy(n, L):
    from swifttn93_b200 import Engine, Options

    codes = _codes(n, L)
    names = [f"s{i}" for i in range(n)]
    eng, o, got = Engine(), Options(threshold=1000.0, mode="resolve", resolve_fraction=0.05, min_overlap=5), []
    for c in (codes, _pinned(codes), codes):
        s = eng.upload(c, names)
        body, summ = eng.run(s, o)
        got.append((body, summ.json(n)))
        eng.free(s)
    assert got[0] == got[1] == got[2]
    eng.close()


def test_batch_upload_in_pieces_equals_single_runs():
    from swifttn93_b200 import Engine, HostAlignment, Options

    o = Options(threshold=1000.0, mode="average", min_overlap=5)
    shapes = [(20, 300), (90, 30011), (3, 262144), (150, 20001)]
    alns = [HostAlignment(_codes(n, L), [f"s{i}" for i in range(n)]) for n, L in shapes]
    eng = Engine()
    got = eng.batch_run(alns, [o] * len(alns))
    for (n, L), (body, summ) in zip(shapes, got):
        s = eng.upload(_pinned(_codes(n, L)), [f"s{i}" for i in range(n)])
        want, ws = eng.run(s, o)
        assert body == want and summ.json(n) == ws.json(n)
        eng.free(s)
    eng.close()
