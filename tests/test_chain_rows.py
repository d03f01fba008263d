"""Sums in groups have the bits of one term after the other where the groups are used: rows of many 128-term groups against
their own distances, each from an alignment of two, and the reductions of a batch and of a server (shares of 2,048 rows by all
warps of a block) against the rows' sums added in order. Copy numbers and distances of zero are among the terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L = 300


def _set(n, seed):
    rng = np.random.default_rng(seed)
    s = np.where(rng.random((n, L)) < 0.05, rng.integers(0, 4, (n, L)), rng.integers(0, 4, L)[None]).astype(np.uint8)
    s[n // 2:n // 2 + 3] = s[0]  # some distances of zero
    s[n // 3:n // 3 + 200] = s[1]
    return s, 1 + np.arange(n) % 2 * (np.arange(n) % 5)


def _names(n):
    return [f"s{i}" for i in range(n)]


def _opts():
    from swifttn93_b200 import Options

    return Options(threshold=0.001, mode="resolve", min_overlap=5, count_only=True)


def _in_order(terms):
    total = 0.0
    for t in terms:
        total += t
    return total


@pytest.mark.parametrize("n", [1500, 2050])
def test_long_rows_equal_sequential_sums(n):
    from swifttn93_b200 import Engine, HostAlignment

    codes, counts = _set(n, n)
    eng, o = Engine(), _opts()
    s = eng.upload(codes, _names(n), counts)
    _, _, rows = eng.run_rows(s, o, 0, n)
    for i in (0, 1, n // 3, n - 140):
        pairs = [HostAlignment(codes[[i, j]], ["a", "b"]) for j in range(i + 1, n)]
        d = [summ.mean[0] for _, summ in eng.batch_run(pairs, [o] * len(pairs))]
        assert min(d) == 0.0 or i == n - 140
        assert rows[i, 0] == _in_order(x * float(counts[i] * counts[j]) for x, j in zip(d, range(i + 1, n)))
    eng.close()


@pytest.mark.parametrize("n", [2047, 2048, 2049, 5000])
def test_reductions_equal_sequential_sums(n):
    from swifttn93_b200 import Engine, Fasta, HostAlignment, ResidentReference, synth

    codes, counts = _set(n, n)
    eng, o = Engine(), _opts()
    s = eng.upload(codes, _names(n), counts)
    _, _, rows = eng.run_rows(s, o, 0, n)
    (_, got), = eng.batch_run([HostAlignment(codes, _names(n), counts)], [o])
    assert got.mean[0] == _in_order(rows[:, 0]) and got.weighted[0] == _in_order(rows[:, 3])
    eng.free(s)
    q, _ = _set(203, 3)
    s = eng.upload(np.concatenate([codes, q]), _names(n + 203))
    _, _, rows = eng.run_rows(s, o, 0, n, n1=n)
    eng.free(s)
    ref = Fasta(synth.to_fasta(_names(n), codes))
    res = ResidentReference(eng, ref, o, 203, 1)
    (_, got), = res.batch([Fasta(synth.to_fasta([f"q{i}" for i in range(203)], q), expect_len=L)])
    assert got.mean[0] == _in_order(rows[:, 0]) and got.weighted[0] == _in_order(rows[:, 3])
    eng.close()
