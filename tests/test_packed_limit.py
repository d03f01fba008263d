"""Packed event sums apply up to 1,023 events in a sequence (the null events that pad a list add nothing): at the limit the pair
stage takes the records path, past it the fused kernel, with the bytes of the popcount path on both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _codes(n, events, seed=4, L=1200):
    rng = np.random.default_rng(seed)
    s = np.where(rng.random((n, L)) < 0.03, rng.integers(0, 4, (n, L)), rng.integers(0, 4, L)[None]).astype(np.uint8)
    s[1, rng.choice(L, events, replace=False)] = rng.choice((5, 6, 7, 8, 9, 10), events)
    return s


def _names(n):
    return [f"s{i}" for i in range(n)]


@pytest.mark.parametrize("entry", ["run", "batch", "server"])
def test_limit_of_the_packed_sums(entry):
    from swifttn93_b200 import Engine, Fasta, HostAlignment, Options, ResidentReference, synth

    o = Options(threshold=1000.0, mode="resolve", resolve_fraction=0.05, min_overlap=20)
    launches = {}
    for events in (1020, 1021, 1023, 1024):
        codes, got = _codes(40, events), {}
        for path in ("popc", "tc"):
            eng = Engine()
            eng.set_count_path(path)
            if entry == "run":
                s = eng.upload(codes, _names(40))
                body, summ = eng.run(s, o)
                got[path] = (body, summ.json(40))
            elif entry == "batch":
                body, summ = eng.batch_run([HostAlignment(codes, _names(40))], [o])[0]
                got[path] = (body, summ.json(40))
            else:
                res = ResidentReference(eng, Fasta(synth.to_fasta(_names(40), codes)), o, 8, 2)
                q = Fasta(synth.to_fasta(_names(5), _codes(5, 10, 9)), expect_len=1200)
                body, summ = res.batch([q])[0]
                got[path] = (body, summ.json(40, 5, second_file=True))
            launches[path, events] = eng.last_launches()
            eng.close()
        assert got["popc"] == got["tc"], events
    assert launches["tc", 1020] == launches["tc", 1021] == launches["tc", 1023] == launches["tc", 1024] + 1
