"""A streamed run that reports few pairs leaves the small bands for large ones after the second band: the text in
order and the summary against the oracle, with links in the small bands, at the change and in the large band; with
undecided pairs (a widened logarithm band); and with a budget that the larger buffers do not fit."""
import numpy as np
import pytest

from tests.conftest import run_tn93
from tests.test_bands import _sparse_links

pytestmark = pytest.mark.gpu
N, L = 2700, 150  # 3.6 M pairs: more than three bands


@pytest.mark.parametrize("links", [(), (0, 1, 70, 71, 140, 900, 2500, 2698), tuple(range(0, 2600, 40))],
                         ids=["none", "few", "spread"])
def test_growing_bands_vs_oracle(engine_cli, oracle_bin, tmp_path, links):
    inp = tmp_path / "a.fa"
    inp.write_bytes(_sparse_links(11, N, L, links))
    flags = ["-t", "0.02", "-a", "resolve", "-l", "50"]
    ro, fo, so, _ = run_tn93(oracle_bin, flags, inp, tmp_path)
    for env in ({}, {"TN93G_LOG_BAND": "0.5", "TN93G_LOG_SPREAD": "17179869184"}):
        rg, fg, sg, eg = run_tn93(engine_cli, flags, inp, tmp_path, extra_env=env)
        assert ro == 0 and rg == 0, eg[-300:]
        assert fg == fo and sg == so, env


def test_budget_keeps_the_small_bands():
    from swifttn93_b200 import Engine, Fasta, Options

    data = _sparse_links(12, N, L, (0, 1, 500, 2600))
    opts = Options(threshold=0.02, min_overlap=50)
    got = []
    # the small bands' buffers need about 60 MB here, the large band's about 330 MB
    for budget in (0, 150 << 20):
        eng = Engine(hbm_budget=budget)
        s = eng.upload(Fasta(data))
        for _ in range(2):
            body, summ = eng.run(s, opts)
            got.append((body, summ.links, summ.mean, summ.max, np.asarray(summ.hist).tolist()))
        eng.free(s)
        eng.close()
    assert got[0][1] >= 4 and all(g == got[0] for g in got)
