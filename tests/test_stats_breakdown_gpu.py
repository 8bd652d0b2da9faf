"""The per-phase times of a solve that runs in one launch (a cluster of one or
more CTAs, a grid), against its per-round times: the rounds are the rounds, and
prep, scans and flatten are reported as themselves."""
import pytest

import ecl_mst as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [1000, 8000, 100_000, 480_000])
@pytest.mark.parametrize("kw", [dict(mode=E.THRESH_NONE), dict(mode=E.THRESH_QUANTILE, quantile=0.2)])
def test_breakdown(nodes, kw):
    g = E.gen_er(nodes, 8.0, nodes, 1 << 20)
    with E.Context(g.nodes, g.edges) as c:
        for _ in range(3):
            _, st = c.run_host(g, E.make_opts(flags=E.FLAG_NO_GRAPH, **kw))
    rounds = sum(sum(r) for p in st["us_round"] for r in p)
    # the device clock steps by up to a microsecond; the last barrier of a phase
    # and its last look at the list (a few microseconds) lie outside the passes
    assert rounds - 4 <= 1e3 * st["ms_rounds"] <= rounds + 10, (rounds, st)
    assert st["ms_scan"] == pytest.approx(st["ms_total"] - st["ms_rounds"], abs=1e-6)
    for p in range(1 + st["filtered"]):
        whole, before, scan = st["us_scan"][p]
        assert before > 0 and scan > 0 and whole == pytest.approx(before + scan, rel=1e-5), st["us_scan"]
    assert sum(st["us_scan"][p][0] for p in range(2)) <= 1e3 * st["ms_scan"] + 4
    if not st["filtered"]:
        assert st["us_scan"][1] == [0, 0, 0]
