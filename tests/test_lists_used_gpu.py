"""That the worklists split by weight are split where they should be (the solves
of test_scan_lists_gpu.py compare forests, which one list would give as well),
and a graph whose rounds run on many CTAs over several segments, on which a
segment table read too late gave 7 to 9 edges too many; against the oracle."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu


def _lists(st, phase):
    """Lists a phase ran: a list's entries only shrink, so one more begins where they grow."""
    w = st["wl_real"][phase][:st["rounds"][phase]]
    return sum(r == 0 or w[r] > w[r - 1] for r in range(len(w)))


@pytest.mark.parametrize("seed,wmax,low", [(1, 1 << 20, 0), (2, 5, 0), (3, 1 << 20, 300_000)])
def test_light_lists(seed, wmax, low):
    g = E.gen_er(1_000_000, 16.0, seed, wmax)
    g = E.Graph(g.nindex, g.nlist, g.eweight - np.int32(low))
    with E.Context(g.nodes, g.edges) as c:
        for kw, lists in ((dict(mode=E.THRESH_NONE), 2), (dict(mode=E.THRESH_QUANTILE, quantile=0.6), 2),
                          (dict(mode=E.THRESH_QUANTILE, quantile=0.05), 1)):
            _, st = c.run_host(g, E.make_opts(flags=E.FLAG_NO_GRAPH, **kw))
            # (quantile 0.05 of five weights keeps a fifth of 8M entries: under the 3M a split takes)
            assert st["status"] == 0 and _lists(st, 0) == lists, (kw, st["wl_real"][0], st["rounds"])


def test_mid_list():
    g = E.gen_er_device((1 << 23) + 5, 12.0, 4, 1 << 30)
    out = np.zeros(g.edges, np.uint8)
    h = g.to_host()
    with E.Context(g.nodes, g.edges) as c:
        _, st = c.run_host(h, E.make_opts(mode=E.THRESH_QUANTILE, quantile=0.1, flags=E.FLAG_NO_GRAPH), out=out)
    assert st["status"] == 0 and _lists(st, 1) == 2, (st["wl_real"][1], st["rounds"])


def test_rounds_of_many_segments():
    g = E.gen_er_device(3_400_000, 32.0, 5, 1 << 20)
    h = g.to_host()
    want, total, count = O.oracle_mst(h.nindex, h.nlist, h.eweight, 87377, 1)
    with E.Context(g.nodes, g.edges) as c:
        for _ in range(8):
            got, st = c.run_host(h, E.make_opts(mode=E.THRESH_EXPLICIT, threshold=87377))
            assert st["status"] == 0 and st["forest_edges"] == count and st["forest_weight"] == total
            assert np.array_equal(got, want)
