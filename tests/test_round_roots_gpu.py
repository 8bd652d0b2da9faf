"""The round kernel's roots pass where it takes the roots from the entries and
keeps no list for the next one (few CTAs on a second light list, whose rounds
the cluster kernel ends); against the oracle, exact."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu


def _core_and_fringe(core, pairs, fringe, links, seed):
    """A dense core of weight 1 and `fringe` vertices that only `links` heavier
    edges reach: the first light list holds the core's entries (over 98 % of
    all), the second the others, and these survive its first offer pass."""
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, core, pairs), rng.integers(0, core, pairs)
    u, v = np.concatenate([a, rng.integers(0, core + fringe, links)]), np.concatenate([b, core + np.arange(links) % fringe])
    w = np.concatenate([np.ones(pairs, np.int64), rng.integers(2, 1000, links)])
    keep = u != v
    lo, hi, w = np.minimum(u, v)[keep], np.maximum(u, v)[keep], w[keep]
    key, at = np.unique(lo * (core + fringe) + hi, return_index=True)
    lo, hi, w = key // (core + fringe), key % (core + fringe), w[at]
    src, dst, wt = np.concatenate([lo, hi]), np.concatenate([hi, lo]), np.concatenate([w, w])
    order = np.argsort(src * (core + fringe) + dst)
    nindex = np.zeros(core + fringe + 1, np.int64)
    np.add.at(nindex, src + 1, 1)
    return E.Graph(np.cumsum(nindex).astype(np.int32), dst[order].astype(np.int32), wt[order].astype(np.int32))


@pytest.mark.parametrize("links", [4200, 6000, 7300])
def test_roots_from_entries_without_a_list(links):
    g = _core_and_fringe(25_000, 3_300_000, 5_000, links, links)
    want, weight, count = O.oracle_mst(g.nindex, g.nlist, g.eweight, 2**31 - 1, 0)
    with E.Context(g.nodes, g.edges) as c:
        for _ in range(3):
            got, st = c.run_host(g, E.make_opts(mode=E.THRESH_NONE, round_min_tiles=32, flags=E.FLAG_NO_GRAPH))
            assert st["status"] == 0 and np.array_equal(got, want)
            assert st["forest_weight"] == weight and st["forest_edges"] == count
    # the second list holds the heavier entries, and what its first offer keeps
    # is for the cluster to go on with and few for the vertices
    real = st["wl_real"][0][:st["rounds"][0] + 1]
    second = real.index(int((g.eweight > 1).sum()) // 2)
    assert 4096 < real[second + 1] and 4 * real[second + 1] < g.nodes, real
