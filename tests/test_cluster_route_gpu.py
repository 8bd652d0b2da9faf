"""Small graphs at the lines where the cluster's CTAs double and where the grid
takes over from it, by vertices and by entries, against the oracle (exact); and
a graph of many vertices and few entries, which must not be slower on the
route it takes than on the grid's."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu


def _sparse(n, edges, seed):
    """A path through `edges` random vertices of n, in random order."""
    rng = np.random.default_rng(seed)
    walk = rng.permutation(n)[:edges + 1]
    u, v, w = walk[:-1], walk[1:], rng.integers(1, 100, edges)
    src, dst, wt = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.lexsort((dst, src))
    nindex = np.zeros(n + 1, np.int64)
    np.add.at(nindex, src + 1, 1)
    return E.Graph(np.cumsum(nindex).astype(np.int32), dst[order].astype(np.int32), wt[order].astype(np.int32))


@pytest.mark.parametrize("nodes", [4096, 8192, 16384, 32768, 65536])
def test_lines(nodes):
    with E.Context(nodes + 1, 2 * nodes) as c:
        for n in (nodes, nodes + 1):
            for edges in (1, n // 10, n // 4, n // 2, n // 2 + 1, n - 1):
                g = _sparse(n, edges, n + edges)
                for kw in (dict(), dict(mode=E.THRESH_EXPLICIT, threshold=30)):
                    got, st = c.run_host(g, E.make_opts(flags=E.FLAG_NO_GRAPH, **kw))
                    want, _, _ = O.oracle_mst(g.nindex, g.nlist, g.eweight, st["threshold"], st["filtered"])
                    assert st["status"] == 0 and np.array_equal(got, want), (n, edges, kw)


@pytest.mark.parametrize("nodes", [40_000, 60_000, 65_536])
def test_few_entries_on_many_vertices(nodes):
    g = E.gen_er(nodes, 0.2, 1, 1 << 20)
    with E.Context(g.nodes, g.edges) as c:
        def ms(**kw):  # replays of the captured solve
            return c.run_host(g, E.make_opts(**kw))[1]["ms_total"]

        default = min(ms() for _ in range(12))
        grid = min(ms(ctas_per_sm=2) for _ in range(12))  # a limit on CTAs per SM: the grid's kernel
    assert default < 1.25 * grid
