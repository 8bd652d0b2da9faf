"""Runs of empty rows (isolated vertices) between a scan thread's entries: short
ones at the step where the row search changes over, and long ones, whose
solve must not take a step per row. One graph per route of the solve (one
cluster, one grid, dense tasks of the light scan) and in a batch; against the
oracle, exact."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu

# vertices of the Erdos-Renyi graph (8 entries each) and options, by route
ROUTES = {"cluster": (4000, {}), "group": (30_000, {}), "dense": (700_000, dict(mode=E.THRESH_NONE))}


def _spread(g, before):
    """g with before[v] empty rows put in before vertex v."""
    at = np.arange(g.nodes) + np.cumsum(before)
    starts = np.full(int(at[-1]) + 2, -1, np.int64)
    starts[at] = g.nindex[:-1]
    starts[-1] = g.edges
    rows = np.where(starts >= 0, np.arange(len(starts)), len(starts))
    nindex = starts[np.minimum.accumulate(rows[::-1])[::-1]]  # an empty row starts where the next one does
    return E.Graph(nindex.astype(np.int32), at[g.nlist].astype(np.int32), g.eweight)


def _long_run(g, rows):
    """`rows` empty rows before a vertex whose entries start inside a thread's four."""
    v = next(v for v in range(g.nodes // 2, g.nodes) if g.nindex[v] % 4 and g.nindex[v] < g.nindex[v + 1])
    before = np.zeros(g.nodes, np.int64)
    before[v] = rows
    return _spread(g, before)


def _solve(ctx, g, kw):
    got, st = ctx.run_host(g, E.make_opts(flags=E.FLAG_NO_GRAPH, **kw))
    want, weight, _ = O.oracle_mst(g.nindex, g.nlist, g.eweight, st["threshold"], st["filtered"])
    assert st["status"] == 0 and np.array_equal(got, want) and st["forest_weight"] == weight
    return st["ms_total"]


@pytest.mark.parametrize("route", ROUTES)
def test_short_runs(route):
    n, kw = ROUTES[route]
    rng = np.random.default_rng(n)
    g = _spread(E.gen_er(n, 8.0, 3, 1 << 20), rng.choice([0, 0, 0, 1, 3, 4, 5, 6, 7, 40], n))
    with E.Context(g.nodes, g.edges) as c:
        _solve(c, g, kw)


# A row per step costs 35 cycles of L1 latency at least: 1 ms per 56 000 rows and scan at 1965 MHz.
@pytest.mark.parametrize("route,rows,limit_ms", [("cluster", 60_000, 1.0), ("group", 1_000_000, 5.0),
                                                 ("dense", 1_000_000, 5.0)])
def test_long_runs(route, rows, limit_ms):
    n, kw = ROUTES[route]
    g = _long_run(E.gen_er(n, 8.0, 5, 1 << 20), rows)
    with E.Context(g.nodes, g.edges) as c:
        assert min(_solve(c, g, kw) for _ in range(3)) < limit_ms


def test_long_run_in_a_batch():
    import torch
    g = _long_run(E.gen_er(4000, 8.0, 7, 1 << 20), 500_000)
    b = E.Batch([g])
    dev = [torch.from_numpy(a).cuda() for a in (b.nindex, b.nlist, b.eweight)]
    out = torch.zeros(b.total_edges, dtype=torch.uint8, device="cuda")
    ctx = E.BatchContext(1, g.nodes, g.edges)
    ms = min(ctx.run(b, *(d.data_ptr() for d in dev), out.data_ptr())["ms_small"] for _ in range(3))
    ctx.close()
    want, _, _ = O.oracle_mst(g.nindex, g.nlist, g.eweight, *E.heuristic_threshold(g))
    assert np.array_equal(b.slice(out.cpu().numpy(), 0), want)
    assert ms < 5.0
