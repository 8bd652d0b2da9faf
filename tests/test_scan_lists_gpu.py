"""The CSR scans at the edges of their 512-entry tasks (ragged ends, a row over
several tasks, tasks of more rows than are looked at one by one, unaligned
arrays, dense and sparse light phases) and the worklists split by weight, one
engine for graphs of every kind, against the oracle. Whole numbers: exact."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = E.Context(1 << 20, 1 << 25)
    yield c
    c.close()


def _csr(n, u, v, w):
    src, dst, wt = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.lexsort((dst, src))
    nindex = np.zeros(n + 1, np.int64)
    np.add.at(nindex, src + 1, 1)
    return E.Graph(np.cumsum(nindex).astype(np.int32), dst[order].astype(np.int32), wt[order].astype(np.int32))


def _small(kind, edges):
    """`edges` undirected edges (2 x edges entries)."""
    rng = np.random.default_rng(edges)
    k = np.arange(edges)
    if kind == "path":
        n, u, v = edges + 1, k, k + 1
    elif kind == "star":  # one row over all tasks, the others of one entry
        n, u, v = edges + 1, np.zeros(edges, np.int64), k + 1
    else:  # pairs far apart: hundreds of empty rows to a task
        n, u, v = 40 * edges + 2, 40 * k, 40 * k + 1 + rng.integers(0, 39, edges)
    return _csr(n, u, v, rng.integers(-3 if kind == "path" else 0, 50, edges))


@pytest.mark.parametrize("edges", [1, 255, 256, 257, 511, 513, 4099])
@pytest.mark.parametrize("kind", ["path", "star", "gaps"])
def test_scan_tasks(ctx, kind, edges):
    import torch
    g = _small(kind, edges)
    for shift in (0, 1):
        dev = [torch.zeros(len(a) + shift, dtype=torch.int32, device="cuda") for a in (g.nindex, g.nlist, g.eweight)]
        for d, a in zip(dev, (g.nindex, g.nlist, g.eweight)):
            d[shift:] = torch.from_numpy(a).cuda()
        for kw in (dict(mode=E.THRESH_NONE), dict(mode=E.THRESH_EXPLICIT, threshold=2),
                   dict(mode=E.THRESH_EXPLICIT, threshold=30)):
            out = torch.full((g.edges + 2,), 7, dtype=torch.uint8, device="cuda")
            # a round variant, so that a small graph takes the scans' route
            st = ctx.run_device(g.nodes, g.edges, *(d[shift:].data_ptr() for d in dev), out[1:].data_ptr(),
                                opts=E.make_opts(flags=E.FLAG_NO_FIND_CACHE, **kw), stats=True)
            want, _, _ = O.oracle_mst(g.nindex, g.nlist, g.eweight, st["threshold"], st["filtered"])
            got = out.cpu().numpy()
            assert got[0] == 7 and got[-1] == 7 and np.array_equal(got[1:-1], want), (shift, kw)


def test_split_lists(ctx):
    """Lists light 0 and 1 (all, or 0.6 of 8M entries in the light phase), then
    single lists again on the same engine, ties and negative weights among them."""
    for seed, wmax, low in ((1, 1 << 20, 0), (2, 5, 0), (3, 1 << 20, 300_000)):
        g = E.gen_er(1_000_000, 16.0, seed, wmax)
        w = g.eweight - np.int32(low)
        g = E.Graph(g.nindex, g.nlist, w)
        for kw in (dict(mode=E.THRESH_NONE), dict(mode=E.THRESH_QUANTILE, quantile=0.6), dict()):
            got, st = ctx.run_host(g, E.make_opts(**kw))
            want, total, count = O.oracle_mst(g.nindex, g.nlist, g.eweight, st["threshold"], st["filtered"])
            assert st["status"] == 0 and np.array_equal(got, want), (seed, kw)
            assert st["forest_weight"] == total and st["forest_edges"] == count


def test_split_lists_mid():
    """The list of the lightest heavy entries, from 2^23 vertices on."""
    d = E.gen_er_device((1 << 23) + 5, 12.0, 4, 1 << 30)
    g = d.to_host()
    with E.Context(g.nodes, g.edges) as c:
        got, st = c.run_host(g, E.make_opts(mode=E.THRESH_QUANTILE, quantile=0.1))
    want, total, _ = O.oracle_mst(g.nindex, g.nlist, g.eweight, st["threshold"], st["filtered"])
    assert st["status"] == 0 and np.array_equal(got, want) and st["forest_weight"] == total
