"""A batch's mid-size graphs, solved by teams of CTAs side by side, down to
graphs of a few entries and at the edges of a team's tiles, next to larger ones
that the engines solve; against the oracle, exact."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu


def _graphs():
    gs = [E.gen_rgg2d(n, 3, 50 + n, 1 << 20) for n in (60, 700, 5000)]
    gs += [E.gen_grid(2, k, k, 9) for k in (5, 341, 342, 343, 20_000)]  # 3k - 2 edges: 2048 entries between
    gs += [E.gen_er(n, 8, n, 1 << 20) for n in (300, 40_000)]
    gs += [E.gen_rmat(s, 8, 0.57, 0.19, 0.19, s, 1 << 20) for s in (8, 13, 16, 17)]
    n = 200_000  # many vertices, no entry
    gs.append(E.Graph(np.zeros(n + 1, np.int32), np.zeros(0, np.int32), np.zeros(0, np.int32)))
    return gs


@pytest.mark.parametrize("large", [0, 2])
@pytest.mark.parametrize("streams", [0, 2, 8])
def test_teams(streams, large):
    import torch
    gs = _graphs() + [E.gen_rmat(18, 8, 0.57, 0.19, 0.19, 90 + i, 1 << 20) for i in range(large)]
    wants = [O.oracle_mst(g.nindex, g.nlist, g.eweight, *(E.heuristic_threshold(g) if g.edges else (2**31 - 1, 0)))[0]
             for g in gs]
    b = E.Batch(gs)
    ni, nl, ew = (torch.from_numpy(a).cuda() for a in (b.nindex, b.nlist, b.eweight))
    out = torch.zeros(b.total_edges, dtype=torch.uint8, device="cuda")
    ctx = E.BatchContext(len(gs), max(g.nodes for g in gs), max(g.edges for g in gs), 64)
    bad = nl.clone()
    bad[int(b.edge_off[8]) + 5] = 1 << 30  # an id out of range in one graph of the batch
    for kw in (dict(), dict(mode=E.THRESH_NONE), dict(mode=E.THRESH_QUANTILE, quantile=0.2, ctas_per_sm=1),
               dict(mode=E.THRESH_LEARNED)):
        opts = E.make_opts(batch_large_streams=streams, **kw)
        with pytest.raises(E.EclError):
            ctx.run(b, ni.data_ptr(), bad.data_ptr(), ew.data_ptr(), out.data_ptr(), opts=opts)
        for _ in range(2):
            out.fill_(3)
            st = ctx.run(b, ni.data_ptr(), nl.data_ptr(), ew.data_ptr(), out.data_ptr(), opts=opts)
            got = out.cpu().numpy()
            assert st["status"] == 0 and st["graphs_large"] >= len(gs) - 1
            for i, want in enumerate(wants):
                assert np.array_equal(b.slice(got, i), want), (kw, i)
    ctx.close()
