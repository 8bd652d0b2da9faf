"""The cluster kernel that ends a list takes over the grid's segments: every CTA
reads them before one of them, which may have no entries of the first round,
publishes its own. Solves whose list comes over with so few entries that some
CTAs have none (4097 to 7168), on four streams at once, whose kernels start each
other's CTAs late; against the oracle, exact."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu

TAIL, SOLO, TILE, CTAS = 32768, 4096, 1024, 8


def _idle_ctas(st):
    """Lists that came over with entries for some of the cluster's CTAs, but not all."""
    n = 0
    for p in range(2):
        w = st["wl_real"][p][:st["rounds"][p]]
        n += sum(0 < r and w[r - 1] > TAIL and SOLO < w[r] <= (CTAS - 1) * TILE for r in range(len(w)))
    return n


def test_few_entries_for_the_cluster():
    import torch
    assert E.learned_load_default()  # with the network's schedule, graphs of 2^20 entries take these kernels
    opts = E.make_opts(mode=E.THRESH_LEARNED, flags=E.FLAG_NO_GRAPH)
    graphs, hits = [], 0
    for i in range(24):
        n = 135_000 + 7000 * i
        d = E.gen_er_device(n, 8.0 + 2 * (i % 3), i, 1 << 20) if i % 2 else E.gen_rmat_device(16 + i % 4 // 2, 16, .57, .19, .19,
                                                                                           i, 1 << 20)
        h = d.to_host()
        ctx = E.Context(d.nodes, d.edges)
        out = torch.zeros(d.edges, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        st = ctx.run_device(d.nodes, d.edges, d.d_nindex, d.d_nlist, d.d_eweight, out.data_ptr(), opts=opts, stats=True)
        hits += _idle_ctas(st)
        want, _, _ = O.oracle_mst(h.nindex, h.nlist, h.eweight, st["threshold"], st["filtered"])
        graphs.append((d, ctx, out, torch.from_numpy(want).cuda()))
    assert hits >= 2, hits
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    for rep in range(30):
        for k, (d, ctx, out, _) in enumerate(graphs):
            ctx.run_device(d.nodes, d.edges, d.d_nindex, d.d_nlist, d.d_eweight, out.data_ptr(), opts=opts,
                           stream=streams[(k + rep) % 4].cuda_stream)
        for d, ctx, out, want in graphs:
            ctx.sync()
            assert torch.equal(out, want), (rep, d.nodes)
    for d, ctx, _, _ in graphs:
        ctx.close()
        d.close()
