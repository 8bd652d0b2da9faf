"""The batch autotuner sets only what it can measure: degree_split changes no
kernel's work, so it stays as the caller set it."""
import pytest

import ecl_mst as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 4])
def test_autotune_leaves_the_degree_split(split):
    import torch
    b = E.Batch([E.gen_er(200 + 900 * i, 8, i, 1 << 20) for i in range(6)])
    dev = [torch.from_numpy(a).cuda() for a in (b.nindex, b.nlist, b.eweight)]
    out = torch.zeros(b.total_edges, dtype=torch.uint8, device="cuda")
    ctx = E.BatchContext(b.num_graphs, int(b.nodes.max()), int(b.edges.max()), 1 << 13)
    best, ms = ctx.autotune(b, *(d.data_ptr() for d in dev), out.data_ptr(), base=E.make_opts(degree_split=split))
    ctx.close()
    assert ms > 0 and best.batch_small_edges > 0 and best.degree_split == split
