"""Graphs of 2^31 - 1 vertices, the most a CSR of 32-bit ids can have, nearly all of
them isolated, by one launch and by separate ones. Leaving out the isolated
vertices keeps the entries' order, so the forest is the small graph's: against
the oracle, exact."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu

N = 2**31 - 1


@pytest.fixture(scope="module")
def ctx():
    import torch
    if torch.cuda.get_device_properties(0).total_memory < 120 << 30:
        pytest.skip("takes 90 GB")
    c = E.Context(N, 6_000_000)
    yield c
    c.close()


@pytest.mark.parametrize("nodes,degree", [(3, 2.0), (50_000, 4.0), (1_300_000, 4.0)])
def test_most_vertices(ctx, nodes, degree):
    import torch
    if nodes == 3:
        g = E.Graph([0, 2, 3, 4], [1, 2, 0, 0], [5, 4, 5, 4])
    else:
        g = E.gen_er(nodes, degree, nodes, 1 << 20)
    rng = np.random.default_rng(nodes)
    at = np.unique(np.concatenate([[0, N - 1], rng.integers(0, N, 2 * nodes)]))
    at = np.concatenate([at[:nodes - 1], [N - 1]])  # where the vertices lie
    # an isolated vertex's row starts where the next one's does
    gaps = np.diff(np.concatenate([[-1], at]))
    values = torch.from_numpy(np.append(g.nindex[:-1], g.edges).astype(np.int32)).cuda()
    nindex = torch.repeat_interleave(values, torch.from_numpy(np.append(gaps, 1)).cuda(), output_size=N + 1)
    nlist = torch.from_numpy(at[g.nlist].astype(np.int32)).cuda()
    eweight = torch.from_numpy(g.eweight).cuda()
    out = torch.zeros(g.edges, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for kw in (dict(), dict(mode=E.THRESH_QUANTILE, quantile=0.3)):
        st = ctx.run_device(N, g.edges, nindex.data_ptr(), nlist.data_ptr(), eweight.data_ptr(), out.data_ptr(),
                            opts=E.make_opts(**kw), stats=True)
        want, _, _ = O.oracle_mst(g.nindex, g.nlist, g.eweight, st["threshold"], st["filtered"])
        assert st["status"] == 0 and np.array_equal(out.cpu().numpy(), want), kw
