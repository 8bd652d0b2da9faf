"""Batches of graphs with many vertices and few edges, beside dense and tiny
ones: every size of cluster and scratch in one call, also where the scratch is
too small for all clusters at once, against the oracle (exact); and the time of
graphs just too large for one CTA's shared memory."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu


def _random(n, pairs, seed):
    """A graph of exactly 2 x `pairs` entries."""
    rng = np.random.default_rng(seed)
    key = np.zeros(0, np.int64)
    while len(key) < pairs:
        u, v = rng.integers(0, n, 2 * pairs), rng.integers(0, n, 2 * pairs)
        lo, hi = np.minimum(u, v), np.maximum(u, v)
        key = np.unique(np.concatenate([key, (lo * n + hi)[lo < hi]]))
    key = rng.permutation(key)[:pairs]
    u, v, w = key // n, key % n, rng.integers(1, 1000, pairs)
    src, dst, wt = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.lexsort((dst, src))
    nindex = np.zeros(n + 1, np.int64)
    np.add.at(nindex, src + 1, 1)
    return E.Graph(np.cumsum(nindex).astype(np.int32), dst[order].astype(np.int32), wt[order].astype(np.int32))


def _run(graphs, opts=None, small_cap=0, reps=2, check=True):
    import torch
    b = E.Batch(graphs)
    dev = [torch.from_numpy(a).cuda() for a in (b.nindex, b.nlist, b.eweight)]
    out = torch.zeros(b.total_edges, dtype=torch.uint8, device="cuda")
    ctx = E.BatchContext(b.num_graphs, int(b.nodes.max()), int(b.edges.max()), small_cap)
    ms = []
    for _ in range(reps):
        st = ctx.run(b, *(d.data_ptr() for d in dev), out.data_ptr(), opts=opts)
        assert st["status"] == 0
        ms.append(st["ms_small"])
    ctx.close()
    if check:
        host, known = out.cpu().numpy(), {}
        for i, g in enumerate(graphs):
            if id(g) not in known:
                mode = opts.threshold_mode if opts else E.THRESH_HEURISTIC
                t, f = E.heuristic_threshold(g) if mode == E.THRESH_HEURISTIC else (opts.threshold, 1)
                known[id(g)] = O.oracle_mst(g.nindex, g.nlist, g.eweight, t, f)[0]
            assert np.array_equal(b.slice(host, i), known[id(g)]), (i, g.nodes, g.edges)
    return min(ms)


@pytest.mark.parametrize("explicit", [False, True])
@pytest.mark.parametrize("count", [1, 3, 40, 160])
def test_sizes(count, explicit):
    """One kind of graph at a time (its share of the chip follows from the count)."""
    opts = E.make_opts(mode=E.THRESH_EXPLICIT, threshold=300) if explicit else None
    for n in (16_384, 16_385, 40_000):
        for pairs in (1, n // 40, n // 8, n // 8 + 1, n, 4 * n if count < 40 else 2 * n):
            _run([_random(n, pairs, n + pairs)] * count, opts)


def test_all_sizes_in_little_scratch():
    dense, held = _random(5000, 10_000, 1), _random(4000, 9500, 2)
    sparse, wide, tiny = _random(16_385, 30, 3), _random(19_000, 30, 4), _random(10, 9, 5)
    _run([dense] * 160 + [sparse] * 150 + [wide, held] + [tiny] * 150, small_cap=20_000)


def test_sparse_graphs_beyond_one_ctas_shared_memory():
    """6 % more vertices must not double the batch's time."""
    inside = _run([_random(16_000, 1000, 6)] * 400, reps=6, check=False)
    beyond = _run([_random(17_000, 1000, 7)] * 400, reps=6, check=False)
    assert beyond < 1.6 * inside, (inside, beyond)
