"""The bench's byte model of the default kernels, pinned to hand-worked counts,
and (on a GPU) its kernel count per solve against the kernel nodes of the
captured launch sequence."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402
import ecl_mst as E  # noqa: E402


def _stats(wl, rounds, kept, filtered=1):
    return {"wl_real": wl, "rounds": rounds, "scan_kept": list(kept), "filtered": filtered}


def test_round_pass_bytes_by_hand():
    # one light list (two ends), one heavy list (one end): the first round of each in place
    st = _stats([[10, 10, 3], [20, 20]], [3, 2], (10, 20))
    light = (16 * 10 + 16 * 10 + 16 * 10 + 16 * 10) + (16 * 10 + 16 * 3 + 8 * 10 + 16 * 3 + 16 * 3 + 16 * 3) + 24 * 3
    heavy = (16 * 20 + 8 * 20 + 16 * 20 + 8 * 20) + 24 * 20
    assert bench.round_pass_bytes(st, 5) == light + heavy + 16 * 5
    # a second light list: compacted from its first round on, one end
    st = _stats([[4, 4, 9, 2], [0]], [4, 0], (13, 0), 0)
    first = (16 * 4 * 4) + 24 * 4
    second = (16 * 9 + 8 * 2 + 8 * 9 + 16 * 2 + 16 * 2 + 8 * 2) + 24 * 2
    assert bench.round_pass_bytes(st, 0) == first + second


def test_scan_pass_bytes_by_hand():
    n, m = 96, 1000
    light, heavy, vertex = bench.scan_pass_bytes(_stats([[7], [5, 5]], [1, 2], (7, 5)), n, m)
    assert light == 4 * 97 + 5 * m + 4 * 14 + 16 * 7
    assert heavy == 4 * 97 + 4 * m + 12 + 28 * 5
    assert vertex == 4 * 97 + 12 * n + 8 * n + 12
    # the lightest heavy entries (3 of 8) are the light scan's, and a test most entries pass reads all ids
    light, heavy, _ = bench.scan_pass_bytes(_stats([[600], [3, 5, 5]], [1, 3], (600, 8)), n, m)
    assert light == 4 * 97 + 5 * m + 4 * m + 16 * 603 and heavy == 4 * 97 + 4 * m + 12 + 28 * 5
    assert bench.scan_pass_bytes(_stats([[7], [0]], [1, 0], (7, 0), 0), n, m)[1:] == (0, 4 * 97 + 12 * n)


SOLVES = [("er", 1000, 8.0, "heuristic"), ("er", 200_000, 8.0, "learned"), ("er", 600_000, 3.0, "learned"),
          ("er", 600_000, 8.0, "none"), ("er", 600_000, 8.0, "quantile"), ("er", 600_000, 8.0, "heuristic"),
          ("er", 1_600_000, 3.0, "heuristic"), ("er", 1_000_000, 16.0, "quantile"), ("er", 1_000_000, 16.0, "none"),
          ("er", (1 << 23) + 1, 8.0, "heuristic"), ("er", (1 << 23) + 1, 8.0, "learned")]


@pytest.mark.gpu
@pytest.mark.parametrize("family,nodes,degree,mode", SOLVES)
def test_solve_launches(family, nodes, degree, mode):
    import torch
    from cuda.bindings import runtime as rt
    assert E.learned_load_default()
    modes = {"heuristic": E.THRESH_HEURISTIC, "none": E.THRESH_NONE, "quantile": E.THRESH_QUANTILE,
             "learned": E.THRESH_LEARNED}
    g = E.gen_er_device(nodes, degree, 1, 1 << 20)
    out = torch.zeros(g.edges, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    opts = E.make_opts(mode=modes[mode], quantile=0.6, flags=E.FLAG_NO_GRAPH)
    stream = torch.cuda.Stream()
    with E.Context(g.nodes, g.edges) as c:
        def solve():
            c.run_device(g.nodes, g.edges, g.d_nindex, g.d_nlist, g.d_eweight, out.data_ptr(), opts=opts,
                         stream=stream.cuda_stream)

        solve()  # uploads the weights, which a capture must not
        c.sync()
        assert rt.cudaStreamBeginCapture(stream.cuda_stream,
                                         rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == 0
        solve()
        err, graph = rt.cudaStreamEndCapture(stream.cuda_stream)
        assert err == 0
        _, _, count = rt.cudaGraphGetNodes(graph)
        _, nodes_, count = rt.cudaGraphGetNodes(graph, count)
        kinds = [rt.cudaGraphNodeGetType(x)[1] for x in nodes_[:count]]
        kernels = sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)
        rt.cudaGraphDestroy(graph)
        solve()  # (what the capture enqueued never ran)
        c.sync()
    assert kernels == bench.solve_launches(g.nodes, g.edges, mode, 0.6)
