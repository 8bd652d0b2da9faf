"""The work a user of this library has it do, as measurable cases.

Every case goes through the public Python binding of the C ABI. Graphs are
drawn on the GPU by the library's own seeded generators, so a seed fixes the
inputs. Outputs are the solve's per-entry inMST bytes (or the CSR arrays of a
graph build): whole numbers, equal for every schedule, so there is no rounding
to bound.

  solve     one device-resident graph through a reusable context, enqueued on
            one stream (the program goes on without waiting)
  noalloc   the allocation-free entry point, which returns after the solve
  oneshot   host CSR in, host inMST out, own workspace per call (the drop-in
            for the reference's gpuMST)
  batch     many independent graphs of uneven sizes in one call
  pairs     an undirected weighted pair list built into a CSR on the device

The entry counts of random graphs vary with the seed; result buffers are the
program's own and are sized for the largest graph its parameters give.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mst-artifact-sc23_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ecl_mst as E  # noqa: E402

_MODES = {"heuristic": E.THRESH_HEURISTIC, "none": E.THRESH_NONE, "quantile": E.THRESH_QUANTILE,
          "learned": E.THRESH_LEARNED}
_stream = None


def _work_stream():
    """The one stream the device-resident solves are enqueued on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
        E.learned_load_default()
    return _stream


def listed():
    return [
        # the smallest call: a service that may not allocate solves a graph of
        # a thousand vertices and waits for it (latency of the whole call)
        {"name": "noalloc_er1k", "kind": "noalloc", "family": "er", "nodes": 1000, "degree": 8.0, "wmax": 1 << 20,
         "mode": "heuristic"},
        # a small power-law graph with default options
        {"name": "rmat14", "kind": "solve", "family": "rmat", "scale": 14, "ef": 16, "wmax": 1 << 24,
         "mode": "heuristic"},
        # 1000 x 1000 four-neighbour grid: long-diameter mesh, many rounds
        {"name": "grid1000", "kind": "solve", "family": "grid", "rows": 1000, "cols": 1000, "wmax": 1_000_000,
         "mode": "heuristic"},
        # sparse random geometric graph (average degree 3, many components),
        # an odd vertex count, learned schedule
        {"name": "rgg_777k", "kind": "solve", "family": "rgg", "nodes": 777_777, "degree": 3.0, "wmax": 1 << 20,
         "mode": "learned"},
        # an ordinary sparse random graph, odd size, default options
        {"name": "er_3m", "kind": "solve", "family": "er", "nodes": 3_000_001, "degree": 8.0, "wmax": 1 << 20,
         "mode": "heuristic"},
        # the headline configuration: RMAT scale 22, learned schedule
        {"name": "rmat22", "kind": "solve", "family": "rmat", "scale": 22, "ef": 16, "wmax": 1 << 24,
         "mode": "learned"},
        # the large configurations: half a billion and a billion entries
        {"name": "er16m", "kind": "solve", "family": "er", "nodes": 1 << 24, "degree": 32.0, "wmax": 1 << 30,
         "mode": "learned"},
        {"name": "rmat25", "kind": "solve", "family": "rmat", "scale": 25, "ef": 16, "wmax": 1 << 30,
         "mode": "learned"},
        # a batch of small graphs, each solved by one CTA
        {"name": "batch_small", "kind": "batch", "count": 400, "nmin": 1000, "nmax": 60_000, "mode": "heuristic",
         "streams": 0, "ctas": 0, "cutoff": 0},
        # the mixed batch: sizes over three decades, the large graphs on
        # concurrent streams (the setting the autotuner picks for it)
        {"name": "batch_mixed", "kind": "batch", "count": 96, "nmin": 1000, "nmax": 2_000_000, "mode": "learned",
         "streams": 8, "ctas": 1, "cutoff": 1 << 19},
        # drop-in call on host arrays: workspace, copies and solve every time
        {"name": "oneshot_rmat16", "kind": "oneshot", "family": "rmat", "scale": 16, "ef": 16, "wmax": 1 << 24,
         "mode": "heuristic"},
        # graph construction from a pair list with given weights
        {"name": "pairs_5m", "kind": "pairs", "nodes": 1_000_003, "pairs": 5_000_011},
    ]


def _log_int(rng, lo, hi):
    return int(round(2 ** rng.uniform(_log2(lo), _log2(hi))))


def _log2(x):
    return math.log2(x)


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "noalloc", "oneshot", "batch", "batch", "pairs"])
    if kind == "batch":
        small = rng.random() < 0.5
        return {"kind": "batch", "count": rng.randint(16, 400 if small else 96), "nmin": 1000,
                "nmax": _log_int(rng, 4000, 100_000) if small else _log_int(rng, 200_000, 2_000_000),
                "mode": rng.choice(["heuristic", "learned"]), "streams": rng.choice([0, 4, 8]),
                "ctas": rng.choice([0, 1]), "cutoff": rng.choice([0, 1 << 19])}
    if kind == "pairs":
        n = _log_int(rng, 1000, 8_000_000)
        return {"kind": "pairs", "nodes": n, "pairs": _log_int(rng, 2 * n, min(16 * n, 50_000_000) + 1)}
    # the allocation-free entry point takes at most 2^18 vertices and 2^20 entries
    top = {"solve": 8_000_000, "noalloc": 100_000, "oneshot": 300_000}[kind]
    case = {"kind": kind, "family": rng.choice(["er", "rmat", "grid", "rgg"]),
            "wmax": rng.choice([1 << 20, 1 << 24, 1 << 30])}
    n = _log_int(rng, 1000, top)
    if case["family"] == "rmat":
        case["scale"] = max(10, int(_log2(n)))
        case["ef"] = 4 if kind == "noalloc" else rng.choice([8, 16, 32])
    elif case["family"] == "grid":
        case["rows"] = max(2, int(n ** rng.uniform(0.3, 0.6)))
        case["cols"] = max(2, n // case["rows"])
    else:
        case["nodes"] = n
        case["degree"] = 3.0 if case["family"] == "rgg" else rng.choice([4.0, 8.0] if kind == "noalloc"
                                                                        else [4.0, 8.0, 16.0, 32.0])
    case["mode"] = rng.choice(["heuristic", "heuristic", "learned", "quantile", "none"])
    if case["mode"] == "quantile":
        case["quantile"] = round(rng.uniform(0.02, 0.5), 3)
    return case


def _graph(case, seed):
    f = case["family"]
    if f == "rmat":
        return E.gen_rmat_device(case["scale"], case["ef"], 0.57, 0.19, 0.19, seed, case["wmax"])
    if f == "er":
        return E.gen_er_device(case["nodes"], case["degree"], seed, case["wmax"])
    if f == "grid":
        return E.gen_grid_device(case["rows"], case["cols"], seed, case["wmax"])
    return E.gen_rgg2d_device(case["nodes"], case["degree"], seed, case["wmax"])


def prepare(case, seed):
    _work_stream()
    kind = case["kind"]
    if kind == "pairs":
        g = torch.Generator(device="cuda").manual_seed(seed)

        def ints(lo, hi):
            return torch.randint(lo, hi, (case["pairs"],), generator=g, device="cuda", dtype=torch.int32)

        room = 2 * case["pairs"]  # both directions of every pair
        return {"kind": kind, "nodes": case["nodes"], "pairs": case["pairs"], "u": ints(0, case["nodes"]),
                "v": ints(0, case["nodes"]), "w": ints(1, 1 << 24),
                "nindex": torch.zeros(case["nodes"] + 1, dtype=torch.int32, device="cuda"),
                "nlist": torch.zeros(room, dtype=torch.int32, device="cuda"),
                "eweight": torch.zeros(room, dtype=torch.int32, device="cuda")}
    if kind == "batch":
        b = E.DeviceBatch(case["count"], seed0=seed * 4096 + 1, nmin=case["nmin"], nmax=case["nmax"])
        opts = E.make_opts(mode=_MODES[case["mode"]], ctas_per_sm=case["ctas"], batch_large_streams=case["streams"])
        opts.batch_small_edges = case["cutoff"]
        ctx = E.BatchContext(b.num_graphs, int(b.nodes.max()), int(b.edges.max()))
        out = torch.zeros(_out_bytes(case), dtype=torch.uint8, device="cuda")
        assert b.total_edges <= out.numel()
        return {"kind": kind, "batch": b, "ctx": ctx, "opts": opts, "out": out}
    g = _graph(case, seed)
    opts = E.make_opts(mode=_MODES[case["mode"]], quantile=case.get("quantile", 1.0))
    assert g.edges <= _out_bytes(case)
    if kind == "oneshot":
        return {"kind": kind, "graph": g.to_host(), "opts": opts, "out": np.zeros(_out_bytes(case), np.uint8)}
    out = torch.zeros(_out_bytes(case), dtype=torch.uint8, device="cuda")
    state = {"kind": kind, "graph": g, "opts": opts, "out": out}
    if kind == "solve":
        state["ctx"] = E.Context(g.nodes, g.edges)
    return state


def _out_bytes(case):
    """inMST bytes of the largest graph (or batch) the case's parameters give:
    Erdos-Renyi and RMAT at most two entries per sample, the geometric graph
    well under twice its mean, a batch six deviations over its mean."""
    if case["kind"] == "batch":
        spread = 6.0 * math.sqrt(case["count"]) * case["nmax"] * 16 / 5
        return int(_batch_nodes(case) * 20 / 3 + spread)
    n, m = _mean_entries(case)
    return int(2 * m + 4096 if case["family"] == "rgg" else m + 2)


class _DeviceArray:
    """A device array of a DeviceGraph, as torch takes it (keeps the graph alive)."""

    def __init__(self, graph, ptr, count):
        self._graph = graph
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (ptr, False), "version": 2}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        g, out = state["graph"], state["out"]
        state["ctx"].run_device(g.nodes, g.edges, g.d_nindex, g.d_nlist, g.d_eweight, out.data_ptr(),
                                opts=state["opts"], stream=_stream.cuda_stream)
        return out
    if kind == "noalloc":
        g, out = state["graph"], state["out"]
        E.run_device_noalloc(g.nodes, g.edges, g.d_nindex, g.d_nlist, g.d_eweight, out.data_ptr(),
                             opts=state["opts"], stream=_stream.cuda_stream)
        return out
    if kind == "oneshot":
        got, out = E.mst(state["graph"], opts=state["opts"])[0], state["out"]
        out[:got.size] = got
        return out
    if kind == "batch":
        b, out = state["batch"], state["out"]
        state["ctx"].run(b, b.d_nindex, b.d_nlist, b.d_eweight, out.data_ptr(), opts=state["opts"],
                         stream=_stream.cuda_stream)
        return out
    # the program copies the built CSR into its own arrays and lets the graph go
    g = E.csr_from_pairs_device(state["nodes"], state["pairs"], state["u"].data_ptr(), state["v"].data_ptr(),
                                state["w"].data_ptr(), rule=E.WEIGHTS_GIVEN, stream=_stream.cuda_stream)
    outs = [state["nindex"], state["nlist"], state["eweight"]]
    with torch.cuda.stream(_stream):
        for dst, ptr, count in zip(outs, (g.d_nindex, g.d_nlist, g.d_eweight), (g.nodes + 1, g.edges, g.edges)):
            dst[:count].copy_(torch.as_tensor(_DeviceArray(g, ptr, count), device="cuda"))
    return outs


def _mean_entries(case):
    """CSR entries of a case's graph, from its family's parameters (the
    generators drop duplicates and self-loops, so this is a little high)."""
    f = case["family"]
    if f == "rmat":
        return (1 << case["scale"]), 2.0 * case["ef"] * (1 << case["scale"])
    if f == "grid":
        r, c = case["rows"], case["cols"]
        return r * c, 2.0 * (r * (c - 1) + c * (r - 1))
    return case["nodes"], case["degree"] * case["nodes"]


def _batch_nodes(case):
    """Expected vertices of a batch (counts log-uniform in [nmin, nmax])."""
    lo, hi = case["nmin"], case["nmax"]
    return case["count"] * (hi - lo) / math.log(hi / lo)


def work(case):
    """Bytes a pass cannot do without: the CSR read once (nindex 4 (n + 1),
    nlist and eweight 4 each per entry) and one inMST byte written per entry;
    a graph build reads its pairs and writes the CSR. No floating point."""
    if case["kind"] == "pairs":
        n, p = case["nodes"], case["pairs"]
        return {"bytes": 12.0 * p + 4.0 * (n + 1) + 16.0 * p, "flops": 0.0}
    if case["kind"] == "batch":
        # families uniform: grid 4, Erdos-Renyi 8, RMAT 16 (2^floor(log2 n)
        # vertices, about 0.72 n), geometric 3 entries per vertex
        n = _batch_nodes(case)
        return {"bytes": 9.0 * n * (4 + 8 + 0.72 * 16 + 3) / 4 + 4.0 * n, "flops": 0.0}
    n, m = _mean_entries(case)
    return {"bytes": 9.0 * m + 4.0 * (n + 1), "flops": 0.0}
