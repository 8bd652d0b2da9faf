"""A label sweep solves a graph once per quantile (no kernel's work depends on
the degree split, the tables' second axis) and once with the heuristic. No GPU:
the solve is a stand-in."""
import numpy as np

import train_filter as TF


class _Graph:
    nodes, edges, d_nindex, d_nlist, d_eweight = 10, 40, 0, 0, 0


def test_one_solve_per_quantile(monkeypatch):
    seen = []

    def solve(ctx, dg, out, opts, reps):
        seen.append((opts.threshold_mode, round(float(opts.quantile), 4)))
        return float(len(seen))

    monkeypatch.setattr(TF, "solve_ms", solve)
    monkeypatch.setattr(TF.E, "graph_features", lambda *a: np.zeros(16, np.float32))
    _, times, heur = TF.sweep(None, _Graph, None, 2)
    assert seen == [(TF.E.THRESH_QUANTILE, q) for q in TF.QUANTILES] + [(TF.E.THRESH_HEURISTIC, 1.0)]
    assert times.shape == (len(TF.QUANTILES), len(TF.SPLITS)) and heur == len(seen)
    assert np.array_equal(times, np.repeat(np.arange(1.0, len(TF.QUANTILES) + 1)[:, None], len(TF.SPLITS), 1))
