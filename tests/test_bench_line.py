"""The bench line holds figures, not a row per request: its reader may cut long
lines."""
import json

import numpy as np

import bench


def _stats(n):
    rng = np.random.default_rng(n)
    t = np.cumsum(rng.random(n))
    return [dict(submit_ms=a, start_ms=a + 1, end_ms=a + 2, beamlets=7, worker=i % 2) for i, a in enumerate(t)]


def test_served_figures_do_not_grow_with_the_requests():
    few, many = (json.dumps(bench.served_stats(_stats(n), 7 * n)) for n in (30, 300))
    assert abs(len(few) - len(many)) < 60 and "[" not in many


def test_served_timeline_has_a_row_per_request():
    rows = bench.served_timeline(_stats(30))
    assert len(rows) == 30 and rows[0][2] == 0 and all(r[3:] == [1.0, 1.0] for r in rows)
