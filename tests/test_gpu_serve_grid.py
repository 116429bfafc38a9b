"""Requests that run as grid-wide launches (above 6,144 cities) beside rounds of
smaller ones: they take turns on the device, and no result depends on it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_grid_wide_requests_and_rounds(lg, inst):
    reqs = []
    for k, n in enumerate((7000, 300, 3500, 6145, 1200, 40, 9000, 4096)):
        xy = inst.uniform_f32(n, 60 + k, 1.0e5) if k % 2 else inst.clustered(n, 60 + k)
        reqs.append((xy, lg.nn_tour(xy), 70 + k))
    with lg.Server(kicks=6, quantum_pairs=3_000_000) as srv:
        ids = [srv.submit(*q) for q in reqs + reqs]
        got = [srv.wait(i) for i in ids]
    for k, (xy, r, seed) in enumerate(reqs):
        with lg.Solver(xy) as s:
            want, st = s.ils(r, 6, seed, lg.KICK_SEGMENT)
        for route, info in (got[k], got[k + len(reqs)]):
            assert info["status"] == 0 and info["best_length"] == st["final_length"]
            assert info["moves"] == st["moves"] and np.array_equal(route, want)
