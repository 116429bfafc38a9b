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


def test_large_requests_within_a_small_budget(lg, inst):
    """A budget without room for a large request's neighbour lists holds the
    request without them: it is charged what it takes and need not wait for the
    others to end."""
    n = 7000
    xy = inst.uniform_f32(n, 81, 1.0e5)
    r = lg.nn_tour(xy)
    small = inst.uniform_f32(4000, 82, 1.0e5)
    rs = inst.random_tour(4000, 83)
    with lg.Solver(xy) as s:
        want, st = s.ils(r, 3, 5, lg.KICK_SEGMENT)
    budget = 92 * n + 3 * 16 * 4000
    with lg.Server(kicks=3, mem_budget=budget, quantum_pairs=100_000) as srv:
        busy = [srv.submit(small, rs, k) for k in range(2)]
        rid = srv.submit(xy, r, 5)
        seen = set()
        while True:
            info = srv.stats()
            assert info["mem_in_use"] <= budget
            if info["running_large"]:
                seen.add((info["mem_in_use"], info["running_small"]))
            got = srv.poll(rid)
            if got is not None:
                break
        for k in busy:
            srv.wait(k)
    assert got[1]["status"] == 0 and got[1]["best_length"] == st["final_length"]
    assert got[1]["moves"] == st["moves"] and np.array_equal(got[0], want)
    # beside the small requests that came first
    assert (92 * n + 2 * 16 * 4000, 2) in seen, seen
