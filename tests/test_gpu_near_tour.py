"""The near-neighbour sweep of a CTA-resident tour (near_tour.cuh) against the
oracle, where its lists, cells and discs can go wrong: fewer cities than list
entries, around multiples of a warp and of a list, the largest instance; many
cities on one point, on a line, in far-apart clumps, far from the origin.
Everything compared is a whole number, so the tolerance is zero."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [3, 4, 5, 7, 8, 9, 16, 17, 18, 31, 32, 33, 63, 65, 127, 129, 255, 257, 500, 513]


def points(inst, kind, n, seed):
    xy = inst.uniform_f32(n, seed, 1.0e4)
    if kind == "line":
        xy[:, 1] = 7.0
    elif kind == "column":
        xy[:, 0] = np.float32(-3.5)
    elif kind == "heaps":  # most cities share one of five points
        xy = np.ascontiguousarray(xy[np.arange(n) % min(n, 5)])
        xy[::7] += np.float32(1.0)
    elif kind == "clumps":
        xy = xy * np.float32(0.001)
        xy[::2] += np.float32(1.2e6)
    elif kind == "offset":
        xy = xy + np.float32(1.0e8)
    elif kind == "lattice":  # ties everywhere
        side = int(np.ceil(np.sqrt(n)))
        k = np.arange(n)
        xy = np.stack([10.0 * (k % side), 10.0 * (k // side)], axis=1).astype(np.float32)
    return np.ascontiguousarray(xy)


def check(lg, oracle_mod, xs, rs, seeds, kicks, kind, **kw):
    want, want_len, want_moves = oracle_mod.ils_batch(xs, rs, seeds, kicks, kind,
                                                      threads=os.cpu_count() or 4)
    with lg.Batch(len(xs), sum(len(r) for r in rs)) as b:
        got, res, _ = b.solve(xs, rs, seeds, kicks=kicks, kind=kind, **kw)
    for k in range(len(xs)):
        assert res[k]["status"] == 0
        assert res[k]["best_length"] == want_len[k], (k, len(rs[k]))
        assert res[k]["moves"] == want_moves[k], (k, len(rs[k]))
        assert np.array_equal(got[k], want[k]), (k, len(rs[k]))


@pytest.mark.parametrize("kind", ["uniform", "line", "column", "heaps", "clumps", "offset",
                                  "lattice"])
def test_points_of_every_shape(lg, inst, oracle_mod, kind):
    xs = [points(inst, kind, n, 900 + n) for n in SIZES]
    rs = [inst.random_tour(n, 70 + n) for n in SIZES]
    check(lg, oracle_mod, xs, rs, [5 + n for n in SIZES], 4, 0)
    check(lg, oracle_mod, xs, rs, [6 + n for n in SIZES], 4, 1, shape=(4, 256, 64))


def test_largest_instance(lg, inst, oracle_mod):
    xy = inst.clustered(4096, 2, clusters=20, sigma_frac=0.03)
    check(lg, oracle_mod, [xy], [lg.nn_tour(xy)], [9], 1, 1)


@pytest.mark.parametrize("kind", ["uniform", "line", "heaps", "clumps", "offset", "lattice"])
@pytest.mark.parametrize("n", [8, 9, 40, 41, 42, 64, 65, 130, 1025])
def test_one_cluster_descent_and_ils(lg, inst, oracle_mod, n, kind):
    """A context's small instance solved by one cluster: from one CTA to
    sixteen, with lists that hold every other city and lists that do not."""
    xy = points(inst, kind, n, 40 + n)
    r = inst.random_tour(n, n)
    with lg.Solver(xy) as s:
        assert s.info()["descent_mode"] == lg.DESCENT_COOPERATIVE
        got, st = s.optimize(r)
        want, moves, _ = oracle_mod.descend(xy, r)
        assert np.array_equal(got, want) and st["moves"] == moves
        got, st = s.ils(want, 3, 7, n % 2)
        want, ost = oracle_mod.ils(xy, want, 3, 7, kind=n % 2)
        assert np.array_equal(got, want) and st["final_length"] == ost["best_length"]


@pytest.mark.parametrize("n", [2048, 2049, 4097])
def test_one_cluster_and_graph_agree(lg, inst, n):
    """Where the cluster's threads change, and above the sizes the oracle
    walks quickly: the graph-driven descent has the same moves."""
    xy = inst.clustered(n, n, clusters=20, sigma_frac=0.03)
    r = lg.nn_tour(xy)
    res = []
    for mode in (lg.DESCENT_GRAPH, lg.DESCENT_COOPERATIVE):
        with lg.Solver(xy) as s:
            s.set_descent_mode(mode)
            t, tr, st = s.optimize_trace(r)
            u, su = s.ils(t, 3, 5, 1)
        res.append((t, tr, st["sweeps"], u, su["final_length"], su["moves"], su["sweeps"]))
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,kind", [(6145, "uniform"), (6999, "heaps"), (7000, "clumps"),
                                    (8000, "line"), (9001, "lattice"), (20011, "uniform")])
def test_grid_and_graph_agree(lg, inst, n, kind):
    """Above the cluster's sizes, the grid-wide launch against the graph-driven
    descent: every move, a bounded descent that goes on, and an ILS call."""
    xy = points(inst, kind, n, 60 + n)
    r = lg.nn_tour(xy)
    res = []
    for mode in (lg.DESCENT_GRAPH, lg.DESCENT_AUTO):
        with lg.Solver(xy) as s:
            s.set_descent_mode(mode)
            s.set_route(r)
            st = s.descend_resident(max_moves=5)
            mid = s.get_route()
            t, tr, sd = s.optimize_trace(mid, max_moves=400)
            u, su = s.ils(t, 2, 5, n % 2)
            step = s.optimize_step(u)
        res.append((st["moves"], st["sweeps"], mid, t, tr, sd["sweeps"], u, su["final_length"],
                    su["moves"], su["sweeps"], su["accepted"], step))
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [8, 2049, 6145, 20000])
def test_whole_calls_and_graph_agree(lg, inst, n):
    """A step and a bounded descent of the caller's route as one launch each,
    from a random tour (at 20000 edges without a list of their own in nearly
    every sweep, and more of them than are listed); a route with a city twice
    or out of range is refused and the next call answered."""
    xy = points(inst, "uniform", n, 80 + n)
    r = inst.random_tour(n, 81 + n)
    res = []
    for mode in (lg.DESCENT_GRAPH, lg.DESCENT_AUTO):
        with lg.Solver(xy) as s:
            s.set_descent_mode(mode)
            step = s.optimize_step(r)
            for city in (r[0], n, 0xFFFFFFFF):
                wrong = r.copy()
                wrong[n // 2] = city
                with pytest.raises(lg.LogoError):
                    s.optimize_step(wrong)
                with pytest.raises(lg.LogoError):
                    s.optimize(wrong)
            t, st = s.optimize(r, max_moves=12)
            res.append((step, t, st["moves"], st["sweeps"], st["start_length"],
                        st["final_length"], s.optimize_step(t), s.get_route()))
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind", ["uniform", "heaps", "clumps", "lattice"])
@pytest.mark.parametrize("n", [8, 33, 1025, 6145, 80000])
def test_neighbour_phase_and_graph_agree(lg, inst, n, kind):
    """The neighbour phase as one launch against its kernels in a graph: from one
    CTA to all, positions in more than one turn (80000), ties everywhere."""
    xy = points(inst, kind, n, 90 + n)
    r = lg.nn_tour(xy) if n > 2000 else inst.random_tour(n, 91 + n)
    for search in (lg.SEARCH_NEIGHBOUR, lg.SEARCH_NEIGHBOUR_OROPT):
        res = []
        for mode in (lg.DESCENT_GRAPH, lg.DESCENT_AUTO):
            with lg.Solver(xy) as s:
                s.set_search(search)
                s.set_descent_mode(mode)
                t, st = s.optimize(r, max_moves=150 if n > 2000 else 0)
                u, su = s.optimize(t, max_moves=20)
            res.append((t, st["moves"], st["sweeps"], st["pair_evals"], u, su["moves"],
                        su["sweeps"], su["final_length"]))
        for a, b in zip(*res):
            assert np.array_equal(a, b)
