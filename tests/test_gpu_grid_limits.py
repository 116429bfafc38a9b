"""The branches of the grid-wide launch (grid_tour.cu) for more edges than its
lists hold, which tours of ordinary sizes do not fill: with the lists' limits
lowered, against the graph-driven descent.  Whole numbers: the tolerance is
zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (edges put off, edges listed for their pairs, cities of a disc, discs put off)
@pytest.mark.parametrize("limits", [(0, 0, 64, 0), (2, 0, 64, 0), (0, 8, 64, 0), (2, 8, 64, 0),
                                    (1, 1, 1, 0), (0, 0, 64, 4096), (2, 8, 64, 1)])
@pytest.mark.parametrize("points", ["uniform", "clustered"])
def test_more_edges_than_the_lists_hold(lg, inst, points, limits):
    n = 7000
    xy = (inst.clustered(n, 5, clusters=12, sigma_frac=0.01) if points == "clustered"
          else inst.uniform_f32(n, 5, 1.0e5))
    r = inst.random_tour(n, 6)
    with lg.Solver(xy) as s:
        s.set_descent_mode(lg.DESCENT_GRAPH)
        want, log, st = s.optimize_trace(r, max_moves=250)
        late, llog, lst = s.optimize_trace(lg.nn_tour(xy), max_moves=60)
    with lg.Solver(xy) as s:
        s.grid_limits(*limits)
        got, trace, gst = s.optimize_trace(r, max_moves=250)
        wides, takers, _ = s.grid_counts()
        # the branches under test were taken: edges were put off, more than are listed
        assert wides > limits[0] and takers > limits[1]
        assert np.array_equal(trace, log) and np.array_equal(got, want)
        assert gst["sweeps"] == st["sweeps"] and gst["final_length"] == st["final_length"]
        got, trace, gst = s.optimize_trace(lg.nn_tour(xy), max_moves=60)
        assert np.array_equal(trace, llog) and np.array_equal(got, late)
        assert s.optimize_step(r) == tuple(int(v) for v in log[0])


def test_limits_above_the_lists_are_refused(lg, inst):
    with lg.Solver(inst.uniform_f32(7000, 1, 1.0e4)) as s:
        for limits in ((1025, 0, 0, 0), (0, 8193, 0, 0), (0, 0, 4097, 0), (0, 0, 0, 4097)):
            with pytest.raises(lg.LogoError):
                s.grid_limits(*limits)


def both_ways(lg, xy, r, moves, limits=(0, 0, 0, 0)):
    res = []
    for mode in (lg.DESCENT_GRAPH, lg.DESCENT_AUTO):
        with lg.Solver(xy) as s:
            s.set_descent_mode(mode)
            s.grid_limits(*limits)
            t, trace, st = s.optimize_trace(r, max_moves=moves)
            counts = s.grid_counts() if len(xy) > 6144 else None
            res.append((t, trace, st["sweeps"], st["final_length"], s.optimize_step(t)))
    for a, b in zip(*res):
        assert np.array_equal(a, b)
    return counts


def test_a_disc_is_counted_by_its_cities(lg, inst):
    """Two heaps far apart: each lies in one cell of the search grid, so a disc
    of one cell holds thousands of cities and has to be put off."""
    xy = inst.uniform_f32(7000, 11, 100.0)
    xy[::2] += np.float32(1.0e6)
    assert both_ways(lg, xy, lg.nn_tour(xy), 120, limits=(0, 0, 1024, 0))[0] > 0


@pytest.mark.parametrize("discs", [4096, 3])
@pytest.mark.parametrize("n,kind", [(6145, "uniform"), (7000, "clustered"), (20000, "uniform"),
                                    (20000, "clustered")])
def test_discs_dealt_to_all_ctas(lg, inst, n, kind, discs):
    """As above 50,000 cities; from a nearest-neighbour and a random tour, and
    with more of them than are listed."""
    xy = (inst.clustered(n, n, clusters=20, sigma_frac=0.03) if kind == "clustered"
          else inst.uniform_f32(n, n, 1.0e5))
    assert both_ways(lg, xy, lg.nn_tour(xy), 300, limits=(0, 0, 0, discs))[2] > discs % 4096
    both_ways(lg, xy, inst.random_tour(n, 1), 80, limits=(0, 0, 0, discs))


@pytest.mark.parametrize("n", [50001, 100003])
def test_above_the_size_where_discs_are_dealt(lg, inst, n):
    xy = inst.clustered(n, 3)
    assert both_ways(lg, xy, lg.nn_tour(xy), 60)[2] > 0
    both_ways(lg, xy, inst.random_tour(n, 1), 20)


@pytest.mark.parametrize("kind", ["stray", "strays", "heaps"])
@pytest.mark.parametrize("n", [1024, 6000, 7000, 20000, 60000])
def test_unevenly_spread_cities(lg, inst, n, kind):
    """Cities far from the rest, which lie outside the search grid's box, and
    heaps that its cells do not tell apart (from 20000 the graph-driven descent
    runs there whatever the mode)."""
    xy = inst.uniform_f32(n, 11 + n, 1.0e4)
    if kind == "stray":
        xy[n // 3] = (1.0e6, 1.0e6)
    elif kind == "strays":
        xy[7::n // 20] *= np.float32(-90.0)
    else:
        xy *= np.float32(0.01)
        xy[::2] += np.float32(1.0e6)
    both_ways(lg, xy, lg.nn_tour(xy), 100)
    if n <= 20000:
        both_ways(lg, xy, inst.random_tour(n, n), 60)


def test_info_says_when_calls_run_over_the_whole_device(lg, inst):
    xy = inst.uniform_f32(20000, 1, 1.0e4)
    with lg.Solver(xy[:6144]) as s:
        assert s.info()["grid_ctas"] == 0
    with lg.Solver(xy) as s:
        assert s.info()["grid_ctas"] > 0
        s.set_descent_mode(lg.DESCENT_GRAPH)
        assert s.info()["grid_ctas"] == 0
        s.set_descent_mode(lg.DESCENT_AUTO)
        assert s.info()["grid_ctas"] > 0
        s.set_kernel(lg.SWEEP_BOXED, 4, 4, 64)
        assert s.info()["grid_ctas"] == 0
    heaps = xy * np.float32(0.01)
    heaps[::2] += np.float32(1.0e6)
    with lg.Solver(heaps) as s:  # its search grid would not tell the cities apart
        assert s.info()["grid_ctas"] == 0
