"""The branches of the grid-wide launch (grid_tour.cu) for more edges than its
lists hold, which tours of ordinary sizes do not fill: with the lists' limits
lowered, against the graph-driven descent.  Whole numbers: the tolerance is
zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (edges put off, edges listed for their pairs, cities of a disc)
@pytest.mark.parametrize("limits", [(0, 0, 64), (2, 0, 64), (0, 8, 64), (2, 8, 64), (1, 1, 1)])
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
        wides, takers = s.grid_counts()
        # the branches under test were taken: edges were put off, more than are listed
        assert wides > limits[0] and takers > limits[1]
        assert np.array_equal(trace, log) and np.array_equal(got, want)
        assert gst["sweeps"] == st["sweeps"] and gst["final_length"] == st["final_length"]
        got, trace, gst = s.optimize_trace(lg.nn_tour(xy), max_moves=60)
        assert np.array_equal(trace, llog) and np.array_equal(got, late)
        assert s.optimize_step(r) == tuple(int(v) for v in log[0])


def test_limits_above_the_lists_are_refused(lg, inst):
    with lg.Solver(inst.uniform_f32(7000, 1, 1.0e4)) as s:
        for limits in ((1025, 0, 0), (0, 8193, 0), (0, 0, 4097)):
            with pytest.raises(lg.LogoError):
                s.grid_limits(*limits)
