"""Grid-wide launches end between two moves after a while and go on in the next
launch, so that other contexts' calls need not wait for a whole descent."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def flat(x):
    if isinstance(x, dict):
        return [v for k, v in sorted(x.items()) if k != "device_ms"]
    if isinstance(x, (list, tuple)):
        return [w for v in x for w in flat(v)]
    return [x]


@pytest.mark.parametrize("io", ["copy", "auto"])
@pytest.mark.parametrize("us", [1, 150])
def test_paused_launches_do_the_same(lg, inst, us, io):
    """A pause after every move, or every few: tours, moves, statistics and
    lengths are those of the graph-driven descent."""
    n = 7000
    xy = inst.uniform_f32(n, 31, 1.0e4)
    r = lg.nn_tour(xy)
    res = []
    for mode in (lg.DESCENT_GRAPH, lg.DESCENT_AUTO):
        with lg.Solver(xy) as s:
            s.set_route_io(lg.ROUTE_IO_COPY if io == "copy" else lg.ROUTE_IO_AUTO)
            s.set_descent_mode(mode)
            s.grid_quantum(us)
            got = [s.optimize_step(r), s.optimize(r, max_moves=1), s.optimize(r, max_moves=30),
                   s.optimize(r, max_moves=31, stats=False)[0],
                   s.optimize_trace(r, max_moves=25)]
            w0 = s.info()["host_waits"]
            got.append(s.optimize(r))
            if mode == lg.DESCENT_AUTO and us == 1:
                assert s.info()["host_waits"] - w0 > got[-1][1]["moves"]
            s.set_route(got[2][0])
            got += [s.descend_resident(max_moves=12), s.length_resident(), s.get_route()]
            for kind in (0, 1):
                got += [s.ils(got[5][0], 4, 9, kind), s.ils(r, 1, 9, kind)]
            s.set_search(lg.SEARCH_NEIGHBOUR)
            got += [s.optimize(r, stats=False)[0]]
        res.append(flat(got))
    assert len(res[0]) == len(res[1])
    for a, b in zip(*res):
        assert np.array_equal(a, b)


def test_a_step_does_not_wait_for_another_context(lg, inst):
    """While one thread's ILS call of a large tour runs, another thread's best
    moves are answered."""
    big, small = inst.uniform_f32(20000, 41, 1.0e6), inst.uniform_f32(7000, 42, 1.0e4)
    rb, rs = lg.nn_tour(big), lg.nn_tour(small)
    with lg.Solver(big) as a, lg.Solver(small) as b:
        start, _ = a.optimize(rb)
        want = b.optimize_step(rs)
        ends = {}

        def run():
            a.ils(start, 10000, 1, 1)  # a second or more
            ends["ils"] = time.perf_counter()

        t = threading.Thread(target=run)
        t.start()
        time.sleep(0.05)
        got = [b.optimize_step(rs) for _ in range(3)]
        ends["steps"] = time.perf_counter()
        running = t.is_alive()
        t.join()
        assert got == [want] * 3
        assert running and ends["steps"] < ends["ils"]


@pytest.mark.parametrize("n", [500, 20000])
def test_info_leaves_a_capture_alone(lg, inst, oracle_mod, n):
    """The context's stream may be under capture (logo_enqueue_sweep is a launch
    like any other): asking for the context's info makes no call on it."""
    torch = pytest.importorskip("torch")
    xy = inst.uniform_f32(n, 5, 1.0e5)
    r = inst.random_tour(n, 6)
    with lg.Solver(xy) as s:
        s.set_route(r)
        s.begin_descent()
        s.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(s.stream)):
            graph.capture_begin(capture_error_mode="thread_local")
            grid = s.info()["grid_ctas"]
            s.enqueue_sweep()
            s.enqueue_apply()
            graph.capture_end()
            graph.replay()
        assert (grid > 0) == (n > 6144)
        s.sync()
        assert s.progress() == (1, False)
        got = s.get_route()
    with lg.Solver(xy) as s:
        want, _ = s.optimize(r, max_moves=1)
    assert np.array_equal(got, want)
