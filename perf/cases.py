"""The work that users of this framework have it do, as cases to be timed.

A case names what is called ("what") and the sizes and options it is called
with.  All go through the public binding, `logo_gpu`; instances and start
tours are made from the seed by the repository's own generators.  The path
takes host buffers (coordinates, routes) and gives host buffers back, except
logo_best_move_noalloc, whose buffers are the caller's device memory.

What a program makes once and keeps is made in prepare(): the instance, its
start tour and the context, batch or server.  A pass is the call (or, for the
server, the calls) that such a program makes with them.

  step      Solver.optimize_step: the best move of a tour, route in, move out
  noalloc   best_move_noalloc on device buffers of the caller's
  move      Solver.optimize_inplace(max_moves=...): the tour a few moves on,
            route in, route out; the buffer goes on from pass to pass
  descent   Solver.optimize: to the local optimum, with its statistics; by the
            search it was set to (exhaustive, or the neighbour lists first)
  ils       Solver.ils: descent, then kicks
  batch     Batch.solve: many instances in one call
  serve     Server.submit for every request of a burst, then Server.wait
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "logo-tsp-solver_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import instances  # noqa: E402
import logo_gpu as lg  # noqa: E402

SEARCH = {"all": lg.SEARCH_EXHAUSTIVE, "near": lg.SEARCH_NEIGHBOUR,
          "oropt": lg.SEARCH_NEIGHBOUR_OROPT}
KICK = {"segment": lg.KICK_SEGMENT, "bridge": lg.KICK_DOUBLE_BRIDGE}
START = {"given": lg.START_GIVEN, "nn": lg.START_NN, "mf": lg.START_MF}


def listed():
    return [
        # the smallest instance in use (berlin52's size): a move asked for by
        # a host program that keeps the loop to itself; all of it is latency
        dict(name="step_52", what="step", n=52, points="int", tour="nn"),
        # the largest sweep that is measured (one million points, random tour)
        dict(name="step_1m", what="step", n=1000000, points="uniform", tour="random"),
        # a caller that owns its device memory, at an odd size
        dict(name="noalloc_20011", what="noalloc", n=20011, points="clustered", tour="nn"),
        # bench.py's headline step through the C ABI: one move of the descent
        # of a large clustered instance, on the caller's buffer
        dict(name="move_100k", what="move", n=100000, moves=1, points="clustered", tour="nn"),
        # the plain single instance (n = 1,000, integer coordinates) from the
        # nearest-neighbour tour to its local optimum
        dict(name="descent_1000", what="descent", n=1000, points="int", tour="nn",
             search="all"),
        # a mid-size instance of an odd size from a random tour, the
        # reference's default start
        dict(name="descent_4461_random", what="descent", n=4461, points="uniform",
             tour="random", search="all"),
        # a large clustered instance as a whole
        dict(name="descent_40009", what="descent", n=40009, points="clustered", tour="nn",
             search="all"),
        # the same kind of instance by the neighbour lists, with Or-opt moves
        dict(name="oropt_25000", what="descent", n=25000, points="clustered", tour="nn",
             search="oropt"),
        # iterated local search of one instance: double bridges at n = 1,500,
        # the reference's own kick on a larger one
        dict(name="ils_1500_bridge", what="ils", n=1500, points="uniform", tour="nn", kicks=100,
             kick="bridge", search="all"),
        dict(name="ils_20000_segment", what="ils", n=20000, points="clustered", tour="nn",
             kicks=20, kick="segment", search="all"),
        # the batched workload (n log-uniform in [50, 2,000], random start
        # tours, segment kicks), with fewer instances and kicks
        dict(name="batch_1024", what="batch", count=1024, lo=50, hi=2000, kicks=40,
             kick="segment", start="given"),
        # a burst of requests to the server: n log-uniform in [100, 6,000],
        # clustered and uniform by turns, NN start tours, 50 kicks each
        dict(name="serve_64", what="serve", count=64, lo=100, hi=6000, kicks=50,
             kick="segment"),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["step", "noalloc", "move", "descent", "descent", "ils", "ils", "batch",
                       "serve"])
    points = rng.choice(["int", "uniform", "clustered"])
    if what == "step":
        return dict(what=what, n=_log_uniform(rng, 52, 1000000), points=points,
                    tour=rng.choice(["nn", "random"]))
    if what == "noalloc":
        return dict(what=what, n=_log_uniform(rng, 52, 65536), points=points,
                    tour=rng.choice(["nn", "random"]))
    if what == "move":
        return dict(what=what, n=_log_uniform(rng, 1000, 200000), moves=rng.choice([1, 1, 3, 10]),
                    points=points, tour="nn")
    if what == "descent":
        tour = rng.choice(["nn", "nn", "random"])
        return dict(what=what, n=_log_uniform(rng, 52, 5000 if tour == "random" else 40009),
                    points=points, tour=tour, search=rng.choice(["all", "all", "near", "oropt"]))
    if what == "ils":
        n = _log_uniform(rng, 100, 20000)
        return dict(what=what, n=n, points=points, tour="nn", kicks=rng.randint(5, 20),
                    kick=rng.choice(["segment", "bridge"]),
                    search=rng.choice(["all", "all", "all", "near"]))
    if what == "batch":
        hi = rng.choice([500, 2000, 4096])
        count = _log_uniform(rng, 8, 1024 if hi <= 2000 else 256)
        return dict(what=what, count=count, lo=50, hi=hi, kicks=rng.randint(0, 40),
                    kick=rng.choice(["segment", "bridge"]),
                    start=rng.choice(["given", "nn", "mf"]))
    return dict(what=what, count=rng.randint(4, 64), lo=100, hi=rng.choice([1000, 4096, 6000]),
                kicks=rng.randint(0, 50), kick=rng.choice(["segment", "bridge"]))


def _points(kind, n, seed):
    if kind == "int":  # TSPLIB-like whole coordinates
        return instances.uniform_int(n, seed, side=10000)
    if kind == "uniform":
        return instances.uniform_f32(n, seed, 1.0e6)
    return instances.clustered(n, seed, side=1.0e6, clusters=200 if n >= 20000 else 20,
                               sigma_frac=0.01 if n >= 20000 else 0.03)


def _sizes(case):
    """The case's instance sizes: the same for every seed, so that the outputs
    of two seeds have one shape."""
    return instances.batch_sizes(case["count"], 3, case["lo"], case["hi"])


def prepare(case, seed):
    lg.load()
    what = case["what"]
    if what == "batch":
        ns = _sizes(case)
        seeds = [instances.instance_seed(seed, k) for k in range(len(ns))]
        xs = [instances.uniform_f32(int(n), s, 1.0e4) for n, s in zip(ns, seeds)]
        rs = [lg.random_tour(int(n), s) for n, s in zip(ns, seeds)]
        return dict(case=case, xs=xs, rs=rs if case["start"] == "given" else None, seeds=seeds,
                    b=lg.Batch(len(ns), int(ns.sum())))
    if what == "serve":
        ns = _sizes(case)
        seeds = [instances.instance_seed(seed, k) for k in range(len(ns))]
        xs = [_points("clustered" if k % 2 else "uniform", int(n), s)
              for k, (n, s) in enumerate(zip(ns, seeds))]
        return dict(case=case, xs=xs, rs=[lg.nn_tour(x) for x in xs], seeds=seeds,
                    server=lg.Server(kicks=case["kicks"], kind=KICK[case["kick"]]))
    n = case["n"]
    xy = _points(case["points"], n, seed)
    route = lg.nn_tour(xy) if case["tour"] == "nn" else lg.random_tour(n, seed)
    if what == "noalloc":
        return dict(case=case, xy=torch.from_numpy(xy).cuda(),
                    route=torch.from_numpy(route.view(np.int32)).cuda(),
                    out=torch.zeros(3, dtype=torch.int32, device="cuda"),
                    status=torch.zeros(1, dtype=torch.int32, device="cuda"))
    solver = lg.Solver(xy)
    if case.get("search", "all") != "all":
        solver.set_search(SEARCH[case["search"]])
    return dict(case=case, solver=solver, route=route, seed=seed)


def _counts(st):
    """The whole numbers of a call's statistics (all but its device time)."""
    return [int(v) for k, v in sorted(st.items()) if not k.endswith("_ms")]


def run(state):
    case = state["case"]
    what = case["what"]
    if what == "step":
        return state["solver"].optimize_step(state["route"])
    if what == "noalloc":
        lg.best_move_noalloc(state["xy"].data_ptr(), state["route"].data_ptr(), case["n"],
                             state["out"].data_ptr(), state["status"].data_ptr(),
                             torch.cuda.current_stream().cuda_stream)
        return state["out"], state["status"]
    if what == "move":
        state["solver"].optimize_inplace(state["route"], max_moves=case["moves"])
        return state["route"]
    if what == "descent":
        route, st = state["solver"].optimize(state["route"])
        return route, np.array(_counts(st), dtype=np.int64)
    if what == "ils":
        route, st = state["solver"].ils(state["route"], case["kicks"], state["seed"],
                                        KICK[case["kick"]])
        return route, np.array(_counts(st), dtype=np.int64)
    if what == "batch":
        routes, res, _ = state["b"].solve(state["xs"], state["rs"], state["seeds"],
                                          kicks=case["kicks"], kind=KICK[case["kick"]],
                                          start=START[case["start"]])
        return np.concatenate(routes), np.array([_counts(r) for r in res], dtype=np.int64)
    server = state["server"]
    ids = [server.submit(x, r, s) for x, r, s in zip(state["xs"], state["rs"], state["seeds"])]
    got = [server.wait(i) for i in ids]
    return (np.concatenate([r for r, _ in got]),
            np.array([_counts(info) for _, info in got], dtype=np.int64))


def work(case):
    """Coordinates and the route in and the route (or the move) out; of
    arithmetic only what any local search has to do, a distance (6 operations)
    for each city and pass over the tour.  How many moves a descent makes is
    the input's affair, and which pairs a sweep may leave out is the path's."""
    what = case["what"]
    if what in ("batch", "serve"):
        lo, hi = case["lo"], case["hi"]
        mean = (hi - lo) / math.log(hi / lo)
        cities, passes = case["count"] * mean, case["kicks"] + 1
        route_in = 4 if case.get("start", "given") == "given" else 0
        return {"bytes": (8 + route_in + 4) * cities, "flops": 6 * cities * passes}
    n = case["n"]
    passes = case.get("kicks", 0) + 1
    out = 12 if what in ("step", "noalloc") else 4 * n
    return {"bytes": 12 * n + out, "flops": 6 * n * passes}


def exact(case, seed):
    """Nothing here is a rounded number: moves, tours, lengths and counts are
    whole numbers, and which move is the best is defined on distances rounded
    to whole numbers from 32-bit coordinates."""
    return None
