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
