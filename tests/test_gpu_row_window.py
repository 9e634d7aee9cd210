"""The row kernel's argsort where its choices change: buckets of up to nine keys are ranked in a
window of neighbours, up to 32 by a loop, larger ones by a bitonic network; equal keys inside a
bucket go by index; TSPJ's two segments stay apart; the last group of four keys is padded.
Permutations against the oracle's, bit for bit."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_ops import B, eval_gpu

pytestmark = pytest.mark.gpu


def crowded_keys(n, crowd, seed):
    """distinct spread keys with `crowd` keys inside one bucket's width: distinct, equal, and at
    either end of the range (the last row ends in NaN)"""
    rng = np.random.default_rng(seed)
    rows = []
    for at in (0.0, 0.37, 1.0 - 1.0 / 4096):
        for equal in (False, True):
            k = (rng.permutation(n) + 0.5) / n
            pick = rng.choice(n, min(crowd, n), replace=False)
            k[pick] = at + (0.0 if equal else 1e-5 / max(n, 16)) * np.arange(pick.size)
            rows.append(k)
    rows[-1][-1] = np.nan
    return np.array(rows, np.float64).astype(np.float32)


@pytest.mark.parametrize("crowd", [1, 5, 6, 7, 8, 9, 10, 31, 32, 33, 40])
@pytest.mark.parametrize("n", [1, 3, 5, 127, 129, 513, 1000, 4097])
def test_window_edges(cuda, n, crowd):
    xy = I.tsp_coords(n, seed=n)
    po = O.OracleProblem(O.TSP_COORDS, n, xy=xy)
    keys = crowded_keys(n, crowd, seed=n * 100 + crowd)
    fit, perm = eval_gpu(B().tsp(xy), keys, cuda)
    np.testing.assert_array_equal(perm, O.decode(keys))
    np.testing.assert_array_equal(fit.view(np.uint32), O.evaluate(po, keys).view(np.uint32))


@pytest.mark.parametrize("crowd", [1, 8, 9, 10, 33])
@pytest.mark.parametrize("c", [1, 2, 31, 64, 101, 700])
def test_window_two_segments(cuda, c, crowd):
    travel, jobs = I.tspj_instance(c, seed=c)
    po = O.OracleProblem(O.TSPJ, 2 * c, mat=travel, mat2=jobs)
    keys = np.concatenate([crowded_keys(c, crowd, seed=c), crowded_keys(c, crowd, seed=c + 1)[::-1]], 1)
    fit, perm = eval_gpu(B().tspj(travel, jobs), np.ascontiguousarray(keys), cuda)
    np.testing.assert_array_equal(perm, O.decode_problem(po, keys))
    np.testing.assert_array_equal(fit.view(np.uint32), O.evaluate(po, keys).view(np.uint32))


@pytest.mark.parametrize("threads", [32, 64, 128, 256, 512, 1024])
def test_every_tile_same_run(cuda, threads, monkeypatch):
    """rows of 1 .. 16 groups of four keys a thread give the same run whatever the tile"""
    n, P, E, M, G = 500, 96, 14, 14, 4
    xy = I.tsp_coords(n, seed=1)
    monkeypatch.setenv("BRKGA_TILE", f"{threads},{-(-n // (4 * threads))}")
    s = B().Solver(B().tsp(xy), B().params(P, E, M, 0.7, G, seed=5))
    assert s.info[0] == threads
    s.run()
    keys, fit = s.get_population()
    from test_gpu_engine import oracle_islands
    rk, rf, rh = oracle_islands(O.OracleProblem(O.TSP_COORDS, n, xy=xy), P, E, M, 0.7, 5, 1, 0, 0, G, n)
    np.testing.assert_array_equal(keys, rk)
    np.testing.assert_array_equal(fit, rf)
    s.close()


@pytest.mark.parametrize("crowd", [9, 10, 20, 31, 32, 33])
@pytest.mark.parametrize("n", [40, 129, 700])
def test_crowded_buckets_of_shifted_keys(cuda, n, crowd):
    """MO-VRP sorts by shifted keys through a bucket map of its own"""
    xy, dem, cap, V = I.movrp_instance(n, seed=n)
    po = O.OracleProblem(O.MOVRP, n, xy=xy, w=dem, machines=V, vcap=cap)
    keys = crowded_keys(n, crowd, seed=n + crowd)[:-1]
    obj, perm = eval_gpu(B().movrp(xy, dem, cap, V), keys, cuda)
    np.testing.assert_array_equal(perm, O.decode_problem(po, keys))
    np.testing.assert_array_equal(obj.view(np.uint32), O.evaluate(po, keys).view(np.uint32))
