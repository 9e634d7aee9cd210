"""Evaluations of few rows, which take more threads a row than many rows of the same length: one
row, an SM's worth and around each multiple of the SMs, against the oracle bit for bit."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_ops import B, eval_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 148, 149, 297, 600])
@pytest.mark.parametrize("n", [3, 33, 129, 260, 513, 921, 2049, 4097])
def test_tsp(cuda, n, P):
    if n * P > 1 << 20:
        P = (1 << 20) // n
    xy = I.tsp_coords(n, seed=n)
    keys = I.keys(P, n, seed=n + P)
    keys[0] = keys[0, 0]  # equal keys
    fit, perm = eval_gpu(B().tsp(xy), keys, cuda)
    np.testing.assert_array_equal(perm, O.decode(keys))
    po = O.OracleProblem(O.TSP_COORDS, n, xy=xy)
    np.testing.assert_array_equal(fit.view(np.uint32), O.evaluate(po, keys).view(np.uint32))


@pytest.mark.parametrize("P", [1, 100, 300])
@pytest.mark.parametrize("n", [130, 967, 3001])
def test_other_orders(cuda, n, P):
    w, v, cap = I.knap_items(n, seed=n)
    keys = I.keys(P, n, seed=n + P)
    fit, _ = eval_gpu(B().knapsack(w, v, cap, greedy=True), keys, cuda)
    np.testing.assert_array_equal(fit, O.evaluate(O.OracleProblem(O.KNAP_GREEDY, n, w=w, v=v, cap=cap), keys))
    c = n // 4
    travel, jobs = I.tspj_instance(c, seed=n)
    keys = I.keys(P, 2 * c, seed=n + P)
    fit, _ = eval_gpu(B().tspj(travel, jobs), keys, cuda)
    po = O.OracleProblem(O.TSPJ, 2 * c, mat=travel, mat2=jobs)
    np.testing.assert_array_equal(fit.view(np.uint32), O.evaluate(po, keys).view(np.uint32))
    xy, dem, vcap, V = I.movrp_instance(c, seed=n)
    keys = I.keys(P, c, seed=n + P)
    obj, _ = eval_gpu(B().movrp(xy, dem, vcap, V), keys, cuda)
    po = O.OracleProblem(O.MOVRP, c, xy=xy, w=dem, machines=V, vcap=vcap)
    np.testing.assert_array_equal(obj.view(np.uint32), O.evaluate(po, keys).view(np.uint32))
