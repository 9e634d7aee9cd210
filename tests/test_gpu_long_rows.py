"""Rows of more chunks than are picked out of the row by passes over it: around that line (about 155 000
keys) and well past it, with ties and keys at the ends of the range; against the oracle."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_ops import B, eval_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100001, 150000, 156000, 160003, 300002])
def test_decode_and_tour(cuda, n):
    xy = I.tsp_coords(n, seed=n)
    keys = I.keys(3, n, seed=n + 1)
    keys[0, ::7] = keys[0, 3]
    keys[1, :50] = np.float32(0.0)
    keys[1, 50:100] = np.float32(1.0)
    keys[1, 100:120] = np.float32(-3.0)
    keys[2, 5] = np.nan
    if n > 200000:
        keys[0, ::7] = np.linspace(0.2, 0.2001, keys[0, ::7].size, dtype=np.float32)
    fit, perm = eval_gpu(B().tsp(xy), keys, cuda)
    np.testing.assert_array_equal(perm, O.decode(keys))
    po = O.OracleProblem(O.TSP_COORDS, n, xy=xy)
    np.testing.assert_array_equal(fit.view(np.uint32), O.evaluate(po, keys).view(np.uint32))


def test_knapsack(cuda):
    n = 200001
    w, v, cap = I.knap_items(n, seed=5)
    keys = I.keys(3, n, seed=6)
    fit, perm = eval_gpu(B().knapsack(w, v, cap, greedy=True), keys, cuda)
    np.testing.assert_array_equal(perm, O.decode(keys))
    np.testing.assert_array_equal(fit, O.evaluate(O.OracleProblem(O.KNAP_GREEDY, n, w=w, v=v, cap=cap), keys))
