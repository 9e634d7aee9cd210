"""Kinds whose fitness comes straight from the keys: every remainder of four keys, several rows a
thread group one after the other, odd strides; against the oracle bit for bit."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_ops import B, eval_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pad", [0, 1, 4])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 127, 130, 513, 4277])
def test_threshold_knapsack(cuda, n, pad):
    w, v, cap = I.knap_items(n, seed=n)
    po = O.OracleProblem(O.KNAP_THRESHOLD, n, w=w, v=v, cap=cap)
    for P in (1, 150, 5000 if n < 600 else 700):
        keys = np.full((P, n + pad), 0.9, np.float32)
        keys[:, :n] = I.keys(P, n, seed=n + P)
        keys[0, :n] = 0.5  # not above one half
        fit, _ = eval_gpu(B().knapsack(w, v, cap, greedy=False), keys, cuda, ld=n + pad)
        np.testing.assert_array_equal(fit, O.evaluate(po, np.ascontiguousarray(keys[:, :n])))


@pytest.mark.parametrize("n", [2, 5, 130, 1000])
def test_sums_in_index_order(cuda, n):
    P = 4000
    keys = I.keys(P, n, seed=n)
    jt = (1.0 + np.random.default_rng(n).random(n) * 99.0).astype(np.float32)
    fit, _ = eval_gpu(B().jobsched(jt, 7), keys, cuda)
    np.testing.assert_array_equal(fit, O.evaluate(O.OracleProblem(O.JOBSCHED, n, jt=jt, machines=7), keys))
    for fn in (0, 2):
        fit, _ = eval_gpu(B().continuous(n, -5.0, 10.0, fn), keys, cuda)
        np.testing.assert_array_equal(fit, O.evaluate(O.OracleProblem(O.CONTINUOUS, n, function=fn, lo=-5.0, hi=10.0), keys))
