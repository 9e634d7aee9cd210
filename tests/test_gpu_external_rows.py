"""Rows that an engine only builds (the caller's fitness): row lengths around the block of threads that
builds them, against the built-in problem on the same seed, bit for bit."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_ops import B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,P", [(1, 40), (5, 700), (128, 64), (129, 64), (4096, 24), (4099, 24), (20001, 8)])
def test_built_rows(cuda, n, P):
    xy = I.tsp_coords(n, seed=n)
    po = O.OracleProblem(O.TSP_COORDS, n, xy=xy)
    G, prm = 4, B().params(P, P // 4, P // 8, 0.7, 4, seed=5)
    want = B().Solver(B().tsp(xy), prm)
    want.initialize()
    want.evolve(G)
    s = B().Solver(B().external(n), prm)
    for _ in range(G + 1):
        s.external_step(lambda rows: O.evaluate(po, rows))
    for a, b in zip(s.get_population(), want.get_population()):
        np.testing.assert_array_equal(a, b)
    s.close()
    want.close()
