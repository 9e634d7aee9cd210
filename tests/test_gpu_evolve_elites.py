"""Populations that are mostly elite copies, in evolve launches: rows whose whole work is a copy
that other CTAs cross over from in the next generation.  Against the oracle, bit for bit."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_evolve import check
from test_gpu_ops import B

pytestmark = pytest.mark.gpu


# 32, 64, 128 and 512 threads a row
@pytest.mark.parametrize("n,P,G", [(52, 256, 40), (1000, 2048, 6), (1500, 1000, 8), (8192, 150, 8)])
def test_mostly_elites(cuda, n, P, G):
    xy = I.tsp_coords(n, seed=n)
    check(B().tsp(xy), O.OracleProblem(O.TSP_COORDS, n, xy=xy), P, P * 9 // 10, 0, G, seed=n)
