"""The numbers of the evolve kernel's steps wrap (2^32 of them, a few hundred steps into every run):
runs across the wrap, inside a launch and between two, one and two steps a generation."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_evolve import check
from test_gpu_ops import B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pieces", [[400], [100, 200, 100], [85] * 4 + [60], [1] * 140 + [260]])
def test_run_across_the_wrap(cuda, pieces):
    n, P = 12, 40
    xy = I.tsp_coords(n, seed=n)
    check(B().tsp(xy), O.OracleProblem(O.TSP_COORDS, n, xy=xy), P, 8, 4, 400, seed=3, pieces=pieces)


def test_searched_run_across_the_wrap(cuda):
    """local search after every generation; launches of one generation each wrap elsewhere"""
    travel, jobs = I.tspj_instance(9, seed=8)
    out = []
    for pieces in ([300], [1] * 300, [127, 2, 100, 71]):
        s = B().Solver(B().tspj(travel, jobs), B().params(60, 12, 6, 0.7, 300, seed=9, local_search_interval=1,
                                                          local_search_individuals=10))
        s.initialize()
        for g in pieces:
            s.evolve(g)
        out.append((*s.get_population(), s.get_fitness_history()))
        s.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
