"""Whole generations in one launch (csrc/evolve.cu) against the oracle, every row and the whole
history bit for bit: the smallest populations, no children or no mutants, sizes about the
changes of threads per row and of rows per CTA, launches that follow each other, local search."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_engine import oracle_islands
from test_gpu_ops import B

pytestmark = pytest.mark.gpu


def check(pb, po, P, E, M, G, seed, pieces=None):
    n = pb.n
    s = B().Solver(pb, B().params(P, E, M, 0.7, G, seed=seed))
    s.initialize()
    for g in pieces or [G]:
        s.evolve(g)
    keys, fit = s.get_population()
    rk, rf, rh = oracle_islands(po, P, E, M, 0.7, seed, 1, 0, 0, G, (n + 3) // 4 * 4)
    np.testing.assert_array_equal(keys, rk)
    np.testing.assert_array_equal(fit, rf)
    np.testing.assert_array_equal(s.get_fitness_history(), rh)
    s.close()


@pytest.mark.parametrize("P,E,M", [(1, 1, 0), (2, 1, 1), (5, 2, 3), (7, 7, 0), (33, 5, 0), (149, 20, 17), (1185, 150, 90)])
@pytest.mark.parametrize("n", [1, 6, 129])
def test_population_shapes(cuda, n, P, E, M):
    xy = I.tsp_coords(n, seed=n + P)
    check(B().tsp(xy), O.OracleProblem(O.TSP_COORDS, n, xy=xy), P, E, M, 6, seed=P)


@pytest.mark.parametrize("n,P", [(513, 300), (1025, 160), (2049, 40), (4097, 24), (8192, 12), (8193, 12)])
def test_row_lengths(cuda, n, P):
    xy = I.tsp_coords(n, seed=n)
    check(B().tsp(xy), O.OracleProblem(O.TSP_COORDS, n, xy=xy), P, P // 5, P // 8, 3, seed=n)


def test_launches_in_pieces(cuda):
    """one, two, 130 generations (two launches), and one more"""
    n, P = 40, 60
    w, v, cap = I.knap_items(n, seed=2)
    for greedy in (True, False):
        po = O.OracleProblem(O.KNAP_GREEDY if greedy else O.KNAP_THRESHOLD, n, w=w, v=v, cap=cap)
        check(B().knapsack(w, v, cap, greedy=greedy), po, P, 12, 6, 134, seed=3, pieces=[1, 2, 130, 1])


def test_other_kinds(cuda):
    d = np.random.default_rng(4).random((60, 60), dtype=np.float32)
    check(B().tsp_matrix(d), O.OracleProblem(O.TSP_MATRIX, 60, mat=d), 80, 16, 8, 12, seed=5)
    jt = (1.0 + np.random.default_rng(5).random(150) * 99.0).astype(np.float32)
    check(B().jobsched(jt, 40), O.OracleProblem(O.JOBSCHED, 150, jt=jt, machines=40), 80, 16, 8, 12, seed=6)
    check(B().continuous(33, -5.0, 10.0, 2), O.OracleProblem(O.CONTINUOUS, 33, function=2, lo=-5.0, hi=10.0), 80, 16, 8, 12,
          seed=7)


def test_searched_runs_same_in_pieces(cuda):
    """TSPJ with local search: one launch of 30 generations and 30 launches of one; the search
    itself is checked against the oracle elsewhere"""
    travel, jobs = I.tspj_instance(31, seed=8)
    out = []
    for pieces in ([30], [1] * 30):
        s = B().Solver(B().tspj(travel, jobs), B().params(150, 30, 15, 0.7, 30, seed=9, local_search_interval=2,
                                                          local_search_individuals=25))
        s.initialize()
        for g in pieces:
            s.evolve(g)
        out.append((*s.get_population(), s.get_fitness_history()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
