"""Work that a caller's parameters can make as long as they like does not run inside launches whose
CTAs wait for each other: with waits of no polls at all (BRKGA_WAIT_POLLS=0) such runs end well,
where a launch of whole generations gives up."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_engine import oracle_islands
from test_gpu_ops import B
from test_gpu_wait_limits import run_population, timeout

pytestmark = pytest.mark.gpu


def searched(moves):
    return B().Solver(B().tspj(*I.tspj_instance(20, seed=3)),
                      B().params(64, 12, 6, 0.7, 6, seed=5, local_search_interval=2, local_search_individuals=3,
                                 local_search_moves=moves))


def test_long_local_search(cuda, monkeypatch):
    monkeypatch.setenv("BRKGA_WAIT_POLLS", "0")
    s = searched(5)
    timeout(s.run)
    s.close()
    s = searched(100_000)
    s.run()
    assert (np.diff(s.get_fitness_history()) <= 0).all()
    s.close()


def test_many_machines(cuda, monkeypatch):
    n, P, G = 200, 24, 3
    jt = (1.0 + np.random.default_rng(4).random(n) * 99.0).astype(np.float32)
    monkeypatch.setenv("BRKGA_WAIT_POLLS", "0")
    s = B().Solver(B().jobsched(jt, 40), B().params(P, 4, 2, 0.7, G, seed=6))
    timeout(s.run)
    s.close()
    M = 5_000_000
    s = B().Solver(B().jobsched(jt, M), B().params(P, 4, 2, 0.7, G, seed=6))
    s.run()
    keys, fit = s.get_population()
    rk, rf, _ = oracle_islands(O.OracleProblem(O.JOBSCHED, n, jt=jt, machines=M), P, 4, 2, 0.7, 6, 1, 0, 0, G, n)
    np.testing.assert_array_equal(keys, rk)
    np.testing.assert_array_equal(fit, rf)
    s.close()


def launches(s):
    out = np.full(5, -1, np.int32)
    B().check(B().lib().brkga_engine_info(s.h, out.ctypes.data, 5))
    return tuple(out)


@pytest.mark.parametrize("n,P", [(52, 256), (300, 140), (1000, 2048), (8192, 2048), (4000, 16384)])
def test_info_of_whole_generations(cuda, n, P):
    """the launches that evolve, not the first population's; one that fills the SMs is short, since
    other streams wait for its end"""
    s = B().Solver(B().tsp(I.tsp_coords(n, seed=n)), B().params(P, P // 5, P // 10, 0.7, 2, seed=1))
    threads, groups, ctas, staged, length = launches(s)
    assert s.info == (threads, groups, ctas, staged)
    assert 4 * threads * groups >= n and ctas <= 148 and staged == 1
    if 2 * ctas < 148:
        assert length == 128
    else:
        # half a millisecond at 1.9 GHz and three cycles a key and SM, or one generation
        assert 1 <= length <= max(1, 0.5e-3 * 1.9e9 / (3.0 * n * P / 148))
    s.close()


def test_info_of_separate_launches(cuda):
    s = B().Solver(B().tsp(I.tsp_coords(100, seed=1)), B().params(200, 40, 20, 0.7, 2, seed=1, num_islands=2))
    assert launches(s)[4] == 0
    s.close()


@pytest.mark.parametrize("n,P", [(300, 600), (600, 1000), (700, 500), (1000, 512), (2000, 256), (3000, 256)])
def test_room_for_other_engines(cuda, n, P):
    """threads a row: an SM's rows leave room for another launch's CTA, unless the row's length asks
    for more; and engines at once give what they give one by one"""
    def solver(seed):
        return B().Solver(B().tsp(I.tsp_coords(n, seed=n)), B().params(P, P // 5, P // 10, 0.7, 60, seed=seed))

    threads = solver(1).info[0]
    assert threads * -(-P // 148) <= 768 or 16 * (threads // 2) < n
    one_by_one = [run_population(solver(i), 40) for i in range(3)]
    together = [solver(i) for i in range(3)]
    for s in together:
        s.initialize()
        s.evolve(40)
    for s, want in zip(together, one_by_one):
        for a, b in zip(s.get_population(), want):
            np.testing.assert_array_equal(a, b)
        s.close()
