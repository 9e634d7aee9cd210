"""The peel of more than 2048 points on eight CTAs, for devices that cannot place clusters of 16
(BRKGA_PEEL_CLUSTER=8): around a CTA's share of 512 points, a quarter's words and the end of the
range; many equal values, one-point fronts, NaN and infinities; survivors of generations."""
import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_ops import B
from test_gpu_peel import points
from test_gpu_wait_limits import TIMEOUT, rank, run_population

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def eight(monkeypatch):
    monkeypatch.setenv("BRKGA_PEEL_CLUSTER", "8")


@pytest.mark.parametrize("shape", ["plain", "ties", "chain", "odd"])
@pytest.mark.parametrize("n", [2049, 2079, 2561, 3071, 3073, 4033, 4095, 4096])
def test_ranks(cuda, n, shape):
    obj = points(n, shape)
    np.testing.assert_array_equal(rank(obj, cuda), O.pareto_ranks(obj))


@pytest.mark.parametrize("P", [1025, 1500, 2048])
def test_generations(cuda, P, monkeypatch):
    pb = B().bitsp(I.tsp_coords(31, seed=P), I.tsp_coords(31, seed=P + 1))
    prm = B().params(P, 0, P // 10, 0.7, 30, seed=5)
    s = B().Solver(pb, prm)
    got = run_population(s, 30)
    monkeypatch.delenv("BRKGA_PEEL_CLUSTER")
    t = B().Solver(pb, prm)
    for a, b in zip(got, run_population(t, 30)):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(s.get_fitness_history(), t.get_fitness_history())
    s.close()
    t.close()


def test_waits_that_run_out(cuda, monkeypatch):
    obj = points(4000, "plain")
    want = O.pareto_ranks(obj)
    for polls in (0, 1, 2, 4, 8, 16, 32):
        monkeypatch.setenv("BRKGA_WAIT_POLLS", str(polls))
        try:
            np.testing.assert_array_equal(rank(obj, cuda), want)
        except RuntimeError as e:
            assert e.code == TIMEOUT
    monkeypatch.delenv("BRKGA_WAIT_POLLS")
    np.testing.assert_array_equal(rank(obj, cuda), want)
