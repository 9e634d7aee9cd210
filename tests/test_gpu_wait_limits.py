"""Waits between the CTAs of one launch that run out: the call says so, nothing is left in flight,
and the next call is as good as any.  BRKGA_WAIT_POLLS shortens the waits; at 0 each gives up
at once, in between some CTAs of a cluster give up a front before others do."""
import numpy as np
import pytest

import oracle as O
from test_gpu_ops import B

pytestmark = pytest.mark.gpu

TIMEOUT = -4


def rank(obj, cuda):
    import torch
    out = torch.full((len(obj),), -7, dtype=torch.int32, device=cuda)
    B().pareto_rank(torch.from_numpy(obj).to(cuda), len(obj), 2, out)
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [200, 1000, 2000, 4096])
def test_ranks_after_waits_ran_out(cuda, n, monkeypatch):
    obj = np.random.default_rng(n).random((n, 2)).astype(np.float32)
    want = O.pareto_ranks(obj)
    for polls in (0, 1, 2, 3, 5, 8, 13, 21):
        monkeypatch.setenv("BRKGA_WAIT_POLLS", str(polls))
        for _ in range(4):
            try:
                got = rank(obj, cuda)
            except RuntimeError as e:
                assert e.code == TIMEOUT
            else:
                assert polls > 0
                np.testing.assert_array_equal(got, want)
    monkeypatch.delenv("BRKGA_WAIT_POLLS")
    np.testing.assert_array_equal(rank(obj, cuda), want)


def run_population(s, gens):
    s.initialize()
    s.evolve(gens)
    return s.get_population()


# 16, 4 and 1 CTAs a cluster; (0 generations: the initial ranking alone)
@pytest.mark.parametrize("n,P", [(30, 2048), (100, 500), (20, 120)])
def test_two_objectives_after_waits_ran_out(cuda, n, P, monkeypatch):
    import instances as I
    pb = B().bitsp(I.tsp_coords(n + 1, seed=n), I.tsp_coords(n + 1, seed=n + 1))
    s = B().Solver(pb, B().params(P, 0, P // 10, 0.7, 40, seed=5))
    want = run_population(s, 8)
    for polls in (0, 3, 10, 30, 100):
        monkeypatch.setenv("BRKGA_WAIT_POLLS", str(polls))
        try:
            got = run_population(s, 8)
        except RuntimeError as e:
            assert e.code == TIMEOUT
        else:
            assert polls > 0
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
        monkeypatch.delenv("BRKGA_WAIT_POLLS")
        for a, b in zip(run_population(s, 8), want):
            np.testing.assert_array_equal(a, b)
    s.close()


# 32, 64 and 128 threads a row, and local search
@pytest.mark.parametrize("n,P,ls", [(52, 256, 0), (300, 700, 0), (1500, 300, 0), (40, 300, 2)])
def test_one_objective_after_waits_ran_out(cuda, n, P, ls, monkeypatch):
    import instances as I
    if ls:
        pb = B().tspj(*I.tspj_instance(n, seed=n))
    else:
        pb = B().tsp(I.tsp_coords(n, seed=n))
    extra = dict(local_search_interval=ls, local_search_individuals=20) if ls else {}
    s = B().Solver(pb, B().params(P, P // 5, P // 10, 0.7, 400, seed=5, **extra))
    want = run_population(s, 200)
    for polls in (0, 1, 2, 4, 16):
        monkeypatch.setenv("BRKGA_WAIT_POLLS", str(polls))
        try:
            got = run_population(s, 200)
        except RuntimeError as e:
            assert e.code == TIMEOUT
        else:
            assert polls > 0
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
        monkeypatch.delenv("BRKGA_WAIT_POLLS")
        for a, b in zip(run_population(s, 200), want):
            np.testing.assert_array_equal(a, b)
    s.close()
