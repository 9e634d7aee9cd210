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


def timeout(call):
    with pytest.raises(RuntimeError) as e:
        call()
    assert e.value.code == TIMEOUT


def solvers():
    import instances as I
    return {"one": lambda: B().Solver(B().tsp(I.tsp_coords(60, seed=1)), B().params(200, 40, 20, 0.7, 30, seed=5)),
            "two": lambda: B().Solver(B().bitsp(I.tsp_coords(31, seed=1), I.tsp_coords(31, seed=2)),
                                      B().params(200, 0, 20, 0.7, 30, seed=5))}


@pytest.mark.parametrize("which", ["one", "two"])
def test_every_call_says_so(cuda, which, monkeypatch):
    s = solvers()[which]()
    monkeypatch.setenv("BRKGA_WAIT_POLLS", "0")
    timeout(s.run)
    timeout(s.synchronize)
    timeout(s.get_fitness_history)
    timeout(s.get_population)
    timeout(lambda: s.evolve(1))
    other = solvers()[which]()  # its flag is its own
    monkeypatch.delenv("BRKGA_WAIT_POLLS")
    other.run()
    timeout(s.synchronize)
    s.run()
    np.testing.assert_array_equal(s.get_fitness_history(), other.get_fitness_history())
    s.close()
    other.close()


def test_batch_says_so(cuda, monkeypatch):
    import instances as I
    pbs = [B().bitsp(I.tsp_coords(31, seed=1), I.tsp_coords(31, seed=2)), B().tsp(I.tsp_coords(40, seed=3))]
    prms = [B().params(100, 0, 10, 0.7, 20, seed=1), B().params(100, 20, 10, 0.7, 20, seed=2)]
    monkeypatch.setenv("BRKGA_WAIT_POLLS", "0")
    batch = B().Batch(pbs, prms)
    timeout(batch.synchronize)
    timeout(lambda: batch.evolve(3))
    timeout(batch.best)
    timeout(lambda: batch.best_keys(1))
    batch.close()
    monkeypatch.delenv("BRKGA_WAIT_POLLS")
    batch = B().Batch(pbs, prms)
    batch.evolve(3)
    assert np.isfinite(batch.best()[0]).all() and np.isfinite(batch.best()[1, 0])
    batch.close()


def test_server_fails_the_request_alone(cuda, monkeypatch):
    import instances as I
    server = B().Server(generations_per_tick=5)
    monkeypatch.setenv("BRKGA_WAIT_POLLS", "0")
    bad = server.submit(prm=B().params(100, 0, 10, 0.7, 20, seed=1), kind=B().BITSP_COORDS, n=30,
                        coords=I.tsp_coords(31, seed=1), coords2=I.tsp_coords(31, seed=2))
    good = server.submit(prm=B().params(100, 20, 10, 0.7, 20, seed=2), kind=B().TSP_COORDS, n=40,
                         coords=I.tsp_coords(40, seed=3))
    server.step()
    monkeypatch.delenv("BRKGA_WAIT_POLLS")
    late = server.submit(prm=B().params(100, 0, 10, 0.7, 20, seed=1), kind=B().BITSP_COORDS, n=30,
                         coords=I.tsp_coords(31, seed=1), coords2=I.tsp_coords(31, seed=2))
    for _ in range(12):
        server.step()
    assert server.poll(bad)[0] == TIMEOUT
    for rid in (good, late):
        status, best, gens, _ = server.poll(rid)
        assert status == 0 and gens == 20 and np.isfinite(best[0])
    server.close()


@pytest.mark.parametrize("value", ["", "many", "-1", "12x", "99999999999999999999"])
def test_limits_that_are_no_number(cuda, value, monkeypatch):
    """a value that is no number, or one past the limit, leaves the limit as it is"""
    monkeypatch.setenv("BRKGA_WAIT_POLLS", value)
    for make in solvers().values():
        s = make()
        s.run()
        s.close()
