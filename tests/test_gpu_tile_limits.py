"""Tiles that BRKGA_TILE or a cache file name: fewer threads than a sixty-fourth of a row's keys, or
a number of threads that no kernel has, are refused before anything is launched; the smallest
that cover a row give its result, crowded keys included."""
import os
import subprocess
import sys

import numpy as np
import pytest

import instances as I
import oracle as O
from test_gpu_ops import B

pytestmark = pytest.mark.gpu

ROWS, N = 40, 8000


def solver(n, P=ROWS):
    return B().Solver(B().tsp(I.tsp_coords(n, seed=n)), B().params(P, 8, 4, 0.7, 2, seed=3))


@pytest.mark.parametrize("tile", ["32,63", "64,32", "96,32", "-32,-63", "2048,1"])
def test_forced_tile_refused(cuda, tile, monkeypatch):
    monkeypatch.setenv("BRKGA_TILE", tile)
    with pytest.raises(RuntimeError, match="no row kernel"):
        solver(N)


@pytest.mark.parametrize("n,threads", [(2048, 32), (2049, 64), (4096, 64), (8192, 128)])
def test_smallest_tile_of_a_row(cuda, n, threads, monkeypatch):
    """up to 64 keys a thread, and buckets whose keys are ranked one by one"""
    monkeypatch.setenv("BRKGA_TILE", f"{threads},16")
    s = solver(n)
    assert s.info[0] == threads and s.info[1] == -(-n // (4 * threads))
    keys = I.keys(ROWS, n, seed=n)
    keys[:, :20 * 97:97] = (0.25 + 1e-7 * np.arange(20)).astype(np.float32)
    keys[:, 1:40:2] = np.float32(0.75)
    s.set_population(keys)
    po = O.OracleProblem(O.TSP_COORDS, n, xy=I.tsp_coords(n, seed=n))
    fit = O.evaluate(po, keys)
    _, got = s.get_population()
    np.testing.assert_array_equal(np.sort(got), np.sort(fit))
    s.close()


@pytest.mark.parametrize("line", ["1 8000 160 32 63", "1 8000 160 0 0"])
def test_cached_tile_refused(cuda, line, tmp_path):
    """(kind, keys, rows, threads, groups); the file is read once a process: a process of its own"""
    path = tmp_path / "tiles"
    path.write_text(line + "\n")
    code = ("import brkga_b200 as B, numpy as np\n"
            "try:\n"
            "    B.Solver(B.tsp(np.random.default_rng(1).random((8000, 2), dtype=np.float32)),\n"
            "             B.params(160, 8, 4, 0.7, 2, seed=3, num_islands=4))\n"
            "except RuntimeError as e:\n"
            "    print(e)\n")
    env = dict(os.environ, BRKGA_TUNE_CACHE=str(path), PYTHONPATH=os.pathsep.join(sys.path))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "no row kernel" in r.stdout
