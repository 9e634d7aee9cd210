"""Front ranks where the cluster peel's split of the points can go wrong: around a mask word, a
pair of words (one CTA's quarter), the 256 points of a CTA, and every cluster size; many equal
values, a chain of one-point fronts (the most exchanges), NaN and infinite objectives.  Ranks
are whole numbers: compared exactly."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def points(n, shape):
    rng = np.random.default_rng(n)
    if shape == "chain":  # every point dominates all later ones
        return np.repeat(rng.permutation(n).astype(np.float32)[:, None], 2, axis=1)
    obj = rng.random((n, 2)).astype(np.float32)
    if shape == "ties":
        obj = np.floor(obj * 12).astype(np.float32)
    if shape == "odd":
        obj[rng.random(n) < 0.05, 0] = np.nan
        obj[rng.random(n) < 0.05, 1] = np.inf
        obj[rng.random(n) < 0.05, 0] = -np.inf
    return obj


@pytest.mark.parametrize("shape", ["plain", "ties", "chain", "odd"])
@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 255, 257, 511, 513, 1024, 1025, 2048, 2049, 3000, 4095, 4096])
def test_ranks_at_split_edges(cuda, n, shape):
    import brkga_b200
    import torch
    obj = points(n, shape)
    rank = torch.full((n,), -7, dtype=torch.int32, device=cuda)
    brkga_b200.pareto_rank(torch.from_numpy(obj).to(cuda), n, 2, rank)
    np.testing.assert_array_equal(rank.cpu().numpy(), O.pareto_ranks(obj))
