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
