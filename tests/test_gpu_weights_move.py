"""Weights in and out of a grid (rbffd_weights_set / _get): what was set comes
back, zero beyond each stencil's length, at sizes around the slices of 32 rows
and chunks of 4 slots, and in one or several parts of the staging buffer."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n", [(1, 1), (31, 4), (32, 5), (33, 7), (500, 31), (20761, 101), (45001, 50)])
def test_round_trip(ctx, N, n):
    rng = np.random.default_rng(N)
    st = rng.integers(0, N, (N, n)).astype(np.int32)
    st[:, 0] = np.arange(N)
    lens = rng.integers(1, n + 1, N).astype(np.int32)
    grid = R.Grid(ctx, R.fibonacci_nodes(N, 4) if N > 1 else np.array([[0.0, 0.0, 1.0]]), st, st_len=lens)
    der = R.RBFFD(R.LSFC, grid, 2)
    W = rng.standard_normal((N, n))
    der.setWeights(R.LSFC, W)
    W[np.arange(n)[None, :] >= lens[:, None]] = 0.0
    assert np.array_equal(der.getWeights(R.LSFC), W)
    der.setWeights(R.HV, 2.0 * W)
    assert np.array_equal(der.getWeights(R.HV), 2.0 * W) and np.array_equal(der.getWeights(R.LSFC), W)
    grid.close()
