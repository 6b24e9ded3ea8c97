"""Grids whose blocks read too many nodes for 16-bit halo positions: counted
once, advanced per stage, and the call that succeeded leaves no error message."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R

pytestmark = pytest.mark.gpu


def test_refused_halo_is_remembered():
    N, n = 120000, 120  # blocks of 832 rows of random stencils read about 67700 nodes
    c = R.Context(0)
    rng = np.random.default_rng(4)
    st = rng.integers(0, N, (N, n)).astype(np.int32)
    st[:, 0] = np.arange(N)
    grid = R.Grid(c, R.fibonacci_nodes(N, 2), st, order=R.ORDER_GIVEN)
    der = R.RBFFD(R.LSFC, grid, 2)
    der.setWeights(R.LSFC, rng.standard_normal((N, n)) / n)
    u0 = rng.standard_normal(N)
    out, held = [], []
    for forced in (False, True):
        pde = R.HeatSphere(grid, der, 0.7, dtype=R.F32)
        if forced:
            pde.setShape(1, 256)
        pde.fillInitialConditions(u0)
        pde.advance(R.RK4, 1e-3, 3)
        held.append(c.mem_info()[0])
        pde.advance(R.RK4, 1e-3, 3)
        assert c.mem_info()[0] == held[-1]
        assert c.L.rbffd_ctx_last_error(c.h) == b""
        out.append(pde.getLocalSolution())
        pde.close()
    assert np.isfinite(out[0]).all()
    assert np.abs(out[0] - out[1]).max() <= 6 * 4 * (n + 8) * 2.0 ** -24 * np.abs(out[1]).max()
    grid.close()
    c.close()


def test_sizes_are_counted_before_the_halo_is_made():
    """A PDE whose weights do not fit beside the halo costs the grid no halo but
    that of its shape."""
    N, n = 150000, 60
    c = R.Context(0)
    xyz = R.fibonacci_nodes(N, 2)
    st = R.knn_stencils_gpu(c, xyz, n)
    rng = np.random.default_rng(4)
    mixed = rng.random(N) < 0.2  # a fifth of the rows read far nodes: some 13000 nodes a block
    st[mixed, 1:] = rng.integers(0, N, (int(mixed.sum()), n - 1))
    W = rng.standard_normal((N, n)) / n
    bytes_ = []
    for run in ("tunes", "tuned", "set"):
        grid = R.Grid(c, xyz, st)
        der = R.RBFFD(R.LAMBDA | R.THETA | R.HV, grid, 2)
        for op in (R.LAMBDA, R.THETA, R.HV):
            der.setWeights(op, W)
        pde = R.Advection(grid, der, rng.standard_normal(N), rng.standard_normal(N), True, dtype=R.F32)
        if run == "set":
            lanes, block, rows = shape
            if rows:
                pde.setTiledShape(rows, lanes, stream_weights=bool(flags & 1), prefetch=bool(flags & 4))
            else:
                pde.setShape(lanes, block)
        pde.advance(R.RK4, 1e-3, 1)
        shape, flags = pde.getShape(), pde.getTileFlags()
        pde.close()
        bytes_.append(grid.nbytes())
        grid.close()
    c.close()
    assert bytes_[1] == bytes_[2]
