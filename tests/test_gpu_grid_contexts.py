"""Device-resident advances of several contexts: those whose thread blocks fit
the device together run at once, the others one behind the other, and a long
advance is issued in launches that leave the device between them."""
import time

import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu


def pdes(count, N, n):
    xyz, st = sphere_problem(N, n, 5)
    out = []
    for k in range(count):
        c = R.Context(0)
        grid = R.Grid(c, xyz, st)
        der = R.RBFFD(R.LSFC, grid, 2)
        der.setWeights(R.LSFC, np.random.default_rng(k).standard_normal((N, n)))
        pde = R.HeatSphere(grid, der, 0.7, dtype=R.F64)
        pde.fillInitialConditions(np.zeros(N))
        out.append((c, grid, der, pde))
    return out


def seconds(ps, steps, repeats=5):
    best = 1e9
    for _ in range(repeats + 1):  # the first builds halos and loads kernels
        t = time.perf_counter()
        for c, grid, der, pde in ps:
            pde.advance(R.RK4, 1e-9, steps, graph=True, asynchronous=True)
        for c, grid, der, pde in ps:
            c.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


def test_small_grids_share_the_device():
    """Four grids of 21 blocks each: about the time of one, not of four."""
    ps = pdes(4, 642, 17)
    one, four = seconds(ps[:1], 2000), seconds(ps, 2000)
    assert four < 2.5 * one, (one, four)
    for c, grid, der, pde in ps:
        pde.close()
        grid.close()
        c.close()


@pytest.mark.parametrize("sizes", [(642, 2562, 4737), (9000, 9000), (300, 4737, 4737, 642, 642)])
def test_same_bits_at_once(sizes):
    """Grids that fit together, some of them, or one at a time, with many launches in flight."""
    runs = []
    for k, N in enumerate(sizes):
        (c, grid, der, pde), = pdes(1, N, 31)
        runs.append((c, grid, der, pde, np.random.default_rng(50 + k).standard_normal(N)))
    for c, grid, der, pde, u0 in runs:
        pde.fillInitialConditions(u0)
    for _ in range(20):
        for c, grid, der, pde, u0 in runs:
            pde.advance(R.RK4, 1e-5, 30, asynchronous=True)
    for c, grid, der, pde, u0 in runs:
        got = pde.getLocalSolution()
        ref = R.HeatSphere(grid, der, 0.7, dtype=R.F64)
        ref.setShape(1, 128)
        ref.fillInitialConditions(u0)
        ref.advance(R.RK4, 1e-5, 600, graph=True)
        assert np.array_equal(got, ref.getLocalSolution())
        ref.close()
        pde.close()
        grid.close()
        c.close()


def test_long_advance_in_several_launches():
    """160000 nodes: an advance of 700 steps takes several launches, whose steps join to the same bits."""
    N, n = 160000, 31
    c = R.Context(0)
    xyz = R.fibonacci_nodes(N, 6)
    grid = R.Grid(c, xyz, R.knn_stencils_gpu(c, xyz, n))
    der = R.RBFFD(R.LSFC, grid, 2)
    der.setWeights(R.LSFC, np.random.default_rng(1).standard_normal((N, n)))
    u0 = np.random.default_rng(2).standard_normal(N)
    out = []
    for forced in (False, True):
        pde = R.HeatSphere(grid, der, 0.7, dtype=R.F64)
        if forced:
            pde.setShape(1, 128)
        pde.fillInitialConditions(u0)
        pde.advance(R.RK4, 1e-7, 700, graph=True)
        out.append(pde.getLocalSolution())
        pde.close()
    assert np.isfinite(out[1]).all() and np.array_equal(out[0], out[1])
    grid.close()
    c.close()
