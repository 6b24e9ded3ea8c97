"""Stage kernels that move the state as 16-byte vectors, and tiles whose weight
stream gives way in L2: each tracer's bits are those of a one-tracer PDE with
one lane per row."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu


def pde_of(grid, der, kind, dtype, T):
    if kind == "heat":
        return R.HeatSphere(grid, der, 0.7, dtype=dtype, ntracers=T)
    rng = np.random.default_rng(5)
    return R.Advection(grid, der, rng.standard_normal(grid.N), rng.standard_normal(grid.N), kind == "hv", dtype=dtype,
                       ntracers=T)


def setup(ctx, N, n, ops, seed):
    if N < 20000:
        xyz, st = sphere_problem(N, n, seed)
    else:
        xyz = R.fibonacci_nodes(N, seed)
        st = R.knn_stencils_gpu(ctx, xyz, n)
    grid = R.Grid(ctx, xyz, st)
    der = R.RBFFD(0, grid, 2)
    for k, op in enumerate(ops):
        der.setWeights(op, np.random.default_rng(seed + k).standard_normal((N, n)) / n)
    return grid, der


@pytest.mark.parametrize("T", [2, 4, 6, 8, 16, 32])
@pytest.mark.parametrize("kind,dtype,comp", [("heat", R.F32, True), ("hv", R.F64, False), ("advect", R.F32, False)])
def test_tracers_equal_single_runs(ctx, T, kind, dtype, comp):
    ops = (R.LSFC,) if kind == "heat" else (R.LAMBDA, R.THETA, R.HV)
    grid, der = setup(ctx, 1999, 23, ops, 3)
    u0 = np.random.default_rng(7).standard_normal((1999, T))
    out = []
    for shape in ("vec", "tile"):
        pde = pde_of(grid, der, kind, dtype, T)
        if comp:
            pde.setCompensatedState(True)
        pde.fillInitialConditions(u0)
        if shape == "vec":
            pde.setShape(1, 128)
        else:
            try:
                pde.setTiledShape(32, 1)
            except R.RbffdError:  # a tracer count the tiles do not take
                pde.close()
                continue
        pde.advance(R.RK4, 1e-2, 6)
        out.append(pde.getLocalSolution())
        pde.close()
    for t in range(T):
        pde = pde_of(grid, der, kind, dtype, 1)
        if comp:
            pde.setCompensatedState(True)
        pde.fillInitialConditions(np.ascontiguousarray(u0[:, t]))
        pde.setShape(1, 128)
        pde.advance(R.RK4, 1e-2, 6)
        ref = pde.getLocalSolution()
        for o in out:
            assert np.array_equal(o[:, t], ref)
        pde.close()
    grid.close()


# stages past the L2: three operators and one, vectors per node 2, 4 and 8
@pytest.mark.parametrize("N,n,kind,dtype,T", [(70000, 60, "hv", R.F64, 16), (110000, 80, "hv", R.F32, 8),
                                              (110000, 80, "hv", R.F32, 16), (160000, 101, "heat", R.F32, 16)])
def test_tiles_past_l2(ctx, N, n, kind, dtype, T):
    ops = (R.LSFC,) if kind == "heat" else (R.LAMBDA, R.THETA, R.HV)
    grid, der = setup(ctx, N, n, ops, 4)
    u0 = np.random.default_rng(7).standard_normal((N, T))
    out = []
    for tile in (False, True):
        pde = pde_of(grid, der, kind, dtype, T)
        pde.fillInitialConditions(u0)
        if tile:
            pde.setTiledShape(64, 1)
        else:
            pde.setShape(1, 256)
        pde.advance(R.RK4, 1e-2, 2)
        out.append(pde.getLocalSolution())
        pde.close()
    assert np.array_equal(out[0], out[1])
    grid.close()
