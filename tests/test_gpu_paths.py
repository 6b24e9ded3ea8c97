"""Which path an advance took (rbffd_pde_get_path), and that the shapes the
device-resident tests compare do run device-resident."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem
from tests.test_gpu_grid_rk4 import make, random_operators

pytestmark = pytest.mark.gpu

P = R.TimeDependentPDE


def test_paths_and_launches(ctx):
    xyz, st = sphere_problem(2000, 31, 3)
    grid, der = random_operators(ctx, xyz, st, 4)
    pde = make(grid, der, "hv", R.F64, 1)
    pde.fillInitialConditions(np.random.default_rng(1).standard_normal(2000))
    assert pde.getPath() == (P.PATH_NONE, 0)
    pde.advance(R.RK4, 1e-4, 5)
    assert pde.getPath() == (P.PATH_RESIDENT, 1) and pde.getShape() == (1, 256, 0)
    pde.advance(R.RK4, 1e-6, 2001)
    assert pde.getPath() == (P.PATH_RESIDENT, 2)
    pde.advance(R.RK4, 1e-6, 3, unfused=True)
    assert pde.getPath() == (P.PATH_UNFUSED, 3 * 4 * 4)
    pde.advance(R.RK4, 1e-6, 3, resident=True)
    assert pde.getPath() == (P.PATH_CLUSTER, 1)
    pde.setShape(1, 256)
    pde.advance(R.RK4, 1e-6, 30, graph=True)
    assert pde.getPath() == (P.PATH_STAGES, 120) and pde.getShape() == (1, 256, 0)
    pde.setTiledShape(64, 2)
    pde.advance(R.RK4, 1e-6, 3)
    assert pde.getPath() == (P.PATH_STAGES, 12) and pde.getShape()[2] == 64
    pde.setShape()  # back to the default
    pde.advance(R.RK4, 1e-6, 3)
    assert pde.getPath() == (P.PATH_RESIDENT, 1) and pde.getShape() == (1, 256, 0)
    pde.close()
    grid.close()


def test_resident_after_a_tuned_tile(ctx):
    """Three operators that do not fit are tuned (to a tile here); the fused
    operator fits, and what is reported is the path it takes."""
    N, n = 163842, 50
    xyz = R.fibonacci_nodes(N, 3)
    grid, der = random_operators(ctx, xyz, R.knn_stencils_gpu(ctx, xyz, n), 4)
    pde = make(grid, der, "hv", R.F64, 1)
    pde.advance(R.RK4, 1e-4, 1)
    tuned = pde.getShape(), pde.getTileFlags()
    assert pde.getPath() == (P.PATH_STAGES, 4) and tuned[0][2] > 0
    pde.setFusedOperator(True)
    pde.advance(R.RK4, 1e-4, 1)
    assert pde.getPath() == (P.PATH_RESIDENT, 1)
    assert pde.getShape() == (1, 256, 0) and pde.getTileFlags() == 0
    pde.setFusedOperator(False)
    pde.advance(R.RK4, 1e-4, 1)
    assert pde.getPath() == (P.PATH_STAGES, 4) and (pde.getShape(), pde.getTileFlags()) == tuned
    pde.close()
    grid.close()


SMALL = [(N, min(N, 31), kind, dtype, 1) for N in (5, 31, 33, 64, 700, 4737)
         for kind, dtype in (("heat", R.F64), ("hv", R.F64), ("advect", R.F32), ("rollup", R.F64), ("fused", R.F32))]
TRACERS = [(3001, 23, kind, dtype, T) for T in (2, 3, 4, 5, 7, 16) for kind, dtype in (("heat", R.F32), ("hv", R.F64))]
LARGE = [(60000, 20, "heat", R.F64, 1), (60000, 60, "hv", R.F64, 1), (160000, 20, "heat", R.F32, 1), (160000, 31, "heat", R.F64, 1),
         (160000, 17, "hv", R.F32, 1),
         (40962, 41, "hv", R.F64, 4), (50000, 20, "heat", R.F32, 4),
         (70000, 25, "advect", R.F64, 2)]


@pytest.mark.parametrize("N,n,kind,dtype,T", SMALL + TRACERS + LARGE)
def test_runs_device_resident(ctx, N, n, kind, dtype, T):
    if N < 20000:
        xyz, st = sphere_problem(N, n, 2)
    else:
        xyz = R.fibonacci_nodes(N, 6)
        st = R.knn_stencils_gpu(ctx, xyz, n)
    grid, der = random_operators(ctx, xyz, st, 1)
    pde = make(grid, der, kind, dtype, T)
    pde.advance(R.RK4, 1e-4, 1)
    assert pde.getPath() == (P.PATH_RESIDENT, 1)
    pde.close()
    grid.close()
