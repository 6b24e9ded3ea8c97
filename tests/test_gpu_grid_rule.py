"""Shapes at which a device-resident stage is slower than the per-stage kernels
advance per stage, and those beside them where it is faster do not."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.test_gpu_grid_rk4 import make, random_operators

pytestmark = pytest.mark.gpu

P = R.TimeDependentPDE
STAGES, RESIDENT = P.PATH_STAGES, P.PATH_RESIDENT


@pytest.mark.parametrize("N,n,kind,dtype,T,path", [
    # long rows, one tracer: 240 slots, 2/13 of the nodes, 480 slots; several tracers keep theirs
    (642, 240, "heat", R.F64, 1, RESIDENT), (642, 241, "heat", R.F64, 1, STAGES), (1200, 255, "heat", R.F32, 1, STAGES),
    (2470, 318, "hv", R.F64, 1, RESIDENT), (1000, 600, "hv", R.F64, 1, STAGES), (5499, 524, "hv", R.F64, 1, STAGES),
    (1200, 255, "heat", R.F64, 4, RESIDENT),
    # FP64 past the L2: two items per thread, three operators
    (163842, 50, "advect", R.F64, 1, STAGES), (163842, 31, "hv", R.F64, 1, RESIDENT),
    (163842, 101, "heat", R.F64, 1, RESIDENT),
    (87246, 87, "hv", R.F64, 1, STAGES), (60578, 91, "hv", R.F64, 1, RESIDENT), (123614, 95, "hv", R.F32, 1, RESIDENT),
    # three operators and several tracers in FP64
    (50000, 90, "hv", R.F64, 4, STAGES), (30000, 120, "hv", R.F64, 4, RESIDENT), (64204, 95, "hv", R.F64, 2, STAGES),
    (50000, 90, "hv", R.F64, 3, RESIDENT)])
def test_path(ctx, N, n, kind, dtype, T, path):
    xyz = R.fibonacci_nodes(N, 6)
    st = R.knn_stencils_gpu(ctx, xyz, n) if n <= 255 else R.knn_stencils(xyz, n)
    grid, der = random_operators(ctx, xyz, st, 1)
    u0 = np.random.default_rng(2).standard_normal((N, T) if T > 1 else N)
    out = []
    for shape in ((), (1, 256)):
        pde = make(grid, der, kind, dtype, T)
        pde.setShape(*shape)
        pde.fillInitialConditions(u0)
        pde.advance(R.RK4, 1e-5, 2)
        assert pde.getPath()[0] == (STAGES if shape else path)
        out.append(pde.getLocalSolution())
        pde.close()
    if path == RESIDENT:
        assert np.array_equal(*out)
    else:  # the tuned shape may split a row's sum: 8 stages of n_ops n + 8 roundings
        scale = np.abs(out[1]).max()
        unit = 2.0 ** (-53 if dtype == R.F64 else -24)
        assert np.abs(out[0] - out[1]).max() <= 8 * (3 * n + 8) * unit * scale
    grid.close()
