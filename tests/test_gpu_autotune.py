"""The stage-shape autotuner, on problems that do not run device-resident: the
state and a compensated state's correction come through its timed steps
untouched, and tiles take the tracer counts they are made for."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.test_gpu_grid_rk4 import make, random_operators

pytestmark = pytest.mark.gpu

P = R.TimeDependentPDE


def set_shape(pde, shape, flags):
    lanes, block, rows = shape
    if rows == 0:
        pde.setShape(lanes, block)
    else:
        pde.setTiledShape(rows, lanes, stream_weights=bool(flags & P.TILE_STREAM_WEIGHTS),
                          slot_schedule=bool(flags & P.TILE_SLOT_SCHEDULE), prefetch=bool(flags & P.TILE_PREFETCH),
                          pipeline=bool(flags & P.TILE_PIPELINE), double_buffer=bool(flags & P.TILE_DOUBLE_BUFFER))


# 16 tracers; and one tracer with rows too long for the resident kernel
@pytest.mark.parametrize("N,n,T", [(20000, 31, 16), (1000, 260, 1)])
@pytest.mark.parametrize("kind,dtype,comp", [("heat", R.F64, False), ("heat", R.F32, False), ("heat", R.F32, True),
                                             ("hv", R.F64, False), ("fused", R.F32, True)])
@pytest.mark.parametrize("graph", [False, True])
def test_state_untouched(N, n, T, kind, dtype, comp, graph):
    c = R.Context(0)  # a fresh context: no tuned shape kept yet
    xyz = R.fibonacci_nodes(N, 6)
    grid, der = random_operators(c, xyz, R.knn_stencils(xyz, n), 1)
    u0 = np.random.default_rng(7).standard_normal((N, T) if T > 1 else N)
    out = []
    for forced in (False, True):
        pde = make(grid, der, kind, dtype, T)
        pde.setCompensatedState(comp)
        pde.fillInitialConditions(u0)
        pde.setShape(1, 128)
        pde.advance(R.RK4, 1e-3, 5)  # the correction is not zero when the tuner runs
        if forced:
            set_shape(pde, shape, flags)
        else:
            pde.setShape()
        pde.advance(R.RK4, 1e-3, 30, graph=graph)
        assert pde.getPath() == (P.PATH_STAGES, 120)
        shape, flags = pde.getShape(), pde.getTileFlags()
        out.append(pde.getLocalSolution())
        pde.close()
    assert np.isfinite(out[1]).all() and np.array_equal(*out)
    grid.close()
    c.close()


# tracers in whole 16-byte vectors, a power of two of them
@pytest.mark.parametrize("kind,dtype,takes", [("heat", R.F32, (1, 4, 8, 16, 32)), ("hv", R.F64, (1, 2, 4, 8, 16, 32)),
                                              ("advect", R.F32, (1, 4, 8, 16, 32))])
def test_tiles_take_their_tracer_counts(ctx, kind, dtype, takes):
    N, n = 1999, 23
    xyz = R.fibonacci_nodes(N, 3)
    grid, der = random_operators(ctx, xyz, R.knn_stencils_gpu(ctx, xyz, n), 1)
    for T in (1, 2, 3, 4, 6, 8, 12, 16, 32):
        pde = make(grid, der, kind, dtype, T)
        if T in takes:
            pde.setTiledShape(32, 1)
            pde.advance(R.RK4, 1e-3, 1)
            assert pde.getShape() == (1, 0, 32) and pde.getPath() == (P.PATH_STAGES, 4)
        else:
            with pytest.raises(R.RbffdError) as e:
                pde.setTiledShape(32, 1)
            assert e.value.status == -5
        pde.close()
    grid.close()
