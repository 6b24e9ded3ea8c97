"""A caller's CUDA graph of the context's stream around asynchronous advances:
recorded per stage, on grids that otherwise advance device-resident too."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("T", [1, 4])
@pytest.mark.parametrize("advance_first", [False, True])
@pytest.mark.parametrize("graph", [False, True])
def test_replayed_advance(T, advance_first, graph):
    N, n, dt = 3000, 31, 1e-3
    c = R.Context(0)
    xyz, st = sphere_problem(N, n, 3)
    grid = R.Grid(c, xyz, st)
    der = R.RBFFD(R.LSFC, grid, 2)
    der.setWeights(R.LSFC, np.random.default_rng(1).standard_normal((N, n)))
    u0 = np.random.default_rng(2).standard_normal((N, T) if T > 1 else N)
    pde, ref = (R.HeatSphere(grid, der, 0.7, dtype=R.F64, ntracers=T) for _ in range(2))
    ref.setShape(1, 128)
    for p in (pde, ref):
        p.fillInitialConditions(u0)
        if advance_first:
            p.advance(R.RK4, dt, 2)
    torch.cuda.synchronize()
    recorded = torch.cuda.CUDAGraph()
    with torch.cuda.graph(recorded, stream=torch.cuda.ExternalStream(c.stream())):
        pde.advance(R.RK4, dt, 30, graph=graph, asynchronous=True)
    for _ in range(3):
        recorded.replay()
    torch.cuda.synchronize()
    ref.advance(R.RK4, dt, 90)
    assert np.array_equal(pde.getLocalSolution(), ref.getLocalSolution())
    # device-resident again afterwards
    for p in (pde, ref):
        p.advance(R.RK4, dt, 5)
    assert np.array_equal(pde.getLocalSolution(), ref.getLocalSolution())
    recorded.reset()
    pde.close()
    ref.close()
    grid.close()
    c.close()
