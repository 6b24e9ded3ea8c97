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


def test_advance_beside_another_capture():
    """An asynchronous advance of a context that shares the device with another,
    issued while a thread captures a stream of its own in the global mode."""
    N, n = 3000, 31
    xyz, st = sphere_problem(N, n, 3)
    runs = []
    for k in range(2):
        c = R.Context(0)
        grid = R.Grid(c, xyz, st)
        der = R.RBFFD(R.LSFC, grid, 2)
        der.setWeights(R.LSFC, np.random.default_rng(1).standard_normal((N, n)))
        pde = R.HeatSphere(grid, der, 0.7, dtype=R.F64)
        pde.fillInitialConditions(np.random.default_rng(2).standard_normal(N))
        pde.advance(R.RK4, 1e-4, 5)
        runs.append((c, grid, der, pde))
    x = torch.ones(1000, device="cuda")
    torch.cuda.synchronize()
    recorded = torch.cuda.CUDAGraph()
    with torch.cuda.graph(recorded):
        y = x + 1
        for c, grid, der, pde in runs:  # another stream, which is not captured
            pde.advance(R.RK4, 1e-4, 20, asynchronous=True)
        y = y * 2
    recorded.replay()
    torch.cuda.synchronize()
    assert float(y.sum()) == 4000.0
    out = [pde.getLocalSolution() for c, grid, der, pde in runs]
    assert np.array_equal(*out)
    c, grid, der, pde = runs[0]
    ref = R.HeatSphere(grid, der, 0.7, dtype=R.F64)
    ref.setShape(1, 128)
    ref.fillInitialConditions(np.random.default_rng(2).standard_normal(N))
    ref.advance(R.RK4, 1e-4, 25)
    assert np.array_equal(out[0], ref.getLocalSolution())
    ref.close()
    recorded.reset()
    for c, grid, der, pde in runs:
        pde.close()
        grid.close()
        c.close()
