"""A device-resident advance whose waits run out (injected): the error
is the advancing PDE's own, reported also after an asynchronous advance, kept
until the state is set again, and nothing else of the context is affected."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu

TIMEOUT = -4
DT = 1e-3


def heat(ctx, N, T):
    xyz, st = sphere_problem(N, 31, 3)
    grid = R.Grid(ctx, xyz, st)
    der = R.RBFFD(R.LSFC, grid, 2)
    der.setWeights(R.LSFC, np.random.default_rng(1).standard_normal((N, 31)))
    return grid, lambda: R.HeatSphere(grid, der, 0.7, dtype=R.F64, ntracers=T)


def expect_timeout(call):
    with pytest.raises(R.RbffdError) as e:
        call()
    assert e.value.status == TIMEOUT


# one tracer: a word per thread; seven: several words per thread
@pytest.mark.parametrize("T", [1, 7])
@pytest.mark.parametrize("asynchronous", [False, True])
def test_wait_runs_out(ctx, T, asynchronous):
    N = 3000
    grid, make = heat(ctx, N, T)
    u0 = np.random.default_rng(2).standard_normal((N, T) if T > 1 else N)
    pde, other, ref = make(), make(), make()
    ref.setShape(1, 128)
    for p in (pde, other, ref):
        p.fillInitialConditions(u0)
        p.advance(R.RK4, DT, 4)
    t = pde.getTime()
    pde.injectWaitFailure()
    if asynchronous:
        pde.advance(R.RK4, DT, 6, asynchronous=True)
        try:
            pde.advance(R.RK4, DT, 6, asynchronous=True)  # refused if the first is known to have ended
        except R.RbffdError as e:
            assert e.status == TIMEOUT
        expect_timeout(ctx.synchronize)
    else:
        expect_timeout(lambda: pde.advance(R.RK4, DT, 6))
    for _ in range(2):  # until the state is set again
        expect_timeout(pde.getLocalSolution)
        expect_timeout(lambda: pde.advance(R.RK4, DT, 1))
        expect_timeout(lambda: pde.advance(R.RK4, DT, 1, unfused=True))
        expect_timeout(ctx.synchronize)
    assert pde.getTime() == t
    # another PDE of the context and grid
    other.advance(R.RK4, DT, 6)
    ref.advance(R.RK4, DT, 6)
    assert np.array_equal(other.getLocalSolution(), ref.getLocalSolution())
    assert other.getTime() == ref.getTime()
    # a new state, no more failures
    pde.injectWaitFailure(False)
    pde.fillInitialConditions(u0)
    ctx.synchronize()
    pde.advance(R.RK4, DT, 10)
    assert np.array_equal(pde.getLocalSolution(), ref.getLocalSolution())
    # destroyed while failed: the context is clean again
    pde.injectWaitFailure()
    expect_timeout(lambda: pde.advance(R.RK4, DT, 1))
    pde.close()
    ctx.synchronize()
    other.close()
    ref.close()
    grid.close()
