"""Device-resident RK4 (the default path of advance on grids whose weights fit
the SMs' shared memory, at least in part): the bits of the per-stage kernels
with one lane per row, for grids of one block, ragged last blocks, full and
partial residence, every right-hand side, type and tracer count it takes."""
import threading

import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu

OPS = R.LSFC | R.LAMBDA | R.THETA | R.HV


def random_operators(ctx, xyz, st, seed, st_len=None, order=None):
    """A grid with seeded weights (sums of products, whatever the numbers)."""
    N, n = st.shape
    grid = R.Grid(ctx, xyz, st, st_len=st_len, order=order)
    der = R.RBFFD(OPS, grid, 2)
    rng = np.random.default_rng(seed)
    for b in range(16):
        if OPS >> b & 1:
            der.setWeights(1 << b, rng.standard_normal((N, n)))
    return grid, der


def make(grid, der, kind, dtype, T, seed=5):
    rng = np.random.default_rng(seed)
    if kind == "heat":
        return R.HeatSphere(grid, der, 0.7, dtype=dtype, ntracers=T)
    cu, cv = rng.standard_normal(grid.N), rng.standard_normal(grid.N)
    pde = R.Advection(grid, der, cu, None if kind == "rollup" else cv, kind != "advect", dtype=dtype, ntracers=T)
    if kind == "fused":
        pde.setFusedOperator(True)
    return pde


def both(grid, der, kind, dtype, T, steps, dt=1e-3, comp=False, graph=True, calls=1):
    """The state after `steps` steps (in `calls` calls), device-resident and with one lane per row per stage."""
    u0 = np.random.default_rng(7).standard_normal((grid.N, T) if T > 1 else grid.N)
    out = []
    for forced in (False, True):
        pde = make(grid, der, kind, dtype, T)
        if comp:
            pde.setCompensatedState(True)
        if forced:
            pde.setShape(1, 128)
        pde.fillInitialConditions(u0)
        for c in range(calls):
            pde.advance(R.RK4, dt, steps, graph=graph)
        out.append(pde.getLocalSolution())
        if not forced:
            assert pde.getShape() == (1, 256, 0) and pde.getTileFlags() == 0
        pde.close()
    assert np.isfinite(out[1]).all()
    return out


@pytest.mark.parametrize("N", [5, 31, 33, 64, 700, 4737])
@pytest.mark.parametrize("kind,dtype", [("heat", R.F64), ("hv", R.F64), ("advect", R.F32), ("rollup", R.F64),
                                        ("fused", R.F32)])
def test_same_bits(ctx, N, kind, dtype):
    n = min(N, 31)
    xyz, st = sphere_problem(N, n, 2)
    grid, der = random_operators(ctx, xyz, st, 1)
    a, b = both(grid, der, kind, dtype, 1, 6)
    assert np.array_equal(a, b)
    grid.close()


@pytest.mark.parametrize("T", [2, 3, 4, 5, 7, 16])
@pytest.mark.parametrize("kind,dtype", [("heat", R.F32), ("hv", R.F64)])
def test_same_bits_tracers(ctx, T, kind, dtype):
    xyz, st = sphere_problem(3001, 23, 4)
    grid, der = random_operators(ctx, xyz, st, 3)
    a, b = both(grid, der, kind, dtype, T, 5)
    assert np.array_equal(a, b)
    grid.close()


# rows per SM and chunks per row: weights on chip, in part on chip, two items per thread, tracer vectors
@pytest.mark.parametrize("N,n,kind,dtype,T", [(60000, 20, "heat", R.F64, 1), (60000, 60, "hv", R.F64, 1),
                                              (160000, 20, "heat", R.F32, 1), (160000, 31, "heat", R.F64, 1),
                                              (160000, 17, "hv", R.F32, 1), (40962, 41, "hv", R.F64, 4),
                                              (50000, 20, "heat", R.F32, 4), (70000, 25, "advect", R.F64, 2)])
def test_same_bits_large(ctx, N, n, kind, dtype, T):
    xyz = R.fibonacci_nodes(N, 6)
    st = R.knn_stencils_gpu(ctx, xyz, n)
    grid, der = random_operators(ctx, xyz, st, 9)
    a, b = both(grid, der, kind, dtype, T, 3, dt=1e-4)
    assert np.array_equal(a, b)
    grid.close()


def test_stencils_read_in_one_direction(ctx):
    """Every block reads the first one, which reads none of them, and lengths
    vary: the exchange still keeps its two buffers apart over many stages."""
    N, n = 1500, 17
    rng = np.random.default_rng(12)
    st = np.zeros((N, n), dtype=np.int32)
    st[:, 0] = np.arange(N)
    st[:, 1:] = rng.integers(0, 32, (N, n - 1))
    xyz = R.fibonacci_nodes(N, 3)
    lens = rng.integers(1, n + 1, N).astype(np.int32)
    grid, der = random_operators(ctx, xyz, st, 2, st_len=lens, order=2)  # the caller's order
    a, b = both(grid, der, "heat", R.F64, 1, 60, dt=1e-4)
    assert np.array_equal(a, b)
    grid.close()


@pytest.mark.parametrize("T", [1, 4])
def test_compensated_state(ctx, T):
    xyz, st = sphere_problem(2562, 31, 8)
    grid, der = random_operators(ctx, xyz, st, 4)
    a, b = both(grid, der, "heat", R.F32, T, 40, comp=True, calls=3)
    assert np.array_equal(a, b)
    grid.close()


def test_many_steps_and_calls(ctx):
    """More steps than one launch takes, and calls of one step."""
    xyz, st = sphere_problem(200, 9, 8)
    grid, der = random_operators(ctx, xyz, st, 4)
    a, b = both(grid, der, "hv", R.F64, 1, 4100, dt=1e-5)
    assert np.array_equal(a, b)
    a, b = both(grid, der, "hv", R.F64, 1, 1, calls=7, graph=False)
    assert np.array_equal(a, b)
    grid.close()


def test_weights_and_operator_changes_are_seen(ctx):
    """New weights, and the fused operator switched on and off, between calls."""
    xyz, st = sphere_problem(1000, 25, 3)
    grid, der = random_operators(ctx, xyz, st, 4)
    u0 = np.random.default_rng(1).standard_normal(1000)
    pde, ref = make(grid, der, "hv", R.F64, 1), make(grid, der, "hv", R.F64, 1)
    ref.setShape(1, 128)
    for p in (pde, ref):
        p.fillInitialConditions(u0)
        p.advance(R.RK4, 1e-3, 5)
    der.setWeights(R.HV, np.random.default_rng(99).standard_normal((1000, 25)))
    for p in (pde, ref):
        p.advance(R.RK4, 1e-3, 5)
        p.setFusedOperator(True)
        p.advance(R.RK4, 2e-3, 5)
        p.setFusedOperator(False)
        p.advance(R.RK4, 2e-3, 3, asynchronous=True)
    assert np.array_equal(pde.getLocalSolution(), ref.getLocalSolution())
    assert pde.getTime() == ref.getTime()
    pde.close()
    ref.close()
    grid.close()


def test_two_contexts_in_two_threads():
    """Device-resident advances issued at once from two contexts' threads go one behind the other."""
    xyz, st = sphere_problem(6000, 31, 5)
    results, errors = {}, []

    def work(k):
        try:
            c = R.Context(0)
            grid, der = random_operators(c, xyz, st, 10 + k)
            pde = make(grid, der, "heat", R.F64, 1)
            pde.fillInitialConditions(np.random.default_rng(k).standard_normal(6000))
            for _ in range(30):
                pde.advance(R.RK4, 1e-4, 20)
            results[k] = pde.getLocalSolution()
            ref = make(grid, der, "heat", R.F64, 1)
            ref.setShape(1, 128)
            ref.fillInitialConditions(np.random.default_rng(k).standard_normal(6000))
            ref.advance(R.RK4, 1e-4, 600, graph=True)
            results[k, "ref"] = ref.getLocalSolution()
            pde.close()
            ref.close()
            grid.close()
            c.close()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(2):
        assert np.array_equal(results[k], results[k, "ref"])
