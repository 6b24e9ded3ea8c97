"""Which elimination solved the weights (rbffd_weights_get_solved): the
row-per-thread one at every size the bit comparisons of the default name, which
all succeed, and the forced ones where they are forced."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem
from tests.test_gpu_weights_rows import ADVECT, EIGHT, SFC

pytestmark = pytest.mark.gpu


def solve(ctx, xyz, st, types, deg, eps, degs=None, st_len=None):
    grid = R.Grid(ctx, xyz, st, st_len=st_len)
    der = R.RBFFD(types, grid, 2)
    der.setEpsilon(eps)
    der.setHVScalars(4, 1e-3)
    der.setPolynomialDegree(deg, degs)
    der.computeAllWeightsForAllStencils()
    solved = der.getSolvedSystems()
    grid.close()
    return solved


@pytest.mark.parametrize("m", [2, 7, 8, 9, 16, 17, 31, 32, 33, 40, 48, 49, 63, 64, 65, 95, 96, 97, 127, 128, 129, 159,
                               160])
@pytest.mark.parametrize("types,eps_h", [(R.LSFC, 0.4), (ADVECT, 1.5), (EIGHT, 0.7)])
def test_rows_at_every_size(ctx, m, types, eps_h):
    N = 700
    xyz, st = sphere_problem(N, 160, 31)
    deg, n = (0, m - 1) if m < 20 else (2, m - 6)
    assert solve(ctx, xyz, np.ascontiguousarray(st[:, :n]), types, deg, eps_h / np.sqrt(4 * np.pi / N)) == {R.ELIM_ROWS: N}


@pytest.mark.parametrize("eps_h", [0.02, 8.0, 14.0, 60.0])
def test_rows_far_from_one(ctx, eps_h):
    N = 900
    xyz, st = sphere_problem(N, 50, 3)
    assert solve(ctx, xyz, st, SFC, 3, eps_h / np.sqrt(4 * np.pi / N)) == {R.ELIM_ROWS: N}


def test_rows_in_mixed_batches_and_forced_methods(ctx):
    N = 12000
    xyz, st = sphere_problem(N, 101, 9)
    rng = np.random.default_rng(2)
    degs = rng.integers(0, 5, N).astype(np.int32)
    lens = rng.choice(np.array([30, 44, 62, 101], dtype=np.int32), N)
    assert solve(ctx, xyz, st, SFC, 0, 0.5 / np.sqrt(4 * np.pi / N), degs, lens) == {R.ELIM_ROWS: N}
    try:
        for method in (R.ELIM_UNBLOCKED, R.ELIM_BLOCKED, R.ELIM_ROW_MAP, R.ELIM_REGISTERS):
            ctx.setWeightsElimination(method)
            assert solve(ctx, xyz[:900], R.knn_stencils(xyz[:900], 60), SFC, 2, 3.0) == {method: 900}
    finally:
        ctx.setWeightsElimination(R.ELIM_AUTO)
    with pytest.raises(R.RbffdError):
        ctx.setWeightsElimination(R.ELIM_ROWS)
