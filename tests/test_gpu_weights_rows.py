"""The default elimination of the weight solves (one row per thread, panels of
8 steps, delayed updates on the FP64 tensor cores, quotients by reciprocals)
against the elimination that applies every step to the whole trailing matrix
with plain divisions and fused multiply-adds: the same weights bit for bit, at
the system sizes where its tiles and warps end."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu

SFC = R.XSFC | R.YSFC | R.ZSFC
ADVECT = R.LAMBDA | R.THETA | R.HV
EIGHT = R.X | R.Y | R.Z | R.LAPL | R.R | R.HV | R.LSFC | R.INTERP


def both(ctx, xyz, st, types, deg, eps, st_len=None, degs=None):
    """Weights by the default and by the unblocked elimination (None where the call refuses)."""
    out = []
    try:
        for method in (R.ELIM_AUTO, R.ELIM_UNBLOCKED):
            ctx.setWeightsElimination(method)
            grid = R.Grid(ctx, xyz, st, st_len=st_len)
            der = R.RBFFD(types, grid, 2)
            der.setEpsilon(eps)
            der.setHVScalars(4, 1e-3)
            der.setPolynomialDegree(deg, degs)
            try:
                der.computeAllWeightsForAllStencils()
                out.append([der.getWeights(1 << b) for b in range(16) if types >> b & 1])
            except R.RbffdError as e:
                out.append(str(e))
            grid.close()
    finally:
        ctx.setWeightsElimination(R.ELIM_AUTO)
    return out


def same(a, b):
    if isinstance(a, str) or isinstance(b, str):
        return a == b
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


# n + polynomial terms: panels (8), warps (32), two rows per thread (33 to 48), the largest
@pytest.mark.parametrize("m", [2, 7, 8, 9, 16, 17, 31, 32, 33, 40, 48, 49, 63, 64, 65, 95, 96, 97, 127, 128, 129, 159,
                               160])
@pytest.mark.parametrize("types,eps_h", [(R.LSFC, 0.4), (ADVECT, 1.5), (EIGHT, 0.7)])
def test_same_bits_at_tile_edges(ctx, m, types, eps_h):
    N = 700
    xyz, st = sphere_problem(N, 160, 31)
    deg, n = (0, m - 1) if m < 20 else (2, m - 6)
    a, b = both(ctx, xyz, np.ascontiguousarray(st[:, :n]), types, deg, eps_h / np.sqrt(4 * np.pi / N))
    assert same(a, b)
    assert isinstance(a, str) or all(np.isfinite(w).all() for w in a)


@pytest.mark.parametrize("eps_h", [0.02, 8.0, 14.0, 60.0])
def test_same_bits_far_from_one(ctx, eps_h):
    """Nearly singular systems, and kernel values that leave the range of the
    reciprocal quotients (2^-400 .. 2^400) down to zero."""
    N = 900
    xyz, st = sphere_problem(N, 50, 3)
    a, b = both(ctx, xyz, st, SFC, 3, eps_h / np.sqrt(4 * np.pi / N))
    assert same(a, b)


@pytest.mark.parametrize("n,deg", [(19, -1), (27, 0), (45, 2), (90, 1)])
def test_same_bits_with_ties(ctx, n, deg):
    """Nodes with the cube's symmetries: equal distances, so equal pivot candidates."""
    k = 8
    g = (np.arange(k) + 0.5) / k * 2 - 1
    face = np.array([(x, y) for x in g for y in g])
    pts = []
    for ax in range(3):
        for sgn in (-1.0, 1.0):
            p = np.insert(face, ax, sgn, axis=1)
            pts.append(p / np.linalg.norm(p, axis=1)[:, None])
    xyz = np.ascontiguousarray(np.concatenate(pts))
    st = R.knn_stencils(xyz, n)
    a, b = both(ctx, xyz, st, SFC, deg, 3.0)
    assert same(a, b)


def test_same_bits_mixed_sizes(ctx):
    """Twenty system sizes in one call, over several waves of systems."""
    N = 12000
    xyz, st = sphere_problem(N, 101, 9)
    rng = np.random.default_rng(2)
    degs = rng.integers(0, 5, N).astype(np.int32)
    lens = rng.choice(np.array([30, 44, 62, 101], dtype=np.int32), N)
    a, b = both(ctx, xyz, st, SFC, 0, 0.5 / np.sqrt(4 * np.pi / N), st_len=lens, degs=degs)
    assert not isinstance(a, str)
    assert same(a, b)
