"""Point sets whose box is thin along an axis, and dense clusters: the host
search's lists, and a search that does not visit every point of a flat set."""
import time

import numpy as np
import pytest

import rbffd_gpu_b200 as R

pytestmark = pytest.mark.gpu


def points(kind, N, rng):
    x = rng.random((N, 3))
    if kind == "cube":
        return x
    if kind == "line":
        return x * (1.0, 0.0, 0.0)
    if kind == "slanted line":
        return np.outer(rng.random(N), (1.0, 0.5, -0.25))
    if kind == "slab":
        return x * (1.0, 1.0, 1e-9)
    if kind == "rod":
        return x * (1e-9, 1.0, 1e-5)
    if kind == "dense half":
        x[N // 2:] *= 1e-3
        return x
    return np.concatenate([x[: N // 3] * 0.01, 0.99 + 0.01 * x[N // 3: N // 2], x[N // 2:]])  # clusters in corners


@pytest.mark.parametrize("kind", ["line", "slanted line", "slab", "rod", "dense half", "corners"])
@pytest.mark.parametrize("N,n", [(40, 40), (700, 5), (4000, 31), (9000, 101)])
def test_host_lists(ctx, kind, N, n):
    xyz = np.ascontiguousarray(points(kind, N, np.random.default_rng(N)))
    dev, td = R.knn_stencils_gpu(ctx, xyz, n, return_ties=True)
    host, th = R.knn_stencils(xyz, n, return_ties=True)
    assert np.array_equal(dev, host) and td == th
    st, ln = R.generate_stencils_gpu(ctx, xyz, n, R.ST_BRUTE_FORCE, 0.3)
    hs, hl = R.generate_stencils(xyz, n, R.ST_BRUTE_FORCE, 0.3)
    assert np.array_equal(ln, hl) and np.array_equal(st, hs)


def test_flat_sets_are_not_searched_whole(ctx):
    """A cell of a flat set holds about the points of one in a cube, so a call takes about as long; visiting all took some 25 times that."""
    N, n = 20000, 31

    def seconds(kind):
        xyz = np.ascontiguousarray(points(kind, N, np.random.default_rng(1)))
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            R.knn_stencils_gpu(ctx, xyz, n)
            best = min(best, time.perf_counter() - t)
        return best

    cube, slab = seconds("cube"), seconds("slab")
    assert slab < 3.0 * cube, (slab, cube)
