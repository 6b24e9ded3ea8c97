"""The device's binning and shell search on point sets that stress them: few
points, points on a line or in a plane (one cell along an axis), dense clusters
in an empty box (many shells, and more candidates than the buffer holds), and
cell counts past one tile of the scan: the host search's lists and tie counts."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R

pytestmark = pytest.mark.gpu


def points(kind, N, rng):
    if kind == "line":
        return np.stack([rng.random(N), np.zeros(N), np.full(N, 3.0)], axis=1)
    if kind == "plane":
        return np.stack([rng.random(N), np.full(N, -1.0), rng.random(N)], axis=1)
    if kind == "clusters":
        x = 1e-4 * rng.standard_normal((N, 3))
        x[: N // 2] += 5.0
        x[0] = (6.0, -0.5, 2.0)
        return x
    if kind == "cube":
        return rng.random((N, 3))
    return np.round(rng.random((N, 3)) * 6) / 6  # a coarse lattice: duplicates and ties


@pytest.mark.parametrize("kind", ["line", "plane", "clusters", "cube", "lattice"])
@pytest.mark.parametrize("N,n", [(1, 1), (2, 2), (33, 33), (300, 7), (5000, 31), (6000, 120)])
def test_host_lists(ctx, kind, N, n):
    xyz = np.ascontiguousarray(points(kind, N, np.random.default_rng(N + n)))
    dev, td = R.knn_stencils_gpu(ctx, xyz, n, return_ties=True)
    host, th = R.knn_stencils(xyz, n, return_ties=True)
    assert np.array_equal(dev, host) and td == th
    st, ln = R.generate_stencils_gpu(ctx, xyz, n, R.ST_BRUTE_FORCE, 0.4)
    hs, hl = R.generate_stencils(xyz, n, R.ST_BRUTE_FORCE, 0.4)
    assert np.array_equal(ln, hl) and np.array_equal(st, hs)
