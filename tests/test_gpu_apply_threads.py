"""Derivatives of different fields taken on one grid by several threads at once:
each gets its own field's, though the buffers kept with the grid are shared."""
import threading

import numpy as np
import pytest

import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# a look-up per slot, a reordered field, and the renumbered stencils of wide records
@pytest.mark.parametrize("N,T,host", [(4000, 1, True), (70000, 1, True), (70000, 1, False), (70000, 2, False),
                                      (4000, 16, False)])
def test_threads(ctx, N, T, host):
    n, K, calls = 9, 4, 60
    if N < 20000:
        xyz, st = sphere_problem(N, n, 5)
    else:
        xyz = R.fibonacci_nodes(N, 5)
        st = R.knn_stencils_gpu(ctx, xyz, n)
    grid = R.Grid(ctx, xyz, st)
    der = R.RBFFD(R.LSFC, grid, 2)
    rng = np.random.default_rng(3)
    W = rng.standard_normal((N, n))
    der.setWeights(R.LSFC, W)
    fields = [rng.standard_normal((N, T)) for _ in range(K)]
    expect = []
    for f in fields:  # products and sums fused one by one, in slot order, by a call of its own
        d, o = torch.from_numpy(f).cuda(), torch.empty(N, T, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        der.applyWeightsForDerivDev(R.LSFC, d.data_ptr(), o.data_ptr(), ntracers=T)
        expect.append(o.cpu().numpy())
    bad = []

    def work(k):
        d, o = torch.from_numpy(fields[k]).cuda(), torch.empty(N, T, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        u = np.ascontiguousarray(fields[k][:, 0])
        for _ in range(calls):
            if host:
                got = der.applyWeightsForDeriv(R.LSFC, u)[:, None]
            else:
                der.applyWeightsForDerivDev(R.LSFC, d.data_ptr(), o.data_ptr(), ntracers=T)
                got = o.cpu().numpy()
            if not np.array_equal(got, expect[k]):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(K)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    grid.close()
