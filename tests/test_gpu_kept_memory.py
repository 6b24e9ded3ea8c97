"""Buffers kept between calls give way: a server's budget has the room it has
without them, and what needs them next has them again."""
import numpy as np
import pytest

import rbffd_gpu_b200 as R

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_server_budget():
    N, n, T = 40000, 50, 16
    xyz = R.fibonacci_nodes(N, 2)
    W = np.random.default_rng(1).standard_normal((N, n)) / n
    u0 = np.random.default_rng(2).standard_normal(N)
    fields = torch.randn(N, T, dtype=torch.float64, device="cuda")
    outs, peak, total = [], None, None
    for apply_first in (False, True):
        c = R.Context(0)
        st = R.knn_stencils_gpu(c, xyz, n)
        grid = R.Grid(c, xyz, st)
        der = R.RBFFD(R.LSFC, grid, 2)
        der.setWeights(R.LSFC, W)
        fraction = 0.5
        if apply_first:
            der.getWeights(R.LSFC)
            der.applyWeightsForDeriv(R.LSFC, u0)
            out = torch.empty_like(fields)
            torch.cuda.synchronize()
            for _ in range(16):
                der.applyWeightsForDerivDev(R.LSFC, fields.data_ptr(), out.data_ptr(), ntracers=T)
            expect = out.cpu().numpy()
            fraction = (peak + (1 << 16)) / total
        srv = R.Server(c, fraction)
        rid = srv.submit(grid, R.heat_params(1.0, R.F64), u0, 1e-5, 5)
        assert srv.wait(rid) == 0
        outs.append(srv.result(rid).copy())
        if not apply_first:
            held, _, total = c.mem_info()
            peak = held + N * 8  # the request's own upload has gone again
        else:  # the buffers are made again
            for _ in range(17):
                der.applyWeightsForDerivDev(R.LSFC, fields.data_ptr(), out.data_ptr(), ntracers=T)
            assert np.array_equal(out.cpu().numpy(), expect)
            assert np.array_equal(der.getWeights(R.LSFC), W)
        srv.stop()
        grid.close()
        c.close()
    assert np.array_equal(*outs)
