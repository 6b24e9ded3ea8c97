"""rbffd_apply / rbffd_apply_dev in the caller's node order (one launch, or one
after a reordering launch on large grids): the oracle's sums bit for bit in
FP64, for tracer counts with and without 16-byte vectors, unaligned buffers,
a result written over its own field, and both arithmetics."""
import numpy as np
import pytest

import oracle as O
import rbffd_gpu_b200 as R
from tests.helpers import sphere_problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def problem(ctx, N, n, seed, lens=False):
    if N < 20000:
        xyz, st = sphere_problem(N, n, seed)
    else:
        xyz = R.fibonacci_nodes(N, seed)
        st = R.knn_stencils_gpu(ctx, xyz, n)
    rng = np.random.default_rng(seed)
    ln = rng.integers(1, n + 1, N).astype(np.int32) if lens else None
    grid = R.Grid(ctx, xyz, st, st_len=ln)
    der = R.RBFFD(R.LSFC, grid, 2)
    W = rng.standard_normal((N, n))
    if lens:
        W[np.arange(n)[None, :] >= ln[:, None]] = 0.0
    der.setWeights(R.LSFC, W)
    return grid, der, st, ln, W


@pytest.mark.parametrize("N,n,lens", [(1, 1, False), (31, 5, False), (700, 17, True), (4096, 31, False),
                                      (65536, 9, False), (65537, 9, False), (70001, 14, True)])
@pytest.mark.parametrize("T", [1, 2, 3, 4, 16])
def test_device_buffers(ctx, N, n, lens, T):
    grid, der, st, ln, W = problem(ctx, N, n, 5, lens)
    u = np.random.default_rng(8).standard_normal((N, T))
    ref = np.stack([O.apply(st, ln, W, np.ascontiguousarray(u[:, t])) for t in range(T)], axis=1)
    d = torch.from_numpy(u).cuda()
    for shift in (0, 1):  # an 8-byte shift: no 16-byte vectors
        buf = torch.zeros(N * T + 1, dtype=torch.float64, device="cuda")
        buf[shift:shift + N * T] = d.reshape(-1)
        out = torch.full((N * T + 1,), 9.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        der.applyWeightsForDerivDev(R.LSFC, buf.data_ptr() + 8 * shift, out.data_ptr() + 8 * shift, ntracers=T)
        got = out.cpu().numpy()
        assert np.array_equal(got[shift:shift + N * T].reshape(N, T), ref)
        assert got[0 if shift else N * T] == 9.0
    if T == 16:  # past the application from which the renumbered stencils are kept
        for _ in range(15):
            out.fill_(9.0)
            torch.cuda.synchronize()
            der.applyWeightsForDerivDev(R.LSFC, d.data_ptr(), out.data_ptr(), ntracers=T)
        assert np.array_equal(out.cpu().numpy()[:N * T].reshape(N, T), ref)
    # over its own field
    torch.cuda.synchronize()
    der.applyWeightsForDerivDev(R.LSFC, d.data_ptr(), d.data_ptr(), ntracers=T)
    assert np.array_equal(d.cpu().numpy(), ref)
    # FP32: each row's n products and sums rounded to 2^-24
    f = torch.from_numpy(u).cuda().float()
    out = torch.empty_like(f)
    torch.cuda.synchronize()
    der.applyWeightsForDerivDev(R.LSFC, f.data_ptr(), out.data_ptr(), dtype=R.F32, ntracers=T)
    bound = np.stack([O.apply(st, ln, np.abs(W), np.ascontiguousarray(np.abs(u[:, t]))) for t in range(T)], axis=1)
    assert (np.abs(out.cpu().numpy() - ref) <= (n + 3) * 2.0 ** -24 * bound + 1e-30).all()
    grid.close()


@pytest.mark.parametrize("N,n", [(700, 17), (70001, 14)])
def test_host_arrays(ctx, N, n):
    grid, der, st, ln, W = problem(ctx, N, n, 6, True)
    u = np.random.default_rng(8).standard_normal(N)
    ref = O.apply(st, ln, W, u)
    assert np.array_equal(der.applyWeightsForDeriv(R.LSFC, u), ref)
    part = der.applyWeightsForDeriv(R.LSFC, u, deriv=np.full(N, 3.0), start_indx=5, nb_stencils=N - 11)
    assert np.array_equal(part[5:N - 6], ref[5:N - 6]) and (part[:5] == 3.0).all() and (part[N - 6:] == 3.0).all()
    f32 = der.applyWeightsForDeriv(R.LSFC, u, dtype=R.F32)
    d = torch.from_numpy(u).cuda().float()
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    der.applyWeightsForDerivDev(R.LSFC, d.data_ptr(), out.data_ptr(), dtype=R.F32)
    assert np.array_equal(f32, out.cpu().numpy().astype(np.float64))
    ctx.setArithmetic(R.ARITH_UNFUSED)
    try:
        plain = der.applyWeightsForDeriv(R.LSFC, u)
    finally:
        ctx.setArithmetic(R.ARITH_FUSED)
    acc = np.zeros(N)
    for s in range(n):  # products and sums rounded one by one, in slot order
        acc = W[:, s] * u[st[:, s]] + acc
    assert np.array_equal(plain, acc)
    grid.close()
