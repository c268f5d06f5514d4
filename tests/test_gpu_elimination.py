"""The FP64 elimination on the tensor cores (asm_dmma.cuh) at the sizes where
its tiling can go wrong, and the stencils that leave its fast path, against
the oracle: the same operations in the same order, so every weight and status
must be equal, bit for bit."""
import numpy as np
import pytest

import oracle as O
import rbf_b200 as R
from rbf_b200 import nodesets as NS

pytestmark = pytest.mark.gpu


def _assemble(ctx, T, x, y, ja, k, P, ops=R.DEFAULT_OPS, scale=True, period=None, pts=None):
    n = x.size
    dev = [T.as_tensor(np.ascontiguousarray(a)).cuda() for a in (x, y, ja)]
    xc = yc = None
    nc = 0
    if pts is not None:
        xc, yc = (T.as_tensor(np.ascontiguousarray(a)).cuda() for a in pts)
        nc = len(pts[0])
    d = R.make_desc(P, 0, ops, R.FP64, scale, period=period, xc=xc, yc=yc, nc=nc)
    vals = [T.full((n * k,), 7.0, dtype=T.float64, device="cuda") for _ in range(R.num_rhs(ops, nc))]
    info = T.full((n,), -7, dtype=T.int32, device="cuda")
    ctx.assemble(d, dev[0], dev[1], k, dev[2], vals, info)
    T.cuda.synchronize()
    return np.stack([v.cpu().numpy() for v in vals]), info.cpu().numpy()


def _check(ctx, T, x, y, ja, k, P, ops=R.DEFAULT_OPS, scale=True, period=None, pts=None):
    W, info = _assemble(ctx, T, x, y, ja, k, P, ops, scale, period, pts)
    Wo, io = O.assemble(x, y, ja, k, P, ops=ops, scale=scale, period=period,
                        xc=None if pts is None else pts[0], yc=None if pts is None else pts[1])
    np.testing.assert_array_equal(info, io)
    np.testing.assert_array_equal(W, Wo)
    return io


# every system size of each class: all remainders of the panels, of the
# column tiles (n + 3 columns) and of the row tiles, and systems too small for
# their degree (singular)
@pytest.mark.parametrize("P,k0,k1", [(2, 3, 26), (3, 7, 38), (4, 12, 65)])
def test_every_size(ctx, torch_cuda, P, k0, k1):
    x, y, _ = NS.jittered_grid(12, 0.3, seed=5, periodic=True)
    for k in range(k0, k1 + 1):
        ja = O.knn_brute(x, y, k, period=(1.0, 1.0))
        _check(ctx, torch_cuda, x, y, ja, k, P, period=(1.0, 1.0))


@pytest.mark.parametrize("ops,pts", [
    (R.OP_DXX | R.OP_DYY | R.OP_DXY, None), (R.OP_LAPLACE, None), (R.OP_DY, None),
    (R.OP_INTERP | R.OP_LAPLACE, (np.array([0.0, 0.02]), np.array([0.0, -0.01]))),
    (R.OP_INTERP, (np.linspace(-0.03, 0.03, 8), np.linspace(0.02, -0.02, 8)))])
def test_right_hand_sides(ctx, torch_cuda, ops, pts):
    x, y, _ = NS.jittered_grid(13, 0.3, seed=6)
    for k, P in ((21, 2), (26, 2)) if pts is not None and len(pts[0]) > 3 else ((21, 2), (35, 3),
                                                                               (47, 4)):
        ja = O.knn_brute(x, y, k)
        _check(ctx, torch_cuda, x, y, ja, k, P, ops=ops, pts=pts)


# coordinates whose scale exponent, distances, phi or pivots leave the fast
# path's range (2^-900 .. 2^900): those stencils are solved again
@pytest.mark.parametrize("e,scale", [(-600, True), (600, True), (-150, False), (-320, False),
                                     (160, False), (-1010, True)])
@pytest.mark.parametrize("k,P", [(21, 2), (35, 3)])
def test_extreme_magnitudes(ctx, torch_cuda, e, scale, k, P):
    x, y, _ = NS.jittered_grid(9, 0.3, seed=7)
    ja = O.knn_brute(x, y, k)
    _check(ctx, torch_cuda, np.ldexp(x, e), np.ldexp(y, e), ja, k, P, scale=scale)


# coincident and collinear nodes among ordinary stencils: singular systems in
# the same launch, status and NaN weights in their rows alone
@pytest.mark.parametrize("k,P", [(21, 2), (23, 2), (28, 3), (35, 3), (36, 3), (64, 4)])
def test_singular_among_regular(ctx, torch_cuda, k, P):
    x, y, _ = NS.jittered_grid(20, 0.3, seed=8)
    x[40], y[40] = x[41], y[41]
    y[300:300 + k] = 3.0
    x[300:300 + k] = 3.0 + np.arange(k) / 64.0
    ja = O.knn_brute(x, y, k)
    info = _check(ctx, torch_cuda, x, y, ja, k, P)
    assert (info != 0).any() and (info == 0).any()


# the uneven launch: every size up to 96 unknowns, every degree and exponent
@pytest.mark.parametrize("phs", [0, 3, 5, 7, 9])
def test_uneven_every_size(ctx, torch_cuda, phs):
    T = torch_cuda
    x, y, _ = NS.jittered_grid(30, 0.3, seed=9)
    n = x.size
    rng = np.random.default_rng(10 + phs)
    deg = rng.integers(2 if phs == 0 else 1, 5, size=n).astype(np.int8)
    npol = (deg.astype(int) + 1) * (deg.astype(int) + 2) // 2
    kvec = 1 + np.arange(n) % (96 - npol)
    kmax = int(kvec.max())
    jaf = O.knn_brute(x, y, kmax).reshape(n, kmax)
    ia = np.zeros(n + 1, np.int32)
    ia[1:] = np.cumsum(kvec)
    ja = np.concatenate([jaf[s, :kvec[s]] for s in range(n)]).astype(np.int32)
    vals = [T.full((int(ia[-1]),), 7.0, dtype=T.float64, device="cuda") for _ in range(3)]
    info = T.full((n,), -7, dtype=T.int32, device="cuda")
    dv = [T.as_tensor(a).cuda() for a in (x, y, ia, ja, deg)]
    ctx.assemble_csr(R.make_desc(2, phs), dv[0], dv[1], dv[2], dv[3], vals, degree=dv[4], info=info)
    T.cuda.synchronize()
    Wo, io = O.assemble_csr(x, y, ia, ja, degree=deg, P=2, Q=phs)
    np.testing.assert_array_equal(info.cpu().numpy(), io)
    np.testing.assert_array_equal(np.stack([v.cpu().numpy() for v in vals]), Wo)
