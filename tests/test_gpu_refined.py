"""The refined form (asm_refined.cuh: FP32 factors, FP64 residuals) at the
sizes where its tiles and blocks can go wrong, and the stencils that it leaves
to the FP64 kernel.

Tolerance: a sweep ends once the predicted error is below 1e-11 of the largest
unknown. The unknowns include the polynomial multipliers, which may exceed the
weights: a factor of 100 covers them. Where the systems are ill-conditioned the
FP64 solution itself is further off the long-double one; a stencil is held to
twice that distance (the FP64 kernel's, where the refinement stalled)."""
import numpy as np
import pytest

import oracle as O
import rbf_b200 as R
from rbf_b200 import nodesets as NS

pytestmark = pytest.mark.gpu


def _run(ctx, T, x, y, ja, k, P, ops=R.DEFAULT_OPS, scale=True, period=None, max_sweeps=0):
    n = x.size
    dev = [T.as_tensor(np.ascontiguousarray(a)).cuda() for a in (x, y, ja)]
    d = R.make_desc(P, 0, ops, R.FP32_IR, scale, max_sweeps=max_sweeps, period=period)
    vals = [T.full((n * k,), 7.0, dtype=T.float64, device="cuda") for _ in range(R.num_rhs(ops, 0))]
    info = T.full((n,), -7, dtype=T.int32, device="cuda")
    st = ctx.assemble(d, dev[0], dev[1], k, dev[2], vals, info, stats=True)
    T.cuda.synchronize()
    return np.stack([v.cpu().numpy() for v in vals]), info.cpu().numpy(), st


def _check(ctx, T, x, y, k, P, period=None, **kw):
    ja = O.knn_brute(x, y, k, period=period)
    W, info, st = _run(ctx, T, x, y, ja, k, P, period=period, **kw)
    Wo, io = O.assemble(x, y, ja, k, P, period=period, **kw)
    Wl, _ = O.assemble_ld(x, y, ja, k, P, period=period, **kw)
    np.testing.assert_array_equal(info, io)
    W, Wo, Wl = (np.asarray(a).reshape(len(a), -1, k) for a in (W, Wo, Wl))
    size = np.abs(Wl).max(axis=2)
    err, own = np.abs(W - Wl).max(axis=2), np.abs(Wo - Wl).max(axis=2)
    assert (err <= 1e-9 * size + 2.0 * own.max(axis=1, keepdims=True)).all()
    return st


# every remainder of the panels, the 8 x 8 tiles and the column vectors, on
# either side of each class and of 32 and 64 rows; 61 stencils leave the last
# CTA with idle warps
@pytest.mark.parametrize("P,ks", [
    (2, [9, 10, 11, 12, 17, 18, 19, 21, 25, 26]),
    (3, [15, 21, 22, 23, 24, 28, 30, 31, 33, 35, 36, 37, 38]),
    (4, [25, 32, 33, 34, 41, 48, 49, 50, 51, 57, 63, 64, 65])])
def test_sizes(ctx, torch_cuda, P, ks):
    x, y, _ = NS.jittered_grid(11, 0.3, seed=5, periodic=True)
    for k in ks:
        _check(ctx, torch_cuda, x, y, k, P, period=(1.0, 1.0))


@pytest.mark.parametrize("ops", [R.OP_LAPLACE, R.OP_DY, R.OP_DXX | R.OP_DXY,
                                 R.OP_DXX | R.OP_DYY | R.OP_DXY])
def test_right_hand_sides(ctx, torch_cuda, ops):
    x, y, _ = NS.jittered_grid(12, 0.3, seed=6)
    for k, P in ((21, 2), (35, 3)):
        _check(ctx, torch_cuda, x, y, k, P, ops=ops)


def test_stencils_left_to_fp64(ctx, torch_cuda):
    """Coincident nodes, systems outside the FP32 range and a sweep limit that
    is too low: the FP64 kernel's weights and status, bit for bit."""
    x, y, _ = NS.jittered_grid(12, 0.3, seed=7)
    k, P = 35, 3
    ja = O.knn_brute(x, y, k)
    for change in ("coincident", "tiny", "limit"):
        xs, ys, scale, sweeps, every = x.copy(), y.copy(), True, 0, True
        if change == "coincident":
            xs[ja[1]], ys[ja[1]], every = xs[ja[0]], ys[ja[0]], False
        elif change == "tiny":  # phi = r^5 far below 2^-126
            xs, ys, scale = x * 1e-12, y * 1e-12, False
        else:
            sweeps = 1
        W, info, st = _run(ctx, torch_cuda, xs, ys, ja, k, P, scale=scale, max_sweeps=sweeps)
        Wo, io = O.assemble(xs, ys, ja, k, P, scale=scale)
        np.testing.assert_array_equal(info, io)
        there = np.ones(x.size, bool) if every else (ja.reshape(-1, k) == ja[1]).any(1) & (
            ja.reshape(-1, k) == ja[0]).any(1)
        assert st["fallback"] >= there.sum() > 0
        got, want = (np.asarray(a).reshape(3, -1, k)[:, there] for a in (W, Wo))
        np.testing.assert_array_equal(got, want)
