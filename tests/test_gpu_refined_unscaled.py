"""The refined form on systems that are not scaled and that end well before the
last block of their class (n <= 8 (NT - 1)): the convergence measure has to
see the unknowns alone. With FP32 factors a sweep reduces the error of these
systems by about cond * 2^-24 << 0.1, so no stencil may go to the FP64 kernel,
and 1e-11 is reached in two or three sweeps at degree 2 and 3, four at degree 4.
Weights: the tolerance of test_gpu_refined.py."""
import numpy as np
import pytest

import oracle as O
import rbf_b200 as R
from rbf_b200 import nodesets as NS

pytestmark = pytest.mark.gpu

SPACING = 10.0  # entries of phi up to about 1e8 at degree 3


@pytest.mark.parametrize("P,k", [(2, 12), (2, 15), (2, 18), (3, 15), (3, 22), (3, 28), (3, 30), (4, 19),
                                 (4, 25), (4, 34)])
def test_unscaled_short_systems(ctx, torch_cuda, P, k):
    T = torch_cuda
    m = 20
    x, y, _ = NS.jittered_grid(m, 0.3, seed=3, periodic=True)
    f = m * SPACING
    x, y, period = x * f, y * f, (f, f)
    ja = O.knn_brute(x, y, k, period=period)
    xd, yd, jd = (T.as_tensor(np.ascontiguousarray(a)).cuda() for a in (x, y, ja))
    W = [T.empty(x.size * k, dtype=T.float64, device="cuda") for _ in range(3)]
    d = R.make_desc(P, 0, R.DEFAULT_OPS, R.FP32_IR, False, period=period)
    st = ctx.assemble(d, xd, yd, k, jd, W, stats=True)
    T.cuda.synchronize()
    assert st["fallback"] == 0
    assert st["sweeps"] <= (3.0 if P < 4 else 5.0) * x.size
    Wo, _ = O.assemble(x, y, ja, k, P, scale=False, period=period)
    Wl, _ = O.assemble_ld(x, y, ja, k, P, scale=False, period=period)
    got = np.stack([w.cpu().numpy() for w in W])
    got, Wo, Wl = (np.asarray(a).reshape(3, -1, k) for a in (got, Wo, Wl))
    size = np.abs(Wl).max(axis=2)
    err, own = np.abs(got - Wl).max(axis=2), np.abs(Wo - Wl).max(axis=2)
    assert (err <= 1e-9 * size + 2.0 * own.max(axis=1, keepdims=True)).all()
