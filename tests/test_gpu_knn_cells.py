"""The cell-by-cell stencil search at the shapes where its blocks, lists and
fall-backs can go wrong, against the oracle's brute force: neighbour lists are
equal, ties by index."""
import numpy as np
import pytest

import oracle as O
import rbf_b200 as R
from rbf_b200 import nodesets as NS

pytestmark = pytest.mark.gpu


def _fold(v, L):
    """The search's fold into [0, L) (src/rbf_spatial.h:39-48), which the
    brute force expects done."""
    v = v - L * np.floor(v / L)
    v = np.where(v >= L, v - L, v)
    return np.where(v < 0, v + L, v)


def _check(ctx, T, x, y, k, period=None):
    n = x.size
    ja = T.full((n * k + 64,), -5, dtype=T.int32, device="cuda")
    xd, yd = (T.as_tensor(np.ascontiguousarray(a)).cuda() for a in (x, y))
    ctx.knn_stencils(xd, yd, k, ja, period=period)
    assert ctx.knn_status() == 0
    got = ja.cpu().numpy()
    assert (got[n * k:] == -5).all()  # nothing past the rows
    if period is not None:
        x, y = _fold(x, period[0]), _fold(y, period[1])
    np.testing.assert_array_equal(got[:n * k], O.knn_brute(x, y, k, period=period))


# every list length class: one, two, three, five and ten entries a lane, up to
# the largest k, with n = k and few cells
@pytest.mark.parametrize("k", [1, 2, 3, 8, 14, 15, 21, 31, 32, 33, 42, 43, 64, 71, 72, 100, 127, 128])
@pytest.mark.parametrize("periodic", [False, True])
def test_every_list_length(ctx, torch_cuda, k, periodic):
    for n in (k, k + 1, 300, 2500):
        if n < k:
            continue
        rng = np.random.default_rng(k + n)
        x, y = rng.uniform(0, 1, n), rng.uniform(0, 1, n)
        _check(ctx, torch_cuda, x, y, k, (1.0, 1.0) if periodic else None)


def _clusters(rng, n):
    c = rng.uniform(0, 1, (6, 2))
    w = 10.0 ** rng.uniform(-6, -1, 6)
    i = rng.integers(0, 6, n)
    p = c[i] + rng.normal(0, 1, (n, 2)) * w[i, None]
    return p[:, 0], p[:, 1]


def _coincident(rng, n):
    x, y = rng.uniform(0, 1, n), rng.uniform(0, 1, n)
    x[: n // 3], y[: n // 3] = 0.25, 0.75  # more than any list holds
    return x, y


def _line(rng, n):
    return rng.uniform(0, 1e-3, n), np.full(n, 2.0)


def _channel(rng, n):
    return rng.uniform(0, 40.0, n), rng.uniform(0, 0.5, n)


def _lattice(rng, n):
    m = int(np.sqrt(n))
    g = np.arange(m) / 8.0
    return tuple(a.ravel() for a in np.meshgrid(g, g))


def _extremes(rng, n):
    return rng.uniform(0, 1e-140, n), rng.uniform(0, 1e-140, n)


@pytest.mark.parametrize("make", [_clusters, _coincident, _line, _channel, _lattice, _extremes])
@pytest.mark.parametrize("k", [9, 35, 64])
def test_node_layouts(ctx, torch_cuda, make, k):
    x, y = make(np.random.default_rng(3 * k), 1600)
    _check(ctx, torch_cuda, x, y, k)


# boxes of few cells (the block covers a whole axis), long boxes, nodes outside
# [0, L) that are folded in
@pytest.mark.parametrize("L", [(1.0, 1.0), (8.0, 0.5), (0.3, 12.0)])
@pytest.mark.parametrize("n,k", [(40, 21), (130, 35), (900, 12), (1500, 64)])
def test_periodic_boxes(ctx, torch_cuda, L, n, k):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-L[0], 2 * L[0], n), rng.uniform(0, L[1], n)
    _check(ctx, torch_cuda, x, y, k, L)


# variable density: one ring, two and three rings, boundaries
@pytest.mark.parametrize("k", [12, 21, 35, 64])
def test_variable_density(ctx, torch_cuda, k):
    x, y, _ = NS.gaussian_bump(4000, seed=k)
    _check(ctx, torch_cuda, x, y, k)
    x, y, _ = NS.unit_disk(4000, nb=200, seed=k)
    _check(ctx, torch_cuda, x, y, k)


# the largest set that one block bins, and the smallest that the grid does
@pytest.mark.parametrize("n", [8192, 8193])
@pytest.mark.parametrize("make", [_clusters, _coincident, _line, _channel, _lattice])
def test_either_side_of_the_one_block_binning(ctx, torch_cuda, make, n):
    x, y = make(np.random.default_rng(n), n)
    for k, period in ((21, None), (35, (2.0, 3.0))):
        _check(ctx, torch_cuda, x, y, k, period)


# cells shared by up to eight warps, and by none; many nodes left over (a density
# that varies a hundredfold)
@pytest.mark.parametrize("n,k", [(70, 9), (400, 61), (3000, 35), (9000, 61), (20000, 21)])
def test_shared_cells_and_leftovers(ctx, torch_cuda, n, k):
    rng = np.random.default_rng(n + k)
    r, t = rng.uniform(0, 1, n) ** 2, rng.uniform(0, 2 * np.pi, n)
    for period in (None, (2.0, 2.0)):
        _check(ctx, torch_cuda, r * np.cos(t), r * np.sin(t), k, period)
