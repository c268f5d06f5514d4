"""The search of the nodes' own stencils on sets of uneven density and on small
sets, against the general search (rbfb_knn_query with the nodes as queries): the same lists, and no
longer than a stated multiple of its time, which lies between what the search by
cells once took on them and what it takes."""
import numpy as np
import pytest

import oracle as O
from rbf_b200 import nodesets as NS

pytestmark = pytest.mark.gpu


def _square(n):
    m = int(np.ceil(np.sqrt(n)))
    x, y, _ = NS.jittered_grid(m, 0.3, 3)
    return x[:n], y[:n]


def _uniform(n):
    r = np.random.default_rng(3)
    return r.random(n), r.random(n)


def _clusters(n):
    """Twenty tight clusters."""
    r = np.random.default_rng(3)
    c, i = r.random((20, 2)), r.integers(0, 20, n)
    return tuple((c[i] + 0.003 * r.standard_normal((n, 2))).T)


def _graded(ratio):
    """Density falling by `ratio` from the centre of a disk to its edge, as r^-1.5."""
    def nodes(n):
        r = np.random.default_rng(3)
        u, t, inner = r.random(n), 2 * np.pi * r.random(n), ratio ** (-1 / 1.5)
        rad = (u * (1 - inner ** 0.5) + inner ** 0.5) ** 2
        return rad * np.cos(t), rad * np.sin(t)
    return nodes


def _layer(n):
    """A boundary layer: thirtyfold density at one side."""
    r = np.random.default_rng(3)
    return r.random(n), (np.exp(r.random(n) * np.log(30.0)) - 1) / 29.0


# (nodes, n, k, multiple): taken once / now
CASES = [
    (_clusters, 3000, 100, 2.0),  # 6.1 / 1.1: all kept distances in one bucket
    (_square, 200, 128, 2.0),     # 14.5 / 1.1: a circle without a bound
    (_uniform, 200, 100, 2.0),    # 4.8 / 1.2
    (_graded(1000), 20000, 13, 0.4),  # 0.84 / 0.11: the general search over cells full of nodes
    (_graded(100), 1000, 13, 1.5),    # 3.5 / 0.68
    (_clusters, 3000, 28, 2.0),  # 3.8 / 1.2: a few cells hold every node
    (_clusters, 8000, 64, 1.5),  # 2.3 / 1.0
    (_layer, 8000, 21, 0.95),    # 1.3 / 0.65
]


def _us(T, f):
    a, b, ts = T.cuda.Event(enable_timing=True), T.cuda.Event(enable_timing=True), []
    for _ in range(7):
        a.record()
        for _ in range(5):
            f()
        b.record()
        T.cuda.synchronize()
        ts.append(200.0 * a.elapsed_time(b))
    return min(ts)


@pytest.mark.parametrize("nodes,n,k,multiple", CASES)
def test_search_against_the_general_one(ctx, torch_cuda, nodes, n, k, multiple):
    T = torch_cuda
    x, y = (T.as_tensor(np.ascontiguousarray(a)).cuda() for a in nodes(n))
    ja, want = (T.empty(n * k, dtype=T.int32, device="cuda") for _ in range(2))
    ctx.knn_stencils(x, y, k, ja)
    ctx.knn_query(x, y, x, y, k, want)
    assert ctx.knn_status() == 0
    assert bool((ja == want).all())
    ratio = sorted(_us(T, lambda: ctx.knn_stencils(x, y, k, ja)) /
                   _us(T, lambda: ctx.knn_query(x, y, x, y, k, want)) for _ in range(3))[1]
    assert ratio < multiple


@pytest.mark.parametrize("scale", [1e-170, 1e-155, 1e150])
def test_extreme_scales_complete(ctx, torch_cuda, scale):
    """Squared distances, and with them the first radius, that underflow to zero, are
    subnormal or near the largest double: the search still finishes, ties by index."""
    T = torch_cuda
    n, k = 700, 24
    x, y = (np.ascontiguousarray(a) * scale for a in _uniform(n))
    ja = T.empty(n * k, dtype=T.int32, device="cuda")
    ctx.knn_stencils(T.as_tensor(x).cuda(), T.as_tensor(y).cuda(), k, ja)
    assert ctx.knn_status() == 0
    np.testing.assert_array_equal(ja.cpu().numpy(), O.knn_brute(x, y, k))
