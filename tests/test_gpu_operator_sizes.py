"""Applying operators of short and of long rows: by tiles or by a thread a row,
the sums are the CPU restatement's bit for bit, and rows of a few entries take no longer
than the thread a row that they were."""
import numpy as np
import pytest

import oracle as O
import rbf_b200 as R

pytestmark = pytest.mark.gpu


def _operator(T, n, k, seed=3):
    off = T.arange(k, device="cuda") * 5
    ja = ((T.arange(n, device="cuda")[:, None] + off) % n).to(T.int32).reshape(-1).contiguous()
    g = T.Generator("cuda").manual_seed(seed)
    return ja, T.rand(n * k, dtype=T.float64, device="cuda", generator=g), T.rand(n, dtype=T.float64, device="cuda",
                                                                              generator=g)


@pytest.mark.parametrize("k", [1, 2, 3, 4, 7, 8, 9, 12, 59, 60, 61, 100, 124, 127, 128, 129])
@pytest.mark.parametrize("n", [15, 1000, 4133])
def test_either_way_gives_the_oracles_sums(torch_cuda, n, k):
    T = torch_cuda
    ja, W, u = _operator(T, n, k)
    out = T.empty(n, dtype=T.float64, device="cuda")
    R.spmv(n, k, ja, W, u, out)
    T.cuda.synchronize()
    want = O.spmv(ja.cpu().numpy(), W.cpu().numpy(), u.cpu().numpy(), k)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


def _us(T, f):
    a, b, ts = T.cuda.Event(enable_timing=True), T.cuda.Event(enable_timing=True), []
    for _ in range(9):
        a.record()
        for _ in range(10):
            f()
        b.record()
        T.cuda.synchronize()
        ts.append(100.0 * a.elapsed_time(b))
    return min(ts)


@pytest.mark.parametrize("k", [1, 2, 4])
def test_short_rows_of_a_large_operator(torch_cuda, k):
    """The same rows with arrays off a 16-byte boundary go by a thread a row."""
    T = torch_cuda
    n = 1000003
    ja, W, u = _operator(T, n, k)
    ja1, W1 = T.cat([ja[:1], ja])[1:], T.cat([W[:1], W])[1:]
    out = T.empty(n, dtype=T.float64, device="cuda")
    ratio = sorted(_us(T, lambda: R.spmv(n, k, ja, W, u, out)) / _us(T, lambda: R.spmv(n, k, ja1, W1, u, out))
                   for _ in range(3))[1]
    assert ratio < 1.4


def test_rows_of_twelve_on_both_sides_of_l2(torch_cuda):
    T = torch_cuda
    for n in (600000, 700001):
        ja, W, u = _operator(T, n, 12)
        ja1, W1 = T.cat([ja[:1], ja])[1:], T.cat([W[:1], W])[1:]
        out, want = (T.empty(n, dtype=T.float64, device="cuda") for _ in range(2))
        R.spmv(n, 12, ja, W, u, out)
        R.spmv(n, 12, ja1, W1, u, want)
        assert bool((out == want).all())
