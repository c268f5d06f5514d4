"""Applying an operator and solving with it at every row length and tile
remainder, against the oracle: the same sums in the same order, so results are
equal bit for bit."""
import numpy as np
import pytest

import oracle as O
import rbf_b200 as R

pytestmark = pytest.mark.gpu


def _operator(rng, n, k):
    """Random rows of k distinct columns, self first and dominant."""
    ja = np.empty((n, k), np.int32)
    ja[:, 0] = np.arange(n)
    step = np.sort(rng.choice(np.arange(1, n), size=k - 1, replace=False)) if k > 1 else []
    for j, d in enumerate(step):
        ja[:, j + 1] = (np.arange(n) + d) % n
    v = rng.uniform(-1.0, 1.0, (n, k))
    v[:, 0] = k + rng.uniform(0.0, 1.0, n)
    return ja.ravel(), v.ravel()


@pytest.mark.parametrize("k", list(range(1, 70)) + [96, 100, 126, 127, 128, 129, 144, 200])
def test_spmv_every_row_length(torch_cuda, k):
    T = torch_cuda
    rng = np.random.default_rng(k)
    for n in (max(k, 1), 257, 1000):
        if n < k:
            continue
        ja, v = _operator(rng, n, k)
        u = rng.standard_normal(n)
        bnd = np.unique(rng.integers(0, n, 5)).astype(np.int32)
        jd, vd, ud, bd = (T.as_tensor(a).cuda() for a in (ja, v, u, bnd))
        out = T.full((n + 8,), 7.0, dtype=T.float64, device="cuda")
        R.spmv(n, k, jd, vd, ud, out, bd)
        T.cuda.synchronize()
        got = out.cpu().numpy()
        assert (got[n:] == 7.0).all()
        np.testing.assert_array_equal(got[:n], O.spmv(ja, v, u, k, bnd))


# rows staged 32 and 16 at a time, and walked from global memory
@pytest.mark.parametrize("k", [8, 21, 33, 40, 64, 70])
@pytest.mark.parametrize("n", [200, 3000])
@pytest.mark.parametrize("ragged", [False, True])
def test_solve_row_lengths(ctx, torch_cuda, k, n, ragged):
    T = torch_cuda
    rng = np.random.default_rng(100 + k)
    ja, v = _operator(rng, n, k)
    ia = None
    if ragged:
        keep = np.arange(k)[None, :] < rng.integers(1, k + 1, n)[:, None]
        keep[: n // 8] = True
        ia = np.zeros(n + 1, np.int32)
        ia[1:] = np.cumsum(keep.sum(1))
        ja, v = ja[keep.ravel()], v[keep.ravel()]
    f = rng.standard_normal(n)
    bnd = np.arange(0, n, 37, dtype=np.int32)
    dv = [T.as_tensor(a).cuda() for a in (v, ja, f, bnd)]
    iad = None if ia is None else T.as_tensor(ia).cuda()
    u = T.zeros(n, dtype=T.float64, device="cuda")
    st, it, rel = ctx.solve_bicgstab(dv[0], dv[1], dv[2], u, k=None if ragged else k, ia=iad,
                                     bnd=dv[3], tol=1e-12, maxit=400)
    sms = T.cuda.get_device_properties(0).multi_processor_count
    ost, ou, oit, orel = O.bicgstab(v, ja, f, np.zeros(n), k=None if ragged else k, ia=ia, bnd=bnd,
                                    tol=1e-12, maxit=400, grid=O.solve_grid(n, sms))
    assert it == oit and rel == orel and (st == R.OK) == (ost == 0)
    np.testing.assert_array_equal(u.cpu().numpy(), ou)


# operators past L2: blocks of four warps
@pytest.mark.parametrize("n,k", [(700003, 17), (500001, 24), (330000, 35)])
def test_spmv_large(torch_cuda, n, k):
    T = torch_cuda
    rng = np.random.default_rng(k)
    ja = rng.integers(0, n, (n, k), dtype=np.int32).ravel()
    v, u = rng.standard_normal(n * k), rng.standard_normal(n)
    bnd = np.arange(0, n, 1000, dtype=np.int32)
    jd, vd, ud, bd = (T.as_tensor(a).cuda() for a in (ja, v, u, bnd))
    out = T.empty(n, dtype=T.float64, device="cuda")
    R.spmv(n, k, jd, vd, ud, out, bd)
    np.testing.assert_array_equal(out.cpu().numpy(), O.spmv(ja, v, u, k, bnd))


# the streaming step at every stencil size: a kernel each up to 32 entries, the
# general one past them; whole and ragged tiles; arrays that are not 16-byte
# aligned
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k", list(range(1, 41)) + [48, 63, 64])
def test_stream_collide_every_row_length(torch_cuda, dtype, k):
    T = torch_cuda
    rng = np.random.default_rng(k)
    for n, shift in ((64, 0), (301, 0), (302, 0), (302, 1)):
        ja = rng.integers(0, n, n * k, dtype=np.int32)
        W = rng.standard_normal(8 * n * k)
        W[rng.random(W.size) < 0.1] = -0.0
        f = rng.uniform(0.5, 1.5, 9 * n).astype(dtype)
        store = T.zeros(8 * n * k + shift, dtype=T.float64, device="cuda")
        Wd = store[shift:]
        Wd.copy_(T.as_tensor(W))
        jd, fd = T.as_tensor(ja).cuda(), T.as_tensor(f).cuda()
        out = T.full((9 * n,), 7.0, dtype=fd.dtype, device="cuda")
        m = [T.empty(n, dtype=fd.dtype, device="cuda") for _ in range(3)]
        R.lbm_stream_collide(k, jd, Wd, 1.2, fd, out, *m)
        want = O.lbm_stream_collide(k, ja, W, 1.2, f)
        for got, w in zip([out] + m, want):
            np.testing.assert_array_equal(got.cpu().numpy(), w)
