"""BiCGSTAB over rows of many lengths: the operator passes stage a warp's rows in
shared memory 32 or 16 at a time, or walk them from global memory where they
do not fit or would meet in a bank. Every way gives the CPU restatement's
iterate, bit for bit, and lengths that meet cost no more than their neighbours."""
import time

import numpy as np
import pytest

import oracle as O
import rbf_b200 as R

pytestmark = pytest.mark.gpu


def _operator(kvec, seed):
    """Diagonally dominant rows of kvec entries, columns near the row's own."""
    n = kvec.size
    rng = np.random.default_rng(seed)
    ia = np.concatenate([[0], np.cumsum(kvec)]).astype(np.int32)
    row = np.repeat(np.arange(n), kvec)
    place = np.arange(ia[-1]) - ia[row]
    ja = ((row + place * 7) % n).astype(np.int32)
    L = -rng.random(ia[-1])
    L[ia[:-1]] = 0.0
    L[ia[:-1]] = 0.1 - 1.001 * np.add.reduceat(L, ia[:-1])
    return ia, ja, L


def _dev(T, a):
    return T.as_tensor(np.ascontiguousarray(a)).cuda()


def _check(ctx, T, kvec, k=None, stream=None):
    n = kvec.size
    ia, ja, L = _operator(kvec, 5)
    f = np.random.default_rng(6).random(n)
    bnd = np.arange(0, n, 41, dtype=np.int32)
    u = T.zeros(n, dtype=T.float64, device="cuda")
    dia = None if k else _dev(T, ia)
    dev = [_dev(T, a) for a in (L, ja, f, bnd)]
    T.cuda.synchronize()
    st, it, rel = ctx.solve_bicgstab(dev[0], dev[1], dev[2], u, k=k, ia=dia, bnd=dev[3], tol=0.0, maxit=5,
                                     stream=stream)
    T.cuda.synchronize()
    ost, ou, oit, orel = O.bicgstab(L, ja, f, np.zeros(n), k=k, ia=None if k else ia, bnd=bnd, tol=0.0, maxit=5,
                                    grid=O.solve_grid(n, T.cuda.get_device_properties(0).multi_processor_count))
    assert (it, rel) == (oit, orel)
    np.testing.assert_array_equal(u.cpu().numpy(), ou)


@pytest.mark.parametrize("k", [1, 7, 8, 16, 24, 31, 32, 33, 40, 48, 56, 63, 64, 65, 96])
def test_fixed_width(ctx, torch_cuda, k):
    _check(ctx, torch_cuda, np.full(1001, k), k=k)


@pytest.mark.parametrize("lengths", [(16, 16, 16, 21), (32,), (64, 64, 5), (1, 90, 90, 16), (60, 62, 66), (40, 40, 41)])
def test_ragged(ctx, torch_cuda, lengths):
    kvec = np.random.default_rng(7).choice(np.array(lengths), 1003)
    _check(ctx, torch_cuda, kvec)
    _check(ctx, torch_cuda, np.sort(kvec), stream=torch_cuda.cuda.Stream())


def _iteration_s(ctx, T, n, k):
    off = T.arange(k, device="cuda") * 3
    ja = ((T.arange(n, device="cuda")[:, None] + off) % n).to(T.int32).reshape(-1).contiguous()
    L = T.full((n, k), -1.0, dtype=T.float64, device="cuda")
    L[:, 0] = k + 0.5
    L, f = L.reshape(-1).contiguous(), T.rand(n, dtype=T.float64, device="cuda")
    u, s, ts = T.zeros_like(f), T.cuda.Stream(), []
    for _ in range(7):
        u.zero_()
        T.cuda.synchronize()
        t = time.perf_counter()
        _, it, _ = ctx.solve_bicgstab(L, ja, f, u, k=k, tol=0.0, maxit=40, stream=s)
        ts.append((time.perf_counter() - t) / max(it, 1))
    return min(ts)


@pytest.mark.parametrize("k", [32, 48, 64])
@pytest.mark.parametrize("n", [32000, 200000])
def test_rows_that_meet_in_a_bank_are_not_slower(ctx, torch_cuda, n, k):
    """A 16-fold conflict would cost 2.5 times the next shorter row."""
    times = sorted(_iteration_s(ctx, torch_cuda, n, k) / _iteration_s(ctx, torch_cuda, n, k - 1) for _ in range(3))
    assert times[1] < 1.6


def test_few_blocks_spread_over_the_chip(ctx, torch_cuda):
    """32,000 rows are one block for most SMs. Two blocks on an SM and none on
    another would take 0.45 of the time of 150,000 rows, one on each takes 0.3."""
    T = torch_cuda
    times = sorted(_iteration_s(ctx, T, 32000, 95) / _iteration_s(ctx, T, 150000, 95) for _ in range(3))
    assert times[1] < 0.38
