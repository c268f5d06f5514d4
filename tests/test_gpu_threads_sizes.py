"""Host threads whose calls need different amounts of shared memory from the
same kernel: every call succeeds and gives what it gives alone."""
import threading

import numpy as np
import pytest

import rbf_b200 as R
from rbf_b200 import nodesets as NS

pytestmark = pytest.mark.gpu

REPS = 5000


def _search(T, k):
    x, y, _ = NS.jittered_grid(24, 0.3, seed=31)
    xd, yd = T.as_tensor(x).cuda(), T.as_tensor(y).cuda()
    ja = T.empty(x.size * k, dtype=T.int32, device="cuda")
    ctx = R.Context(0)
    return lambda s: ctx.knn_stencils(xd, yd, k, ja, stream=s), ja


def _rows(T, k, n=512):
    rng = np.random.default_rng(k)
    ja = T.as_tensor(rng.integers(0, n, n * k).astype(np.int32)).cuda()
    return ja, rng


def _apply(T, k):
    ja, rng = _rows(T, k)
    n = ja.numel() // k
    W, u = T.as_tensor(rng.random(n * k)).cuda(), T.as_tensor(rng.random(n)).cuda()
    out = T.empty(n, dtype=T.float64, device="cuda")
    return lambda s: R.spmv(n, k, ja, W, u, out, stream=s), out


def _stream(T, k):
    ja, rng = _rows(T, k)
    n = ja.numel() // k
    W, pdf = T.as_tensor(rng.random(8 * n * k)).cuda(), T.as_tensor(rng.random(9 * n)).cuda()
    out = T.empty_like(pdf)
    return lambda s: R.lbm_stream_collide(k, ja, W, 1.1, pdf, out, stream=s), out


# each pair: two sizes of one kernel, far apart in shared memory
@pytest.mark.parametrize("make,sizes", [(_search, (80, 128)), (_apply, (64, 128)), (_apply, (63, 127)),
                                        (_stream, (34, 62))],
                         ids=["search", "apply-padded", "apply", "stream"])
def test_two_sizes_at_a_time(torch_cuda, make, sizes):
    T = torch_cuda
    calls, alone, errors = [], [], []
    for k in sizes:
        f, out = make(T, k)
        st = T.cuda.Stream()
        T.cuda.synchronize()
        f(st)
        st.synchronize()
        calls.append((f, out, st))
        alone.append(out.clone())
    start = threading.Barrier(2)

    def work(f, st):
        try:
            start.wait(timeout=60)
            for _ in range(REPS):
                f(st)
        except Exception as e:  # reported on the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(f, st)) for f, _, st in calls]
    for _, out, _ in calls:
        out.zero_()
    T.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert not any(t.is_alive() for t in threads), "a worker thread did not finish"
    T.cuda.synchronize()
    assert not errors, errors
    for (_, out, _), want in zip(calls, alone):
        assert bool((out == want).all())
