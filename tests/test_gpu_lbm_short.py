"""The time of a streaming step with stencils of few nodes (their results:
test_gpu_operator.py)."""
import pytest

import rbf_b200 as R

pytestmark = pytest.mark.gpu


def _inputs(T, n, k, dtype):
    g = T.Generator("cuda").manual_seed(9)
    off = T.arange(k, device="cuda") * 11
    ja = ((T.arange(n, device="cuda")[:, None] + off) % n).to(T.int32).reshape(-1)
    W = T.rand(8 * n * k, dtype=T.float64, device="cuda", generator=g) / k
    pdf = T.rand(9 * n, dtype=T.float64, device="cuda", generator=g).to(dtype) + 0.5
    return ja.contiguous(), W, pdf


def _us(T, f):
    a, b, ts = T.cuda.Event(enable_timing=True), T.cuda.Event(enable_timing=True), []
    for _ in range(9):
        a.record()
        for _ in range(5):
            f()
        b.record()
        T.cuda.synchronize()
        ts.append(200.0 * a.elapsed_time(b))
    return min(ts)


# a step of one entry against one of 5, each by its bytes: between what batches of
# eight cost (2.02, 2.84) and a plain loop (1.21, 1.72)
@pytest.mark.parametrize("dtype,k,limit", [("float64", 1, 1.6), ("float32", 1, 2.2)])
def test_a_step_costs_what_it_moves(torch_cuda, dtype, k, limit):
    T = torch_cuda
    n, size = 600000, 8 if dtype == "float64" else 4
    times = []
    for q in (k, 5):
        ja, W, pdf = _inputs(T, n, q, getattr(T, dtype))
        out, m = T.empty_like(pdf), [T.empty_like(pdf[:n]) for _ in range(3)]
        moved = n * (8 * 8 * q + 4 * q + 18 * size)
        us = sorted(_us(T, lambda: R.lbm_stream_collide(q, ja, W, 1.3, pdf, out, *m)) for _ in range(3))[1]
        times.append(us / moved)
    assert times[0] < limit * times[1]
