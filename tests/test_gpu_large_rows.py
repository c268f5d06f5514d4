"""Fixed-width assembly of a batch with more than 2^31 stored entries: the
offsets of its last rows need 64 bits. The node set is one small periodic set
repeated, every row refers to the first copy, and so every copy's weights are
the small set's, bit for bit."""
import pytest

import rbf_b200 as R
from rbf_b200 import nodesets as NS

pytestmark = pytest.mark.gpu

M, K, P = 64, 26, 2
NEED = 40 << 30  # bytes on the device: 8.6 GB of ja, 17.2 GB of weights, and the comparison


@pytest.mark.parametrize("precision", [R.FP64, R.FP32_IR], ids=["fp64", "refined"])
def test_more_than_2_31_entries(ctx, torch_cuda, precision):
    T = torch_cuda
    T.cuda.empty_cache()
    if T.cuda.mem_get_info()[0] < NEED:
        pytest.skip("not enough device memory")
    x, y, _ = NS.jittered_grid(M, 0.3, seed=11, periodic=True)
    n0 = x.size
    copies = (1 << 31) // (n0 * K) + 4
    assert copies * n0 * K - (1 << 31) > 2 * n0 * K
    d = R.make_desc(P, 0, R.OP_LAPLACE, precision, True, period=(1.0, 1.0))
    x0, y0 = T.as_tensor(x).cuda(), T.as_tensor(y).cuda()
    ja0 = T.empty(n0 * K, dtype=T.int32, device="cuda")
    ctx.knn_stencils(x0, y0, K, ja0, period=(1.0, 1.0))
    want = T.empty(n0 * K, dtype=T.float64, device="cuda")
    ctx.assemble(d, x0, y0, K, ja0, [want])

    xs, ys, ja = x0.repeat(copies), y0.repeat(copies), ja0.repeat(copies)
    got = T.zeros(copies * n0 * K, dtype=T.float64, device="cuda")
    info = T.full((copies * n0,), -1, dtype=T.int32, device="cuda")
    ctx.assemble(d, xs, ys, K, ja, [got], info)
    T.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    rows = got.view(copies, n0 * K)
    for part in rows.split(4096):  # a bounded temporary
        assert bool((part == want).all())
