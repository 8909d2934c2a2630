"""Device memory that a batched Floyd-Warshall takes for itself."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def taken(gpu, dtype, mats, preds):
    """Bytes of device memory that a call on a new handle leaves allocated."""
    ctx = gpu.Context(0)
    try:
        ctx.floyd_batched(dtype, [torch.zeros((1, 1), dtype=mats[0].dtype, device="cuda")], None)  # modules loaded
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ctx.floyd_batched(dtype, mats, preds)
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()


@pytest.mark.parametrize("kind", ["f32_small", "i32_wide"])
def test_no_scratch_for_matrices_without_lookahead(gpu, kind):
    """Many matrices of one block, and int32 matrices outside the packed range,
    need descriptors (below 4 KB a matrix) and no scratch beside them; every
    matrix of the batch is closed."""
    if kind == "f32_small":
        count, n, dtype, inf, scale = 20000, 16, gpu.DTYPE_F32, 1e8, 1
    else:
        count, n, dtype, inf, scale = 3000, 65, gpu.DTYPE_I32, 1 << 30, 1 << 20
    rng = np.random.default_rng(n)
    a = np.where(rng.random((n, n)) < 2.0 / n, rng.integers(1, 9, (n, n)) * scale, inf)
    np.fill_diagonal(a, 0)
    tdt = torch.float32 if dtype == gpu.DTYPE_F32 else torch.int32
    one = torch.from_numpy(a).to("cuda", tdt)
    rows = torch.arange(n, dtype=torch.int32, device="cuda")[:, None].expand(n, n)
    d = one.expand(count, n, n).clone()
    p = torch.where(one < inf, rows, -1).expand(count, n, n).clone()
    torch.cuda.synchronize()
    assert taken(gpu, dtype, list(d.unbind(0)), list(p.unbind(0))) < count * 4096 + (8 << 20)
    w = torch.from_numpy(np.where(a < inf, a, np.inf)).cuda()
    for k in range(n):
        w = torch.minimum(w, w[:, k:k + 1] + w[k:k + 1])
    ref = torch.where(torch.isinf(w), float(inf), w).to(tdt)
    assert bool((d == ref).all()) and bool((p == p[0]).all())
