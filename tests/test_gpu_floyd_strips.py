"""Strips of 4 to 8 column tiles of the Floyd-Warshall remaining tiles (fw_rest.cu)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    c = gpu.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("size, count", [(640, 40), (700, 32), (770, 48), (900, 24), (1090, 24)])
def test_evened_strips_agree_with_one_tile_strips(ctx, f32, size, count):
    """Batches whose strips are 5 and 4, 5, 6, 7, and 8 and 6 tiles long on 152 SMs
    (launches of two to eight strips an SM): every copy of a matrix comes out as it
    does alone (strips of one or two tiles), with the distances of naive
    Floyd-Warshall."""
    rng = np.random.default_rng(size)
    inf = np.float32(1e8) if f32 else np.int32(1 << 30)
    a = np.full((size, size), inf)
    edge = rng.random((size, size)) < 4.0 / size
    a[edge] = rng.uniform(0.5, 10, edge.sum()).astype(np.float32) if f32 else rng.integers(1, 50, edge.sum())
    np.fill_diagonal(a, 0)
    p = np.where(a < inf, np.arange(size, dtype=np.int32)[:, None], -1).astype(np.int32)
    outs = []
    for many in (1, count):
        ds = torch.from_numpy(a).cuda().expand(many, size, size).clone()
        ps = torch.from_numpy(p).cuda().expand(many, size, size).clone()
        torch.cuda.synchronize()
        ctx.floyd_batched(0 if f32 else 1, list(ds.unbind(0)), list(ps.unbind(0)))
        torch.cuda.synchronize()
        outs.append((ds, ps))
    assert bool((outs[1][0] == outs[0][0]).all()) and bool((outs[1][1] == outs[0][1]).all())
    w = torch.from_numpy(np.where(a < inf, a, np.inf).astype(np.float64)).cuda()
    for k in range(size):
        w = torch.minimum(w, w[:, k:k + 1] + w[k:k + 1, :])
    w = torch.where(torch.isinf(w), float(inf), w)
    # FP32: at most size - 1 sums, each rounded once (relative 2^-24)
    tol = size * 2.0 ** -24 * w if f32 else torch.zeros_like(w)
    assert bool(((outs[0][0][0].double() - w).abs() <= tol).all())
