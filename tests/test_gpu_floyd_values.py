"""FP32 values outside the plain range: negative entries and -0.0 of small
matrices of a batched Floyd-Warshall, values above "unreached", graph weights of
-0.0."""
import numpy as np
import pytest
import torch

from fastapsp_gb300 import graphs

pytestmark = pytest.mark.gpu

UNREACHED = np.float32(1e8)


@pytest.fixture(scope="module")
def ctx(gpu):
    c = gpu.Context(0)
    yield c
    c.close()


def digraph(rng, n):
    """Whole-number weights, about two edges out of a vertex, zero diagonal, predecessors."""
    a = np.full((n, n), UNREACHED)
    edge = rng.random((n, n)) < 2.0 / n
    a[edge] = rng.integers(1, 9, edge.sum())
    np.fill_diagonal(a, 0)
    return a, edge & ~np.eye(n, dtype=bool)


def preds_of(a):
    n = a.shape[0]
    return np.where(a < UNREACHED, np.arange(n, dtype=np.int32)[:, None], -1).astype(np.int32)


def sequential(a, p):
    """Floyd-Warshall in ascending steps, strict improvements only."""
    d, p = a.copy(), p.copy()
    for k in range(a.shape[0]):
        via = d[:, k:k + 1] + d[k:k + 1]
        better = via < d
        d, p = np.where(better, via, d), np.where(better, np.broadcast_to(p[k], p.shape), p)
    return d, p


def run(ctx, mats, preds):
    ds = [torch.from_numpy(a).cuda() for a in mats]
    ps = [torch.from_numpy(p).cuda() for p in preds] if preds else None
    torch.cuda.synchronize()
    ctx.floyd_batched(0, ds, ps)
    torch.cuda.synchronize()
    return [d.cpu().numpy() for d in ds], [p.cpu().numpy() for p in ps] if preds else None


@pytest.mark.parametrize("kind", ["negative", "minus_zero"])
@pytest.mark.parametrize("sizes", [(1, 2, 40, 63, 64), (64, 200, 33, 65)])
def test_negative_entries_of_small_matrices(ctx, kind, sizes):
    """Matrices of at most 64 vertices close with negative entries (without
    negative cycles) and -0.0, alone and in a batch with larger ones."""
    rng = np.random.default_rng(sum(sizes))
    mats = []
    for n in sizes:
        a, edge = digraph(rng, n)
        if n <= 64 and kind == "negative":  # potentials: every cycle keeps its length
            h = rng.integers(0, 6, n).astype(np.float32)
            a[edge] += (h[:, None] - h[None, :])[edge]
        elif n <= 64:
            a[edge & (rng.random((n, n)) < 0.3)] = -0.0
        mats.append(a)
    preds = [preds_of(a) for a in mats]
    got, gotp = run(ctx, mats, preds)
    plain, _ = run(ctx, mats, None)
    for a, p, d, q, e in zip(mats, preds, got, gotp, plain):
        ref, refp = sequential(a, p)
        reached = ref < UNREACHED / 2
        assert np.array_equal(d[reached], ref[reached])
        if a.shape[0] <= 64:  # (blocks take equal paths in another order)
            assert np.array_equal(q[reached], refp[reached])
        assert (d[~reached] > UNREACHED / 2).all() and (q[~reached] == -1).all()
        assert np.array_equal(e, d)


@pytest.mark.parametrize("absent", [np.inf, 3e8, np.nan])
@pytest.mark.parametrize("n", [65, 128, 130, 300])
def test_values_above_unreached(ctx, n, absent):
    """Matrices of more than one block with missing edges at infinity (or any value
    above "unreached") close as with 1e8 there, with predecessors and without."""
    rng = np.random.default_rng(n)
    a, _ = digraph(rng, n)
    preds = [preds_of(a)] * 3
    above, some = a.copy(), a.copy()
    above[a >= UNREACHED] = absent
    some[(a >= UNREACHED) & (rng.random((n, n)) < 0.5)] = absent
    for p in (preds, None):
        got, gotp = run(ctx, [a, above, some], p)
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
        if p:
            assert np.array_equal(gotp[0], gotp[1]) and np.array_equal(gotp[0], gotp[2])


@pytest.mark.parametrize("n, parts", [(50, 2), (400, 3)])
def test_graph_weights_of_minus_zero(gpu, n, parts):
    """Weights of -0.0 count as 0: the same rows as with +0.0."""
    g = graphs.small_random_graph(n, 4 * n, True, True, seed=n)
    gid, _ = gpu.partition(g.row_offset, g.col_val, parts)
    w = g.weight.copy()
    w[::5] = -0.0
    outs = []
    for weight in (w, np.abs(w)):
        with gpu.Engine(n, g.row_offset, g.col_val, weight, parts, graph_id=gid, dtype=gpu.DTYPE_F32) as eng:
            d, p = np.empty((n, n), np.float32), np.empty((n, n), np.int32)
            eng.solve(d, p)
            outs.append((d, p))
    assert np.array_equal(outs[0][0].view(np.uint32), outs[1][0].view(np.uint32))
    assert np.array_equal(outs[0][1], outs[1][1])
