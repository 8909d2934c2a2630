"""Parity of the standalone sm_103a kernels against the CPU oracle, called
through the C ABI on device memory."""
import numpy as np
import pytest
import torch
from helpers import INF_I32, MAXV, check_pred_tight

from fastapsp_gb300 import graphs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    c = gpu.Context(0)
    yield c
    c.close()


def rand_dist(rng, shape, inf_frac, f32):
    if f32:
        a = rng.uniform(0.1, 50.0, size=shape).astype(np.float32)
        a[rng.random(shape) < inf_frac] = MAXV
    else:
        a = rng.integers(0, 1000, size=shape).astype(np.int32)
        a[rng.random(shape) < inf_frac] = INF_I32
    return a


def as_oracle(a):
    if a.dtype == np.int32:
        o = a.astype(np.float32)
        o[a >= INF_I32] = MAXV
        return o
    return a


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (31, 33, 7), (64, 64, 64), (65, 129, 33), (200, 300, 130),
                                   (130, 70, 0), (5, 1000, 257), (300, 2100, 29), (129, 2053, 48),
                                   (257, 4100, 49), (150, 700, 100), (70, 300, 101), (200, 2200, 32),
                                   (131, 1100, 33)])
def test_minplus_matches_oracle(ctx, oracle_lib, f32, M, N, K):
    rng = np.random.default_rng(M * 1000 + N * 10 + K)
    A = rand_dist(rng, (M, K), 0.2, f32)
    B = rand_dist(rng, (K, N), 0.2, f32)
    # ties: force duplicate minima so the first-k rule matters, within a group
    # of four steps (k = 0, 1) and across groups (k = 2, 6)
    if K > 3:
        B[1] = B[0]
        A[:, 1] = A[:, 0]
    if K > 6:
        B[6] = B[2]
        A[:, 6] = A[:, 2]
    Bp = rng.integers(0, 10**6, size=(K, N)).astype(np.int32)
    ref_c, ref_p = oracle_lib.min_plus(as_oracle(A), as_oracle(B), Bp)
    dt = torch.float32 if f32 else torch.int32
    dA = torch.from_numpy(A).cuda()
    dB = torch.from_numpy(B).cuda()
    dBp = torch.from_numpy(Bp).cuda()
    dC = torch.full((M, N), 7, dtype=dt, device="cuda")
    dCp = torch.full((M, N), 7, dtype=torch.int32, device="cuda")
    ctx.minplus(0 if f32 else 1, dA, dB, dC, dBp, dCp, M=M, N=N, K=K,
                lda=max(K, 1), ldb=N, ldc=N)
    torch.cuda.synchronize()
    c = dC.cpu().numpy()
    assert np.array_equal(as_oracle(c).view(np.int32), ref_c.view(np.int32))
    assert np.array_equal(dCp.cpu().numpy(), ref_p)


def make_dense(rng, n, density, f32):
    W = rand_dist(rng, (n, n), 1.0 - density, f32)
    if f32:
        W = np.where(W < MAXV, W, MAXV).astype(np.float32)
    np.fill_diagonal(W, 0)
    P = np.where(as_oracle(W) < MAXV, np.arange(n)[:, None], -1).astype(np.int32)
    return W, P


@pytest.mark.parametrize("f32", [False, True])
def test_floyd_batched_matches_oracle(ctx, oracle_lib, f32):
    rng = np.random.default_rng(7 + f32)
    # (sizes that are multiples of 4 have 16-byte rows: their remaining tiles
    # are staged by bulk tensor copies, boxes past the edge included)
    sizes = [1, 5, 63, 64, 65, 130, 132, 200, 257, 260]
    mats, preds, dev_d, dev_p = [], [], [], []
    for n in sizes:
        W, P = make_dense(rng, n, 0.08, f32)
        mats.append(W)
        preds.append(P)
        dev_d.append(torch.from_numpy(W).cuda())
        dev_p.append(torch.from_numpy(P).cuda())
    ctx.floyd_batched(0 if f32 else 1, dev_d, dev_p)
    torch.cuda.synchronize()
    for W, P, dd, dp in zip(mats, preds, dev_d, dev_p):
        n = W.shape[0]
        ref_d, _ = oracle_lib.floyd_path(as_oracle(W), P)
        got = as_oracle(dd.cpu().numpy())
        gp = dp.cpu().numpy()
        if f32:
            fin = ref_d < MAXV
            assert np.array_equal(fin, got < MAXV)
            assert np.allclose(got[fin], ref_d[fin], rtol=1e-6, atol=0)
        else:
            assert np.array_equal(got, ref_d)
        # predecessors: tight edges of the input matrix
        Wf = as_oracle(W).astype(np.float64)
        Wf[Wf >= MAXV] = np.inf
        np.fill_diagonal(Wf, np.inf)
        ro = np.zeros(n + 1, np.int64)
        rows, cols = np.nonzero(np.isfinite(Wf))
        np.add.at(ro, rows + 1, 1)
        ro = np.cumsum(ro)
        check_pred_tight(got, gp, np.arange(n), n, ro, cols, Wf[rows, cols],
                         rtol=1e-6 if f32 else 0.0)


@pytest.mark.parametrize("kind", ["grid", "knn_int", "road_f32", "rand_dir_int"])
def test_sssp_matches_dijkstra_bit_for_bit(gpu, oracle_lib, kind):
    if kind == "grid":
        g, dtype = graphs.grid_graph(40, 40, seed=1), gpu.DTYPE_I32
    elif kind == "knn_int":
        g, dtype = graphs.geometric_knn(3000, seed=2), gpu.DTYPE_I32
    elif kind == "road_f32":
        g, dtype = graphs.road_like(5000, seed=3), gpu.DTYPE_F32
    else:
        g, dtype = graphs.small_random_graph(500, 1500, True, True, seed=4), gpu.DTYPE_I32
    rng = np.random.default_rng(0)
    src = rng.choice(g.n, size=min(70, g.n), replace=False).astype(np.int32)
    with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, 2, dtype=dtype) as eng:
        dt = torch.int32 if dtype == gpu.DTYPE_I32 else torch.float32
        d = torch.empty((len(src), g.n), dtype=dt, device="cuda")
        p = torch.empty((len(src), g.n), dtype=torch.int32, device="cuda")
        eng.sssp(src, d, p)
        torch.cuda.synchronize()
        d = as_oracle(d.cpu().numpy())
        p = p.cpu().numpy()
    for i, s in enumerate(src):
        rd, rp = oracle_lib.dijkstra_path(int(s), g.row_offset, g.col_val, g.weight)
        assert np.array_equal(d[i].view(np.int32), rd.view(np.int32)), f"row {i}"
        assert np.array_equal(p[i], rp), f"pred row {i}"


@pytest.mark.parametrize("kind", ["grid", "road_f32"])
def test_sssp_result_independent_of_near_far_step(gpu, oracle_lib, kind):
    """The near-far step and the batch width only order the work: any of
    them gives the reference Dijkstra's distances and predecessors."""
    if kind == "grid":
        g, dtype = graphs.grid_graph(30, 30, seed=2), gpu.DTYPE_I32
    else:
        g, dtype = graphs.road_like(3000, seed=5), gpu.DTYPE_F32
    src = np.random.default_rng(3).choice(g.n, size=40, replace=False).astype(np.int32)
    dt = torch.int32 if dtype == gpu.DTYPE_I32 else torch.float32
    outs = []
    with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, 2, dtype=dtype) as eng:
        lo = 1e-3 if dtype == gpu.DTYPE_F32 else 1
        for delta, lanes in ((lo, 0), (0.0, 0), (1e9, 0), (0.0, 8), (0.0, 16), (0.0, 32)):
            eng.set_option(gpu._lib.OPT_SSSP_DELTA, delta)
            eng.set_option(gpu._lib.OPT_SSSP_LANES, lanes)
            d = torch.empty((len(src), g.n), dtype=dt, device="cuda")
            p = torch.empty((len(src), g.n), dtype=torch.int32, device="cuda")
            eng.sssp(src, d, p)
            torch.cuda.synchronize()
            outs.append((d.cpu().numpy(), p.cpu().numpy()))
    for d, p in outs[1:]:
        assert np.array_equal(d, outs[0][0]) and np.array_equal(p, outs[0][1])
    for i, s in enumerate(src):
        rd, rp = oracle_lib.dijkstra_path(int(s), g.row_offset, g.col_val, g.weight)
        assert np.array_equal(as_oracle(outs[0][0][i]).view(np.int32), rd.view(np.int32))
        assert np.array_equal(outs[0][1][i], rp)


def test_sssp_large_graph_bitmaps_in_global_memory(gpu, oracle_lib):
    """n = 450,000: the frontier bitmaps (3 x n bits) exceed the shared-memory
    budget and live in device memory; results stay bit-exact."""
    g = graphs.road_like(450_000, seed=21)
    n = g.n
    gid = np.where(np.arange(n) < n // 2, 1, 2).astype(np.int32)
    src = np.random.default_rng(9).choice(n, size=24, replace=False).astype(np.int32)
    with gpu.Engine(n, g.row_offset, g.col_val, g.weight, 2, graph_id=gid, dtype=gpu.DTYPE_F32) as eng:
        d = torch.empty((len(src), n), dtype=torch.float32, device="cuda")
        p = torch.empty((len(src), n), dtype=torch.int32, device="cuda")
        eng.sssp(src, d, p)
        torch.cuda.synchronize()
        d = d.cpu().numpy()
        p = p.cpu().numpy()
    for i in (0, 7, 23):
        rd, rp = oracle_lib.dijkstra_path(int(src[i]), g.row_offset, g.col_val, g.weight)
        assert np.array_equal(d[i].view(np.int32), rd.view(np.int32)), f"row {i}"
        assert np.array_equal(p[i], rp), f"pred row {i}"


@pytest.mark.parametrize("lanes", [0, 32])
def test_sssp_fp64_option_rounds_once(gpu, oracle_lib, lanes):
    """With FP64 search the FP32 output is the FP64 distance rounded once
    (16-source batches by default, 32-source batches forced)."""
    g = graphs.road_like(4000, seed=8)
    src = np.random.default_rng(2).choice(g.n, size=33, replace=False).astype(np.int32)
    with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, 2, dtype=gpu.DTYPE_F32) as eng:
        eng.set_option(gpu._lib.OPT_SSSP_FP64, 1)
        eng.set_option(gpu._lib.OPT_SSSP_LANES, lanes)
        d = torch.empty((len(src), g.n), dtype=torch.float32, device="cuda")
        p = torch.empty((len(src), g.n), dtype=torch.int32, device="cuda")
        eng.sssp(src, d, p)
        torch.cuda.synchronize()
        d = d.cpu().numpy()
        p = p.cpu().numpy()
    for i, s in enumerate(src):
        d64 = oracle_lib.dijkstra_f64(int(s), g.row_offset, g.col_val, g.weight)
        f = d64 < 1e299
        assert np.array_equal(f, d[i] < 1e8)
        assert np.array_equal(d[i][f], d64[f].astype(np.float32))  # round-to-nearest of FP64
    n = g.n
    check_pred_tight(d.astype(np.float64), p, src, n, g.row_offset, g.col_val, g.weight, rtol=1e-6)


@pytest.mark.parametrize("lanes", [0, 32])
def test_engine_fp64_sssp_option_meets_1e6_on_road_graph(gpu, oracle_lib, lanes):
    g = graphs.road_like(6000, seed=12)
    K = 8
    with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, K, dtype=gpu.DTYPE_F32) as eng:
        eng.set_option(gpu._lib.OPT_SSSP_FP64, 1)
        eng.set_option(gpu._lib.OPT_SSSP_LANES, lanes)
        n = g.n
        d = torch.empty((n, n), dtype=torch.float32, device="cuda")
        p = torch.empty((n, n), dtype=torch.int32, device="cuda")
        eng.solve(d, p, gpu.MODE_BATCHED)
        torch.cuda.synchronize()
        mapping = eng.mapping()
        rows = np.arange(0, n, 97)
        dd = d[torch.from_numpy(rows).cuda()].cpu().numpy()
    worst = 0.0
    for i, r in enumerate(rows):
        d64 = oracle_lib.dijkstra_f64(int(mapping[r]), g.row_offset, g.col_val, g.weight)
        f = d64 < 1e299
        assert np.array_equal(f, dd[i] < 1e8)
        worst = max(worst, float(np.max(np.abs(dd[i][f] - d64[f]) / np.maximum(d64[f], 1e-30))))
    assert worst <= 1e-6, worst


def test_speed_options_reject_unsupported_widths(gpu):
    """Batch and tile widths are limited to the kernels that exist; a rejected
    value leaves the option as it was."""
    g = graphs.grid_graph(16, 16, seed=4)
    with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, 2, dtype=gpu.DTYPE_I32) as eng:
        for opt, bad, good in ((gpu._lib.OPT_SSSP_LANES, 12, 8), (gpu._lib.OPT_TILE_COLS, 48, 128)):
            eng.set_option(opt, good)
            with pytest.raises(gpu._lib.FapError):
                eng.set_option(opt, bad)
            assert eng.get_option(opt) == good


def test_addmin_peak_probe_modes(ctx):
    """The register-only add-min probe (the roofline denominator) runs every
    form and rejects unknown ones; the DPX form outruns the forms that keep
    an index beside each value."""
    rates = {m: ctx.addmin_peak(m) for m in range(13)}
    assert all(r > 1e11 for r in rates.values()), rates
    assert rates[0] > rates[3] and rates[12] > rates[3]
    from fastapsp_gb300._lib import FapError
    with pytest.raises(FapError):
        ctx.addmin_peak(13)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("size", [129, 513, 530])
def test_floyd_strip_lengths_agree(ctx, oracle_lib, f32, size):
    """A launch's strips are 1, 2, 4 or 8 column tiles long, by how many
    matrices it holds; every copy of a matrix in a batch of any size comes
    out as the same bits, and as the distances of naive Floyd-Warshall."""
    rng = np.random.default_rng(size)
    inf = np.float32(1e8) if f32 else np.int32(1 << 30)
    a = np.full((size, size), inf)
    edge = rng.random((size, size)) < 0.02
    a[edge] = rng.uniform(0.5, 10, edge.sum()).astype(np.float32) if f32 else rng.integers(1, 50, edge.sum())
    np.fill_diagonal(a, 0)
    p = np.where(a < inf, np.arange(size, dtype=np.int32)[:, None], -1).astype(np.int32)
    first = None
    for count in (1, 24, 48, 90):
        ds = [torch.from_numpy(a).cuda() for _ in range(count)]
        ps = [torch.from_numpy(p).cuda() for _ in range(count)]
        ctx.floyd_batched(0 if f32 else 1, ds, ps)
        torch.cuda.synchronize()
        first = first or (ds[0], ps[0])
        for d, q in zip(ds, ps):
            assert torch.equal(d, first[0]) and torch.equal(q, first[1])
    for ld in (size + 1, (size + 7) // 4 * 4):  # rows past the matrix, aligned or not
        d, q = torch.zeros((size, ld), dtype=first[0].dtype, device="cuda"), torch.zeros((size, ld), dtype=torch.int32,
                                                                                          device="cuda")
        d[:, :size], q[:, :size] = torch.from_numpy(a).cuda(), torch.from_numpy(p).cuda()
        torch.cuda.synchronize()
        ctx.floyd_batched(0 if f32 else 1, [d[:, :size]], [q[:, :size]])
        torch.cuda.synchronize()
        assert torch.equal(d[:, :size], first[0]) and torch.equal(q[:, :size], first[1])
        assert not d[:, size:].any() and not q[:, size:].any()
    w = torch.from_numpy(np.where(a < inf, a, np.inf).astype(np.float64)).cuda()
    for k in range(size):
        w = torch.minimum(w, w[:, k:k + 1] + w[k:k + 1, :])
    w = torch.where(torch.isinf(w), float(inf), w)
    # FP32: at most size - 1 sums, each rounded once (relative 2^-24)
    tol = size * 2.0 ** -24 * w if f32 else torch.zeros_like(w)
    assert bool(((first[0].double() - w).abs() <= tol).all())


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("n,sources", [(33, 1), (1025, 33), (4097, 152), (4097, 153), (60000, 5)])
def test_sssp_one_cta_per_source_matches_batches(gpu, f32, n, sources):
    """Few sources (distances in shared memory, or past its size in the rows)
    and more than one per SM give the batched search's rows bit for bit, on
    graphs with unreached vertices, parallel edges, self loops, degrees past
    one lane group's four edges and frontiers past the shared-memory list; a
    vertex of more than 64 edges keeps the batched search."""
    rng = np.random.default_rng(n + sources)
    hubs = [graphs.small_random_graph(n, 3 * n, True, True, seed=n, integer=not f32)]
    star = np.r_[np.zeros(min(n - 1, 200), np.int64), rng.integers(0, n, 2 * n)]
    ends = np.r_[1 + np.arange(min(n - 1, 200)), rng.integers(0, n, 2 * n)]
    hubs.append(graphs.csr_from_lines(n, star, ends, rng.integers(1, 9, star.shape[0]).astype(np.float32), True, True))
    for g in hubs:
        src = rng.permutation(n)[:sources].astype(np.int32)
        with gpu.Engine(n, g.row_offset, g.col_val, g.weight, 1, graph_id=np.ones(n, np.int32),
                        dtype=gpu.DTYPE_F32 if f32 else gpu.DTYPE_I32) as eng:
            out = []
            for lanes, delta, pred in ((8, 0.0, True), (0, 0.0, True), (0, 2.0, True), (0, 0.0, False)):
                eng.set_option(gpu._lib.OPT_SSSP_LANES, lanes)
                eng.set_option(gpu._lib.OPT_SSSP_DELTA, delta)
                d = torch.full((sources, n + 3), 7, dtype=torch.float32 if f32 else torch.int32, device="cuda")
                p = torch.full((sources, n + 3), 7, dtype=torch.int32, device="cuda")
                eng.sssp(src, d, p if pred else None, ld=n + 3)
                torch.cuda.synchronize()
                out.append((d, p))
            for d, p in out[1:3]:
                assert torch.equal(d, out[0][0]) and torch.equal(p, out[0][1])
            assert torch.equal(out[3][0], out[0][0]) and bool((out[3][1] == 7).all())


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("n", [130, 4100, 70001])
def test_minplus_strip_lengths_agree(ctx, f32, n):
    """Strips of 128 to 2,048 columns (by how many the product has) give the
    rows of the same product in slices of 100 columns."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    m, k = max(260, 6100000 // n), 19

    def side(r, c):
        x = torch.rand(r, c, device="cuda", generator=gen) * 100
        x = x if f32 else x.int()
        return x.masked_fill_(torch.rand(r, c, device="cuda", generator=gen) < 0.3, 1e8 if f32 else 1 << 30)

    a, b = side(m, k), side(k, n)
    bp = torch.randint(0, n, (k, n), device="cuda", generator=gen, dtype=torch.int32)
    c, cp = torch.empty((m, n), dtype=a.dtype, device="cuda"), torch.empty((m, n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.minplus(0 if f32 else 1, a, b, c, Bp=bp, Cp=cp)
    for j in range(0, n, max(100, n // 20)):
        w = min(100, n - j)
        d, dp = torch.empty((m, w), dtype=a.dtype, device="cuda"), torch.empty((m, w), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ctx.minplus(0 if f32 else 1, a, b[:, j:j + w], d, Bp=bp[:, j:j + w], Cp=dp)
        assert torch.equal(d, c[:, j:j + w]) and torch.equal(dp, cp[:, j:j + w])


@pytest.mark.parametrize("pred", [True, False])
@pytest.mark.parametrize("kind", ["f32", "packed", "wide"])
@pytest.mark.parametrize("m, n, k, pad", [(64, 64, 101, 0), (65, 63, 128, 1), (1, 130, 192, 0), (130, 257, 500, 3),
                                          (200, 64, 129, 3), (61, 192, 260, 4)])
def test_minplus_of_many_steps(ctx, kind, pred, m, n, k, pad):
    """More steps than the strip form takes: the rows of a step-by-step product
    (strict improvements, ascending steps), at edges of tiles, chunks and
    alignments; `wide` has int32 values past the packed range."""
    gen = torch.Generator(device="cuda").manual_seed(m * 1000 + n + k)
    dt, inf = (torch.float32, 1e8) if kind == "f32" else (torch.int32, 1 << 30)

    def side(r, c):  # few distinct values: ties within and across groups and chunks
        x = torch.randint(0, 40, (r, c + pad), device="cuda", generator=gen) * ((1 << 22) if kind == "wide" else 1)
        x = (x * 0.1 if kind == "f32" else x).to(dt)
        return x.masked_fill_(torch.rand(r, c + pad, device="cuda", generator=gen) < 0.4, inf)[:, :c]

    a, b = side(m, k), side(k, n)
    b[:, n // 2] = inf  # a column that nothing reaches
    bp = torch.randint(0, n, (k, n), device="cuda", generator=gen, dtype=torch.int32)
    ref = torch.full((m, n), inf, dtype=dt, device="cuda")
    refp = torch.full((m, n), -1, dtype=torch.int32, device="cuda")
    for i in range(k):
        v = a[:, i, None] + b[i]
        better = (v < ref) & (a[:, i, None] < inf) & (b[i] < inf)
        ref, refp = torch.where(better, v, ref), torch.where(better, bp[i].expand(m, n), refp)
    c = torch.full((m, n + pad), 7, dtype=dt, device="cuda")
    cp = torch.full((m, n + pad), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    if pred:
        ctx.minplus(0 if kind == "f32" else 1, a, b, c[:, :n], Bp=bp, Cp=cp[:, :n])
        assert torch.equal(cp[:, :n], refp) and bool((cp[:, n:] == 7).all())
    else:
        ctx.minplus(0 if kind == "f32" else 1, a, b, c[:, :n])
    assert torch.equal(c[:, :n], ref) and bool((c[:, n:] == 7).all())


@pytest.mark.parametrize("f32", [False, True])
def test_solve_with_many_boundary_vertices(gpu, f32):
    """Parts whose boundaries exceed the strip form's steps and the packed index:
    int32 rows equal the wide form's, FP32 rows (integer weights) the same values."""
    g = graphs.small_random_graph(901, 5000, True, True, seed=9)
    gid, _ = gpu.partition(g.row_offset, g.col_val, 3)
    outs = []
    for dtype, form in ((gpu.DTYPE_I32, 1), (gpu.DTYPE_F32 if f32 else gpu.DTYPE_I32, 0)):
        with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, 3, graph_id=gid, dtype=dtype) as eng:
            assert max(eng.part_info(p)[1] for p in range(1, 4)) > 127
            if dtype == gpu.DTYPE_I32:
                eng.set_option(gpu._lib.OPT_INT32_FORM, form)
            d = torch.empty((g.n, g.n), dtype=torch.int32 if dtype == gpu.DTYPE_I32 else torch.float32, device="cuda")
            p = torch.empty((g.n, g.n), dtype=torch.int32, device="cuda")
            eng.solve(d, p, gpu.MODE_BATCHED)
            eng.solve(d, p, gpu.MODE_BATCHED)  # the captured graph
            torch.cuda.synchronize()
            outs.append((as_oracle(d.cpu().numpy()), p.cpu().numpy()))
    assert np.array_equal(outs[0][0], outs[1][0])
    assert np.array_equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("pred", [True, False])
@pytest.mark.parametrize("m, n, k, off", [(128, 65537, 1, 1), (129, 65600, 4, 3), (3, 2800001, 19, 0),
                                          (4100, 2049, 33, 5), (6100, 1001, 40, 7)])
def test_minplus_of_rows_off_boundaries(ctx, m, n, k, off, pred):
    """Packed products into rows that start off 16-byte boundaries (odd lengths and
    offsets) equal those into aligned rows."""
    gen = torch.Generator(device="cuda").manual_seed(m + n * k)

    def side(r, c):
        x = torch.randint(0, 50, (r, c), device="cuda", generator=gen, dtype=torch.int32)
        return x.masked_fill_(torch.rand(r, c, device="cuda", generator=gen) < 0.5, 1 << 30)

    a, b = side(m, k), side(k, n)
    b[:, : min(n, 200)] = 1 << 30  # tiles without a step
    bp = torch.randint(0, n, (k, n), device="cuda", generator=gen, dtype=torch.int32)
    outs = []
    for ld, o in ((n + 32 - n % 32, 0), (n | 1, off)):
        c, p = (torch.full((m * ld + 64,), 7, dtype=torch.int32, device="cuda") for _ in range(2))
        cv, pv = (x[o:o + m * ld].view(m, ld)[:, :n] for x in (c, p))
        torch.cuda.synchronize()
        ctx.minplus(1, a, b, cv, Bp=bp if pred else None, Cp=pv if pred else None)
        outs.append((cv.clone(), pv.clone()))
        cv[:], pv[:] = 7, 7
        assert bool((c == 7).all()) and bool((p == 7).all())  # nothing outside the rows
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("n, parts", [(3001, 3), (1537, 12)])
def test_solve_of_odd_rows_matches_wide_form(gpu, n, parts):
    g = graphs.geometric_knn(n, seed=n)
    gid, _ = gpu.partition(g.row_offset, g.col_val, parts)
    outs = []
    for form in (0, 1):
        with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, parts, graph_id=gid, dtype=gpu.DTYPE_I32) as eng:
            eng.set_option(gpu._lib.OPT_INT32_FORM, form)
            d, p = (torch.empty((g.n, g.n), dtype=torch.int32, device="cuda") for _ in range(2))
            eng.solve(d, p, gpu.MODE_BATCHED)
            eng.solve(d, p, gpu.MODE_BATCHED)  # the captured graph
            torch.cuda.synchronize()
            outs.append((d, p))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
