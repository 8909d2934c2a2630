"""The boundary searches of one engine: options changed between solves, parts with
few boundary vertices, many sources on graphs of many edges."""
import numpy as np
import pytest
import torch

from fastapsp_gb300 import graphs

pytestmark = pytest.mark.gpu


def solve(eng, n):
    d = torch.empty((n, n), device="cuda")
    p = torch.empty((n, n), dtype=torch.int32, device="cuda")
    eng.solve(d, p)
    launches = eng.last_launches()
    eng.solve(d, p)
    torch.cuda.synchronize()
    return d, p, launches - eng.last_launches()  # kernels of the first run's trials


def test_each_search_has_its_own_step(gpu):
    """The search with one CTA per source leaves the batched one's step to be
    tuned on its own first run, and keeps 64 x the mean weight before and after;
    the rows are the same, the FP64 search's within its rounding."""
    g = graphs.road_like(3001, seed=5)
    gid, _ = gpu.partition(g.row_offset, g.col_val, 4)
    mean = float(np.mean(g.weight.astype(np.float64)))
    L = gpu._lib
    with gpu.Engine(g.n, g.row_offset, g.col_val, g.weight, 4, graph_id=gid, dtype=gpu.DTYPE_F32) as eng:
        d0, p0, _ = solve(eng, g.n)
        assert eng.get_option(L.OPT_SSSP_DELTA) == pytest.approx(64 * mean)
        eng.set_option(L.OPT_SSSP_FP64, 1)
        assert eng.get_option(L.OPT_SSSP_DELTA) == pytest.approx(8 * mean)
        eng.set_option(L.OPT_SSSP_FP64, 0)
        eng.set_option(L.OPT_SSSP_LANES, 16)
        assert eng.get_option(L.OPT_SSSP_DELTA) == pytest.approx(8 * mean)
        d1, p1, trials = solve(eng, g.n)
        assert trials >= 9  # nine steps were tried
        tuned = eng.get_option(L.OPT_SSSP_DELTA)
        eng.set_option(L.OPT_SSSP_LANES, 0)
        assert eng.get_option(L.OPT_SSSP_DELTA) == pytest.approx(64 * mean)
        d2, p2, _ = solve(eng, g.n)
        assert all(torch.equal(a, d0) for a in (d1, d2)) and all(torch.equal(a, p0) for a in (p1, p2))
        eng.set_option(L.OPT_SSSP_LANES, 8)
        assert eng.get_option(L.OPT_SSSP_DELTA) == tuned
        assert solve(eng, g.n)[2] == 0
        eng.set_option(L.OPT_SSSP_DELTA, 3.0)  # a step of the program's own is every search's
        for lanes in (0, 16):
            eng.set_option(L.OPT_SSSP_LANES, lanes)
            assert eng.get_option(L.OPT_SSSP_DELTA) == 3.0
            d, p, trials = solve(eng, g.n)
            assert trials == 0 and torch.equal(d, d0) and torch.equal(p, p0)
        eng.set_option(L.OPT_SSSP_LANES, 0)
        eng.set_option(L.OPT_SSSP_DELTA, 0)
        eng.set_option(L.OPT_SSSP_FP64, 1)
        d, _, _ = solve(eng, g.n)
        # FP32 sums of at most n weights against one rounding
        assert bool(((d - d0).abs() <= g.n * 2.0 ** -24 * d).all())


def test_parts_with_few_boundary_vertices(gpu):
    """60 parts of a chain have 118 boundary vertices, whose lists of eight have 480
    places: the search takes a CTA, and its scratch (24 bytes a vertex), a source."""
    n, parts = 20001, 60
    src = np.arange(n - 1)
    g = graphs.csr_from_lines(n, src, src + 1, np.random.default_rng(1).integers(1, 9, n - 1), False, True)
    gid = (np.arange(n) * parts // n + 1).astype(np.int32)
    L = gpu._lib
    with gpu.Engine(n, g.row_offset, g.col_val, g.weight, parts, graph_id=gid, dtype=gpu.DTYPE_F32) as eng:
        info = [eng.part_info(q) for q in range(1, parts + 1)]
        sources = sum(b for _, b, _ in info)
        assert sources == 118
        d = torch.empty((n, n), device="cuda")
        p = torch.empty((n, n), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        eng.solve(d, p)
        torch.cuda.synchronize()
        taken = before - torch.cuda.mem_get_info()[0]
        closures = sum(8 * (-(-s // 64) * 64) ** 2 + 49152 for s, _, _ in info)
        assert taken < closures + sources * 24 * n + (48 << 20)
        e, q = torch.empty_like(d), torch.empty_like(p)
        eng.set_option(L.OPT_SSSP_LANES, 8)
        eng.solve(e, q)
        torch.cuda.synchronize()
        assert torch.equal(d, e) and torch.equal(p, q)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("n, degree, sources", [(100001, 5, 580), (100001, 5, 570), (100001, 4, 580),
                                                (230001, 5, 255)])
def test_wide_ctas_in_turns_match_batches(gpu, f32, n, degree, sources):
    """Past four edges a vertex and 220 MB of rows at once: sources in turns of one an
    SM; on either side of each line the rows of the batched search."""
    g = graphs.small_random_graph(n, degree * n + (degree == 5), True, True, seed=n, integer=not f32)
    src = np.random.default_rng(n).permutation(n)[:sources].astype(np.int32)
    L = gpu._lib
    with gpu.Engine(n, g.row_offset, g.col_val, g.weight, 1, graph_id=np.ones(n, np.int32),
                    dtype=gpu.DTYPE_F32 if f32 else gpu.DTYPE_I32) as eng:
        out = []
        for lanes in (0, 32, 0):
            eng.set_option(L.OPT_SSSP_LANES, lanes)
            d = torch.empty((sources, n), dtype=torch.float32 if f32 else torch.int32, device="cuda")
            p = torch.empty((sources, n), dtype=torch.int32, device="cuda")
            eng.sssp(src, d, p)
            eng.sssp(src[:200], d[:200], p[:200])  # fewer, with what the scratch holds
            torch.cuda.synchronize()
            out.append((d, p))
        for d, p in out[1:]:
            assert torch.equal(d, out[0][0]) and torch.equal(p, out[0][1])


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("degree, factor", [(3, 64.0), (4, 190 / 16), (8, 190 / 64), (24, 0.5)])
def test_step_by_edges_a_vertex(gpu, f32, degree, factor):
    """The automatic step of the search with one CTA per source shortens with the
    edges a vertex has; the rows do not depend on it."""
    n = 3001
    g = graphs.small_random_graph(n, degree * n, True, True, seed=degree)
    mean = float(np.mean(g.weight.astype(np.float64)))
    want = factor * mean if f32 else max(1.0, np.floor(factor * mean))
    src = np.arange(0, n, 7, dtype=np.int32)
    with gpu.Engine(n, g.row_offset, g.col_val, g.weight, 1, graph_id=np.ones(n, np.int32),
                    dtype=gpu.DTYPE_F32 if f32 else gpu.DTYPE_I32) as eng:
        assert eng.get_option(gpu._lib.OPT_SSSP_DELTA) == pytest.approx(want)
        out = []
        for delta in (0.0, 64 * mean):
            eng.set_option(gpu._lib.OPT_SSSP_DELTA, delta)
            d = torch.empty((len(src), n), dtype=torch.float32 if f32 else torch.int32, device="cuda")
            p = torch.empty((len(src), n), dtype=torch.int32, device="cuda")
            eng.sssp(src, d, p)
            torch.cuda.synchronize()
            out.append((d, p))
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
