"""The boundary-graph method with eight and four sources a CTA (csrc/bgraph.cu): by
how many boundary vertices there are, and by what their table takes."""
import numpy as np
import pytest
import torch

from fastapsp_gb300 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("parts, low, high", [(150, 0, 1216), (220, 1217, 1600), (280, 1610, 2800)])
def test_boundary_graph_widths_match_the_search(gpu, f32, parts, low, high):
    """9,000 vertices with up to 8 x 152 boundary vertices (four), more (eight), and
    more than 1,600 (four with 8-byte distances, of whose tables an SM holds one):
    the rows of the whole-graph search."""
    g = graphs.road_like(9000, seed=10)
    w = g.weight if f32 else np.maximum(1, np.round(g.weight))
    gid, _ = gpu.partition(g.row_offset, g.col_val, parts)
    dtype, tdt = (gpu.DTYPE_F32, torch.float32) if f32 else (gpu.DTYPE_I32, torch.int32)
    outs = []
    for method in (2, 1):
        with gpu.Engine(g.n, g.row_offset, g.col_val, w, parts, graph_id=gid, dtype=dtype) as eng:
            assert low <= sum(eng.part_info(q)[1] for q in range(1, parts + 1)) <= high
            eng.set_option(gpu._lib.OPT_SSSP_METHOD, method)
            eng.set_option(gpu._lib.OPT_SSSP_FP64, 1 if f32 else 0)
            d = torch.empty((g.n, g.n), dtype=tdt, device="cuda")
            p = torch.empty((g.n, g.n), dtype=torch.int32, device="cuda")
            eng.solve(d, p)
            torch.cuda.synchronize()
            assert (eng.sssp_stats()["batches"] == 0) == (method == 2)
            outs.append((d, p))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
