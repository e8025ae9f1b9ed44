"""GPU: allocation-free grid queries on a mesh made mostly of needles are answered by the double kernel, which
keeps no list: they share nothing, so calls may overlap on several streams (calls on other meshes share the
library's array and may not), the first call of a process may be captured, and a capture holds one kernel."""

import numpy as np
import pytest
import torch

import ssdf_b200 as S
from ssdf_b200 import workloads as W
from test_zz_no_alloc import allocating, call_noalloc

pytestmark = pytest.mark.gpu


def test_overlapping_calls_on_needles():
    mesh = W.beam_lattice(60)
    dm = S.DeviceMesh(mesh)
    assert 2 * dm.filter_info()["slivers"] > mesh.nt
    streams = [torch.cuda.Stream() for _ in range(3)]
    grids = [W.Grid.padded_nodes(mesh, n, 0.2) for n in (31, 64, 47)]
    want = [allocating(dm, g, S.PREC_F64, torch.cuda.current_stream())[:2] for g in grids]
    outs = [(torch.empty(g.size, dtype=torch.float64, device="cuda"),
             torch.empty(g.size, dtype=torch.int32, device="cuda")) for g in grids]
    for _ in range(5):
        for o, t in outs:
            o.fill_(-1.0)
            t.fill_(-7)
        torch.cuda.synchronize()
        for g, (o, t), s in zip(grids, outs, streams):
            assert call_noalloc(dm, g, o, t, s) == S.SSDF_OK, S.last_error()
        torch.cuda.synchronize()
        for (o, t), (d, i) in zip(outs, want):
            assert np.array_equal(o.cpu().numpy(), d) and np.array_equal(t.cpu().numpy(), i)
    dm.close()


def test_captured_call_on_needles_is_one_kernel():
    mesh = W.beam_lattice(40)
    dm = S.DeviceMesh(mesh)
    grid = W.Grid.padded_nodes(mesh, 32, 0.2)
    out = torch.empty(grid.size, dtype=torch.float64, device="cuda")
    tri = torch.empty(grid.size, dtype=torch.int32, device="cuda")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        assert call_noalloc(dm, grid, out, tri, torch.cuda.current_stream()) == S.SSDF_OK, S.last_error()
    from cuda.bindings import runtime

    err, _, n = runtime.cudaGraphGetNodes(graph.raw_cuda_graph())
    assert int(err) == 0 and n == 1
    graph.replay()
    torch.cuda.synchronize()
    want, wtri, _ = allocating(dm, grid, S.PREC_F64, torch.cuda.current_stream())
    assert np.array_equal(out.cpu().numpy(), want) and np.array_equal(tri.cpu().numpy(), wtri)
    dm.close()
