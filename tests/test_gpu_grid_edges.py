"""GPU: grids whose last bricks are partly outside (one column, one row, one plane, or only a corner inside),
in which a lane other than the brick's centre one ranks the children; and blocks that walk 1 to 8 steps
upwards. Distances and indices must equal the oracle's brute force bit for bit (either order of the children
finds the same triangle, so there is no tolerance)."""

import numpy as np
import pytest
import torch

import oracle
import ssdf_b200 as S
from ssdf_b200 import workloads as W

pytestmark = pytest.mark.gpu


def nodes(n, lo, hi):
    """x-fastest node coordinates by the kernels' rule: lo + i h with h = (hi - lo) / (n - 1), or lo for n = 1."""
    ax = [l + np.arange(k) * ((h - l) / (k - 1) if k > 1 else 0.0) for k, l, h in zip(n, lo, hi)]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return np.stack([x.ravel(), y.ravel(), z.ravel()])


@pytest.mark.parametrize("steps", ["1", "2", "4", "8"])
@pytest.mark.parametrize("n", [(1, 1, 1), (5, 4, 4), (4, 5, 4), (4, 4, 5), (9, 5, 3), (6, 13, 1), (7, 3, 37)])
def test_grids_with_partly_filled_bricks(n, steps, monkeypatch):
    monkeypatch.setenv("SSDF_B200_GRID_STEPS", steps)
    mesh = W.torus(nu=30, nv=15, jitter=0.02)
    lo, hi = (tuple(float(v) for v in b) for b in (mesh.bbox()[0] - 0.2, mesh.bbox()[1] + 0.3))
    grid = W.Grid(n, lo, hi)
    want, wtri = oracle.edf(nodes(n, lo, hi), mesh, with_index=True)
    dm = S.DeviceMesh(mesh)
    for budget in (None, "2"):
        if budget:
            monkeypatch.setenv("SSDF_B200_WARP_BUDGET", budget)
        for prec in (S.PREC_F64, S.PREC_F32_FIXUP):
            out = torch.full((grid.size,), torch.finfo(torch.float64).max, dtype=torch.float64, device="cuda")
            tri = torch.full((grid.size,), -1, dtype=torch.int32, device="cuda")
            dm.query_grid(grid, out, tri, precision=prec, output=S.OUT_EDF)
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want) and np.array_equal(tri.cpu().numpy(), wtri), (prec, budget)
    dm.close()


@pytest.mark.parametrize("prec", [S.PREC_F64, S.PREC_F32_FIXUP])
def test_captured_grid_equals_the_plain_call(prec):
    mesh = W.torus(nu=30, nv=15, jitter=0.02)
    grid = W.Grid.padded_nodes(mesh, 21, 0.2)
    dm = S.DeviceMesh(mesh)
    plain, replayed = (torch.zeros(grid.size, dtype=torch.float64, device="cuda") for _ in range(2))
    dm.query_grid(grid, plain, precision=prec)
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        dm.query_grid(grid, replayed, precision=prec, stream=stream)
    for _ in range(2):
        replayed.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(plain, replayed)
    del graph
    dm.close()
